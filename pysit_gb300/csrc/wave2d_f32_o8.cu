// 2D tile kernels, float, order 8 (one translation unit per type and order: they compile side by side)
#include "wave2d_tile.cuh"

namespace pgb {
PGB_INSTANTIATE_2D(float, 4)
}  // namespace pgb
