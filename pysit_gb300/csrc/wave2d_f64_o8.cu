// 2D tile kernels, double, order 8 (one translation unit per type and order: they compile side by side)
#include "wave2d_tile.cuh"

namespace pgb {
PGB_INSTANTIATE_2D(double, 4)
}  // namespace pgb
