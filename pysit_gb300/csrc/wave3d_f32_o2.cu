// 3D tile kernels, float, order 2 (one translation unit per type and order: they compile side by side)
#include "wave3d_tile.cuh"

namespace pgb {
PGB_INSTANTIATE_3D(float, 1)
}  // namespace pgb
