// 3D tile kernels, float, order 6 (one translation unit per type and order: they compile side by side)
#include "wave3d_tile.cuh"

namespace pgb {
PGB_INSTANTIATE_3D(float, 3)
}  // namespace pgb
