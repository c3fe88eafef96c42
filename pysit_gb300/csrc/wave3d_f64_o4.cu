// 3D tile kernels, double, order 4 (one translation unit per type and order: they compile side by side)
#include "wave3d_tile.cuh"

namespace pgb {
PGB_INSTANTIATE_3D(double, 2)
}  // namespace pgb
