// Plane kernels of the FP64 engine up to 96^3.
#include "plane.cuh"

namespace glia {
PlaneKernel plane_kernel_f64_small(int n) {
  switch (n) {
    case 16: return plane_entry<double, 16>();
    case 24: return plane_entry<double, 24>();
    case 32: return plane_entry<double, 32>();
    case 40: return plane_entry<double, 40>();
    case 48: return plane_entry<double, 48>();
    case 56: return plane_entry<double, 56>();
    case 64: return plane_entry<double, 64>();
    case 72: return plane_entry<double, 72>();
    case 80: return plane_entry<double, 80>();
    case 88: return plane_entry<double, 88>();
    case 96: return plane_entry<double, 96>();
    default: return PlaneKernel{};
  }
}
}  // namespace glia
