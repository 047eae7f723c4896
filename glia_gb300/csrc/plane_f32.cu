// Plane kernels of the mixed engine up to 128^3.
#include "plane.cuh"

namespace glia {
PlaneKernel plane_kernel_f32_small(int n) {
  switch (n) {
    case 16: return plane_entry<float, 16>();
    case 24: return plane_entry<float, 24>();
    case 32: return plane_entry<float, 32>();
    case 40: return plane_entry<float, 40>();
    case 48: return plane_entry<float, 48>();
    case 56: return plane_entry<float, 56>();
    case 64: return plane_entry<float, 64>();
    case 72: return plane_entry<float, 72>();
    case 80: return plane_entry<float, 80>();
    case 88: return plane_entry<float, 88>();
    case 96: return plane_entry<float, 96>();
    case 104: return plane_entry<float, 104>();
    case 112: return plane_entry<float, 112>();
    case 120: return plane_entry<float, 120>();
    case 128: return plane_entry<float, 128>();
    default: return PlaneKernel{};
  }
}
}  // namespace glia
