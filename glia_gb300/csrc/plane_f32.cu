// Plane kernels of the mixed engine: the sizes whose plane leaves room for two CTAs per SM. 256^3
// has passes of its own (xpass.cuh, ownfft.cuh, zpass2.cuh), which stream through HBM.
#include "plane.cuh"

namespace glia {
template <>
PlaneKernel plane_kernel<float>(int n) {
  switch (n) {
    case 16: return plane_entry<float, 16>();
    case 32: return plane_entry<float, 32>();
    case 64: return plane_entry<float, 64>();
    case 96: return plane_entry<float, 96>();
    case 128: return plane_entry<float, 128>();
    default: return PlaneKernel{nullptr, 0, 0, 0, false};
  }
}
}  // namespace glia
