// Plane kernels of the FP64 engine. 256^3 is split (no plane fits): 45 -> 10.3 ms a solve, against
// cuFFT transforms that run at the FP64 units' rate.
#include "plane.cuh"

namespace glia {
template <>
PlaneKernel plane_kernel<double>(int n) {
  switch (n) {
    case 16: return plane_entry<double, 16>();
    case 32: return plane_entry<double, 32>();
    case 64: return plane_entry<double, 64>();
    case 96: return plane_entry<double, 96>();
    case 120: return plane_entry<double, 120>();
    case 128: return plane_entry<double, 128>();
    case 256: return plane_entry<double, 256>();
    default: return PlaneKernel{nullptr, 0, 0, 0, false};
  }
}
}  // namespace glia
