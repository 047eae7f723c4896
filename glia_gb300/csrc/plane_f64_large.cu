// Plane kernels of the FP64 engine above 144^3: split, no plane fits in shared memory. A solve at 256^3
// takes 11.4 ms against 53 with cuFFT transforms, which run at the FP64 units' rate.
#include "plane.cuh"

namespace glia {
PlaneKernel plane_kernel_f64_large(int n) {
  switch (n) {
    case 160: return plane_entry<160>();
    case 176: return plane_entry<176>();
    case 192: return plane_entry<192>();
    case 208: return plane_entry<208>();
    case 224: return plane_entry<224>();
    case 240: return plane_entry<240>();
    case 256: return plane_entry<256>();
    default: return PlaneKernel{};
  }
}
}  // namespace glia
