// Plane kernels of the mixed engine above 128^3, as long as a plane fits in shared memory. 256^3 has
// passes of its own (xpass.cuh, ownfft.cuh, zpass2.cuh), which stream through HBM; 240 = 15 x 16 does
// not fit. us a solve, cuFFT's transforms -> this kernel: 144^3 540 -> 509, 160^3 802 -> 617, 176^3
// 1303 -> 1140, 192^3 1230 -> 910, 208^3 2827 -> 2016, 224^3 4244 -> 2364.
#include "plane.cuh"

namespace glia {
PlaneKernel plane_kernel_f32_large(int n) {
  switch (n) {
    case 144: return plane_entry<float, 144>();
    case 160: return plane_entry<float, 160>();
    case 176: return plane_entry<float, 176>();
    case 192: return plane_entry<float, 192>();
    case 208: return plane_entry<float, 208>();
    case 224: return plane_entry<float, 224>();
    default: return PlaneKernel{};
  }
}
}  // namespace glia
