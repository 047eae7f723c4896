// Plane kernels of the FP64 engine, 104^3 to 144^3 (one CTA per SM).
#include "plane.cuh"

namespace glia {
PlaneKernel plane_kernel_f64_mid(int n) {
  switch (n) {
    case 104: return plane_entry<104>();
    case 112: return plane_entry<112>();
    case 120: return plane_entry<120>();
    case 128: return plane_entry<128>();
    case 144: return plane_entry<144>();
    default: return PlaneKernel{};
  }
}
}  // namespace glia
