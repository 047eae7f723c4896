// Plane kernels of the FP64 engine up to 96^3.
#include "plane.cuh"

#include <cmath>

namespace glia {
PlaneKernel plane_kernel_f64_small(int n) {
  switch (n) {
    case 16: return plane_entry<16>();
    case 24: return plane_entry<24>();
    case 32: return plane_entry<32>();
    case 40: return plane_entry<40>();
    case 48: return plane_entry<48>();
    case 56: return plane_entry<56>();
    case 64: return plane_entry<64>();
    case 72: return plane_entry<72>();
    case 80: return plane_entry<80>();
    case 88: return plane_entry<88>();
    case 96: return plane_entry<96>();
    default: return PlaneKernel{};
  }
}
void plane_twiddles(int n, int4* out) {
  static_assert(sizeof(FxTw) == sizeof(int4), "table entry");
  for (int j = 0; j < n; j++) {
    const long double a = 2.0L * 3.14159265358979323846264338327950288L * j / n;
    const FxTw w{fx_from(std::cos(a)), fx_from(std::sin(a))};
    std::memcpy(&out[j], &w, sizeof(w));
  }
}
}  // namespace glia
