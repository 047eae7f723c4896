// plane.hpp — interface of the persistent plane kernels (plane.cuh), one instantiation per grid size,
// compiled in translation units of their own.
#pragma once

#include "kernels.cuh"
#include "plane_steps.hpp"

namespace glia {

enum PlaneProg {
  PP_SOLVE = 0,  // one Crank-Nicolson solve, in -> out
  PP_APPLY,      // D in -> out
  PP_SMOOTH,     // in convolved with mulk -> out
  PP_SPEC,       // spectrum of in -> chat
  PP_DOT         // acc[6] += kdot_weight <cx, D in>
};

struct PlaneArgs {
  using C = double2;
  int prog, which;
  // field transformed, and what acts on it as it is read: 0 nothing, 1 the logistic step (half
  // receives the field itself when not null), 2 its linearisation at lin
  const double* in;
  int pre;
  const double* rho;
  const double* lin;
  double* half;
  double dt;
  double* out;
  const double* k;
  C *chat, *xhat, *rhat, *phat;  // spectrum of in, PCG vectors
  C *G, *M;                      // scratch: [G_x, G_0], [M_x, M_y, M_z]
  C* W;                          // scratch of split kernels: line pairs per component
  const C* cx;                   // spectrum whose product with D in joins acc[6] (may be null)
  const C* mulk;
  double a_cn, pc_c, rtol, abstol, divtol, kdot_weight;
  int maxit;
  DevScalars* sc;
  double* part;    // kPlanePartials values per CTA
  unsigned* bar;   // two counters, zero between launches
  long long wait;  // longest wait at a grid barrier, in SM clocks
  const void* tw;  // exp(2 pi i j / n), j < n, as FxTw (fx.cuh)
  const double* pf;  // the preconditioner 1 / (1 + pc_c |w|^2) per spectrum element
};

struct PlaneKernel {
  const void* fn;  // null: the grid size has no plane kernel
  int threads, smem;
  int items;       // most work items of a phase
  bool split;      // needs W
};
// One instantiation per grid size, in translation units by size: every multiple of 8 that factors
// into R1 <= 16 and R2 = 4, 8 or 16 (plane.cuh). That leaves 136, 152, 168, 184, 200, 216, 232 and
// 248 (a factor of 17 or more) on cuFFT's transforms. Time of a solve with cuFFT's transforms over
// this kernel's: 2.2 to 5.7 at every size.
PlaneKernel plane_kernel_f64_small(int n);
PlaneKernel plane_kernel_f64_mid(int n);
PlaneKernel plane_kernel_f64_large(int n);
void plane_twiddles(int n, int4* out);  // exp(2 pi i j / n), j < n, as FxTw (fx.cuh)
inline PlaneKernel plane_kernel(int n) {
  return n <= 96    ? plane_kernel_f64_small(n)
         : n <= 144 ? plane_kernel_f64_mid(n)
                    : plane_kernel_f64_large(n);
}

}  // namespace glia
