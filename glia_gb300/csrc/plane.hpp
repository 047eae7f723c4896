// plane.hpp — interface of the persistent plane kernels (plane.cuh), one instantiation per type and
// grid size, compiled in translation units of their own.
#pragma once

#include "kernels.cuh"

namespace glia {

enum PlaneProg {
  PP_SOLVE = 0,  // one Crank-Nicolson solve, in -> out
  PP_SOLVE_SPEC, // the same on spectra: chat -> xhat (times 1/n^3)
  PP_APPLY,      // D in -> out
  PP_SMOOTH,     // in convolved with mulk -> out
  PP_SPEC,       // spectrum of in -> chat
  PP_DOT         // acc[6] += kdot_weight <cx, D in>
};

constexpr int kPlanePartials = 6;  // partial-sum slots per CTA

template <typename R>
struct PlaneArgs {
  using C = typename CT<R>::C;
  int prog, which;
  // field transformed, and what acts on it as it is read: 0 nothing, 1 the logistic step (half
  // receives the field itself when not null), 2 its linearisation at lin
  const R* in;
  int pre;
  const R* rho;
  const R* lin;
  R* half;
  R dt;
  R* out;
  const R* k;
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
  const void* tw;  // exp(2 pi i j / n), j < n: float2, or FxTw for double
  const R* pf;     // double: the preconditioner 1 / (1 + pc_c |w|^2) per spectrum element
};

struct PlaneKernel {
  const void* fn;  // null: the grid size has no plane kernel
  int threads, smem;
  int items;       // most work items of a phase
  bool split;      // needs W
};
template <typename R>
PlaneKernel plane_kernel(int n);

}  // namespace glia
