// plane_steps.hpp — the phases of the plane kernel (plane.cuh) and the slots of its partial sums.
// Plain C++: the host test of the slots' schedule includes it.
#pragma once

namespace glia {

enum PlaneStep {
  PS_FWD = 0,   // planes: real field -> y, z forward
  PS_GRAD,      // planes: G -> gradient, times k, -> M
  PS_BACK,      // planes: G_0 -> real field
  PS_YINV,      // SPLIT: columns of planes, y inverse, G -> W (Z pairs)
  PS_LINE,      // SPLIT: line pairs in W, z inverse, k, z forward (GRAD; FWD: z forward only;
                //        BACK: z inverse only)
  PS_YFWD,      // SPLIT: columns of planes, y forward, W -> M
  PS_SPEC,      // columns: M_0 -> spectrum (stored)
  PS_ENTER,     // columns: M_0 -> spectrum (stored) -> G_x, G_0
  PS_SMOOTH,    // columns: M_0 -> spectrum times mulk -> G_0
  PS_SETUP,     // columns: M -> D c, solve set-up, first direction -> G_x, G_0
  PS_UPDATE,    // columns: M -> D p, x and r
  PS_DIR,       // columns: next direction -> G_x, G_0
  PS_LEAVE,     // columns: x -> G_0
  PS_APPLY,     // columns: M -> D u -> G_0
  PS_DOT        // columns: M -> <cx, D u>
};

// Partial sums. A phase writes its own slots at its end; every CTA reads the totals it needs right
// after the barrier that follows, and goes on to the next phase without another one. So no phase may
// write a slot that is read at its start: a CTA that is late out of the barrier would add a slot
// that others have begun to overwrite, and decide otherwise than they do. (PS_SETUP has slots apart
// from PS_GRAD's for this: PS_GRAD is the phase after it.)
struct PlaneSlots {
  int first, count;
};
#ifdef __CUDACC__
__host__ __device__
#endif
constexpr PlaneSlots plane_sums(int step) {  // what a phase writes
  return step == PS_DIR      ? PlaneSlots{0, 1}  // |p|^2
         : step == PS_GRAD   ? PlaneSlots{1, 1}  // k |grad p|^2
         : step == PS_UPDATE ? PlaneSlots{2, 2}  // ||z||^2, <z, r>
         : step == PS_DOT    ? PlaneSlots{2, 1}  // <cx, D u>
         : step == PS_SETUP  ? PlaneSlots{2, 4}  // ||P b||^2, ||z||^2, <z, r>, <cx, D c>
                             : PlaneSlots{0, 0};
}
constexpr PlaneSlots kPlaneAlphaSums{0, 2};  // read at the start of PS_UPDATE, for alpha
constexpr int kPlanePartials = 6;            // slots

}  // namespace glia
