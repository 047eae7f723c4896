// The schedule of the plane kernel's partial sums (plane_steps.hpp): over every order of phases, no
// phase writes a slot that is read at its start (after the barrier before it, with none between),
// and every slot read holds the sums of the phase that it is read for.
#include "../../glia_gb300/csrc/plane_steps.hpp"

#include <cstdio>
#include <vector>

using namespace glia;

int bad = 0;
int holder[kPlanePartials];  // the phase whose sums a slot holds

// one phase: `reads` are added by every CTA at its start, as sums of `from`
void phase(int step, PlaneSlots reads, std::vector<int> from) {
  const PlaneSlots w = plane_sums(step);
  if (w.first < 0 || w.first + w.count > kPlanePartials) bad++, std::printf("range %d\n", step);
  for (int q = 0; q < reads.count; q++) {
    const int s = reads.first + q;
    if (holder[s] != from[q]) bad++, std::printf("slot %d of phase %d is lost\n", s, from[q]);
    if (s >= w.first && s < w.first + w.count)
      bad++, std::printf("phase %d writes slot %d, which is read at its start\n", step, s);
  }
  for (int q = 0; q < w.count; q++) holder[w.first + q] = step;
}

int main() {
  const PlaneSlots none{0, 0};
  const std::vector<int> setup(4, PS_SETUP), update(2, PS_UPDATE);
  for (int iterations = 0; iterations < 4; iterations++) {
    for (int broken = 0; broken < 2; broken++) {  // PS_UPDATE finds the operator indefinite
      for (int& h : holder) h = -1;
      phase(PS_FWD, none, {});
      phase(PS_ENTER, none, {});
      phase(PS_GRAD, none, {});
      phase(PS_SETUP, none, {});
      PlaneSlots after = plane_sums(PS_SETUP);
      std::vector<int> of = setup;
      for (int i = 0; i < iterations; i++) {
        if (i) {
          phase(PS_DIR, after, of);
          after = none;
          of.clear();
        }
        phase(PS_GRAD, after, of);
        // the first direction's |p|^2 is one of the set-up's sums
        const PlaneSlots alpha = i ? kPlaneAlphaSums : plane_sums(PS_GRAD);
        const std::vector<int> parts = i ? std::vector<int>{PS_DIR, PS_GRAD}
                                         : std::vector<int>{PS_GRAD};
        if (broken && i == iterations - 1) {
          phase(PS_LEAVE, alpha, parts);
          after = none;
          of.clear();
          break;
        }
        // slot 0 is read (and not used) in the first iteration, too
        for (int q = 0; q < plane_sums(PS_UPDATE).count; q++)
          if (plane_sums(PS_UPDATE).first + q < kPlaneAlphaSums.first + kPlaneAlphaSums.count)
            bad++, std::printf("PS_UPDATE writes alpha's sums\n");
        phase(PS_UPDATE, alpha, parts);
        after = plane_sums(PS_UPDATE);
        of = update;
      }
      phase(PS_LEAVE, after, of);
      phase(PS_BACK, none, {});
    }
  }
  for (int& h : holder) h = -1;
  for (int step : {PS_FWD, PS_ENTER, PS_GRAD, PS_DOT}) phase(step, none, {});
  phase(PS_BACK, plane_sums(PS_DOT), {PS_DOT});
  return bad != 0;
}
