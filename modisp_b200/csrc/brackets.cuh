// brackets.cuh -- rules on a trace's bracket slots.  Plain C++: host programs build
// them too.
#pragma once
#include <stddef.h>

#if defined(__CUDACC__)
#define MD200_BRACKET_FN __host__ __device__ __forceinline__
#else
#define MD200_BRACKET_FN inline
#endif

namespace md200 {

constexpr int SLOT = 5;  // doubles per bracket slot: lo, hi, flo, fhi, root

// Does any point of bracket i, of the n brackets in `slots`, give the same result as
// its root, where that root is a guard (not reported)?  It counts, keeps its rank,
// and decides whether a neighbour is close.  So the bracket has to be clear of every
// other by more than the close-root distance, and its rank has to stay: an exact zero
// that two earlier brackets share becomes one root, and every rank after it moves down
// by one, a guard's among the reported ones.  Earlier brackets that touch are not
// settled for that reason.
MD200_BRACKET_FN bool guard_is_clear(const double *slots, int n, int i, double close_rtol) {
  const double lo = slots[static_cast<size_t>(i) * SLOT], hi = slots[static_cast<size_t>(i) * SLOT + 1];
  double before = 0.;  // (velocities are positive)
  for (int j = 0; j < n; ++j) {
    const double l = slots[static_cast<size_t>(j) * SLOT], h = slots[static_cast<size_t>(j) * SLOT + 1];
    if (j < i && !(l > before && lo - h > close_rtol * hi)) return false;
    if (j > i && !(l - hi > close_rtol * h)) return false;
    before = h;
  }
  return true;
}

// Do the FP64 values at a bracket's ends confirm it: finite, nonzero, of opposite
// signs?  (Refinement fails a bracket with an infinite end, so its product of signs
// must not settle one.)
MD200_BRACKET_FN bool ends_confirm(double fa, double fb) {
  return fa - fa == 0. && fb - fb == 0. && ((fa < 0. && fb > 0.) || (fa > 0. && fb < 0.));
}

}  // namespace md200
