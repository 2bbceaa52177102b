// Host arithmetic of the refinement's last correction (eig_refine.cu), apart from
// the kernels so that a host compiler can check it.
#pragma once

namespace tnad {

// Newton–Schulz steps that bring X·(I + E) back to orthogonality at FP64 rounding,
// em = max|E|: it is orthogonal up to ~4E², and every step squares that.
// 0: E is not a correction (em above 0.1, infinite or NaN) — a rotation of the
// last groups can leave two equal eigenvalues in different ones, and from em = ½
// on the squares do not shrink.  At most 4.
inline int orth_steps(float em) {
  if (!(em <= 0.1f)) return 0;
  int steps = 1;
  for (double d = 16.0 * (double)em * em * em * em; d > 1e-16; d *= d) ++steps;
  return steps;
}

}  // namespace tnad
