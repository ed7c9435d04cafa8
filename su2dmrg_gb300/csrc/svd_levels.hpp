// Host rules of the truncation's refinement levels (svd.cu), on eigenvalues in
// ascending order.
#pragma once
#include <vector>

namespace su2g {

constexpr double kDecade = 0.1;     // a level's top decade: from a tenth of the largest on
constexpr double kStepMax = 1e-3;   // larger first steps: an eigendecomposition

// index after the last eigenvalue below a tenth of the largest (tensor.cpp:1492-1497)
inline int small_count(const std::vector<double>& w, int n) {
  for (int i = n - 1; i >= 0; --i)
    if (w[i] / w[n - 1] < 1.e-1) return i + 1;
  return 0;
}

// whether the subspace of the first n values holds nothing that a truncation at
// `cut` keeps (cut 0: everything counts)
inline bool beyond_cut(const std::vector<double>& w, int n, double cut) { return cut > 0 && w[n - 1] < kDecade * cut; }

// Whether step `it` of a level's refinement may be taken: its eigenvalue
// estimates h, its largest correction `step`.  The top decade must follow the
// rest and be in ascending order, and a level that leaves a subspace beyond the
// cut is the last one, after whichever step that shows: the estimates below
// its decade are neither resolved nor sorted, so it takes an eigendecomposition.
inline bool level_settled(const std::vector<double>& h, double step, int it, double cut) {
  const int n = (int)h.size(), t0 = small_count(h, n);
  bool good = step <= (it > 0 ? 10 * kStepMax : kStepMax) && h[n - 1] > 0;
  for (int i = 0; i < n && good; ++i) {
    const bool in_top = h[i] >= kDecade * h[n - 1];
    good = in_top == (i >= t0) && (i <= t0 || h[i] >= h[i - 1]);
  }
  return good && !(t0 > 1 && beyond_cut(h, t0, cut));
}

}  // namespace su2g
