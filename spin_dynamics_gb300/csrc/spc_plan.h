// Host arithmetic of bounds and memory plans, free of CUDA so that it can be
// tested by itself.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <vector>

namespace spc {

// A bound on ||H|| from the |re| + |im| of a CSR's entries (0-based; val: re, im
// pairs): sqrt of the largest row sum times the largest column sum (Hoelder), the
// row sum itself where H is symmetric in magnitude. NaN if an entry is.
inline double csr_norm_bound(int n, const int* rowptr, const int* col, const double* val) {
  std::vector<double> cols(n, 0.0);
  double row = 0.0, column = 0.0;
  for (int r = 0; r < n; ++r) {
    double t = 0.0;
    for (int k = rowptr[r]; k < rowptr[r + 1]; ++k) {
      const double a = std::fabs(val[2 * (size_t)k]) + std::fabs(val[2 * (size_t)k + 1]);
      t += a;
      cols[col[k]] += a;
    }
    if (t > row || t != t) row = t;
  }
  for (double t : cols)
    if (t > column || t != t) column = t;
  return std::sqrt(row) * std::sqrt(column);
}

// Memory plan of a yield gradient: checkpoints every K steps, whether a segment's
// node states are kept (one Krylov build a step saved), and the costate node
// states formed at a time.
struct GradPlan {
  int K = 1;
  bool keep = false;
  int nodes = 1;
  bool fits = true;
};
// extra(K, keep, nodes): bytes beyond what is held. K = 0 asks for a spacing: of
// those whose states fit, the one that recomputes the fewest steps (all but the
// last segment are recomputed), the larger on a tie; with none, the spacing of
// least memory. Spacing and kept states save builds and come first; the costate's
// node states take what is left, from all at once down to one after the other.
// `slack` is what the small buffers may use of the memory kept free.
template <class Extra>
GradPlan plan_gradient(int nsteps, int nq, int K, double avail, double slack, const Extra& extra) {
  GradPlan p;
  p.K = K;
  if (K == 0) {
    int64_t best = -1;
    for (int k = nsteps; k >= 1; --k) {
      if (extra(k, true, 1) > avail) continue;
      const int64_t recomputed = (int64_t)((nsteps - 1) / k) * k;
      if (best < 0 || recomputed < best) {
        best = recomputed;
        p.K = k;
      }
    }
    p.keep = p.K > 0;
    if (!p.keep) p.K = std::max(1, (int)std::lround(std::sqrt((double)nsteps)));
  } else {
    p.keep = extra(K, true, 1) <= avail;
  }
  p.nodes = nq;
  while (p.nodes > 1 && extra(p.K, p.keep, p.nodes) > avail) --p.nodes;
  p.fits = p.keep || extra(p.K, false, 1) <= avail + slack;
  return p;
}

}  // namespace spc
