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

}  // namespace spc
