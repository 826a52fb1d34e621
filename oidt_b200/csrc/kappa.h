// kappa.h -- the kappa dx tables of an axis (host code).
#pragma once

#include <cstddef>
#include <vector>

namespace oidt {

// kappa dx of an axis' n cells and their reciprocals, RN(1 / kappa dx) in T
// (EXACT divisions rely on it), as rows of `padded` cells.  The padding holds 1:
// the 3D vector form tests the reciprocals of a whole group for the fast
// quotient's range, and a zero would send the last group of every row of a
// length that is no multiple of the group to direct division, with all lanes
// of its warp (97 x 114 x 187 float64 EXACT 99 us per step, 79.5 with 1; float32
// EXACT 74 and 64; at a length of 188 78 and 64).  No update of the padding is
// kept.
template <typename T> void kappa_rows(const T *kd, size_t n, size_t padded, std::vector<T> &k, std::vector<T> &r) {
  k.assign(padded, T(1));
  r.assign(padded, T(1));
  for (size_t i = 0; i < n; ++i) {
    k[i] = kd[i];
    r[i] = (T)1 / kd[i];
  }
}

}  // namespace oidt
