// The row swaps of an elimination in place, undone on the host.
#pragma once
#include <utility>

namespace cvb {

// Column q of the inverse is column map[q] of the matrix that the elimination with the
// row swaps (c, perm[c]), c = 0 .. n - 1 in order, left: the swaps become column swaps
// in reverse order.  false, with nothing indexed by it, where an entry is no row from c
// on.
inline bool undo_row_swaps(const int *perm, int n, int *map) {
  for (int c = 0; c < n; c++)
    if (perm[c] < c || perm[c] >= n) return false;
  for (int q = 0; q < n; q++) map[q] = q;
  for (int c = n - 1; c >= 0; c--) std::swap(map[c], map[perm[c]]);
  return true;
}

}  // namespace cvb
