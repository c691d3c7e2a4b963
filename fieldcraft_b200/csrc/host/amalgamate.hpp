// The device factor's supernodes: the reference's, with small neighbours in the tree merged.
//
// The reference's fundamental supernodes keep the exact fill pattern; on the device each of them is
// a front to assemble, a level's launches and an update matrix written and read once. Merging a
// supernode into its parent stores some explicit zeros and takes the child's update matrix and often
// a level away. On the 48^3 hex8 block the 36 407 supernodes become 5 627, the 93 levels 14, the update
// matrices' lower triangles 5.7e9 entries 1.3e9, for 1.8 % more entries in L (7.4 % more bytes: the panels
// are stored as rectangles) and 0.4 % more operations. A solve multiplies by the inverses of wider blocks
// and sums in another order: its residual is 1.18 times that on the supernodes unmerged, its error 1.09
// times (geometric means over 48 boxes and plates of 2 000 to 9 000 unknowns).
#pragma once

#include <cstdint>
#include <vector>

#include "symbolic.hpp"

namespace fc {

// The structure the device factors by: merged supernodes over a new order of the columns (each
// supernode's columns together, descendants before ancestors). Rows are new columns, each
// supernode's own first, sorted.
struct Amalgamated {
  int64_t ns = 0;
  std::vector<int32_t> place;    // n: the new column of each postordered column
  std::vector<int32_t> column;   // n: the postordered column of each new one
  std::vector<int64_t> first;    // ns + 1
  std::vector<int64_t> rptr;     // ns + 1
  std::vector<int32_t> rows;
  std::vector<int64_t> sparent;  // NONE at roots
  int64_t width(int64_t s) const { return first[s + 1] - first[s]; }
  int64_t height(int64_t s) const { return rptr[s + 1] - rptr[s]; }
};

// Whether a child of w_child columns is merged into a parent of w_parent: `zeros` of the merged
// trapezoid's `entries` would be explicit zeros. Cheap where the merged supernode is narrow (such a
// front is launches and dependent loads, not arithmetic), a few per cent where it is wide, and always
// while the zeros are few: MERGE_ZEROS of them are 32 KB, less than a launch costs. Measured against
// no merging (factor and solve; and without the last rule): 24 624 unknowns, 7 loads 5.5 -> 3.3 ms
// (3.4); 345 744, 64 loads 158 -> 117 (119); 40 uneven boxes 9.6 -> 5.5 (5.8); mixed precision,
// 154 000, 16 loads 46 -> 21.6 (23); one solve, 107 163 2.5 -> 0.92 (1.0). Shares of 0.2 and 0.6 at 64
// and 32 columns came out within 3 % of these, 0.2 everywhere cost more arithmetic than it saved.
constexpr double MERGE_ZEROS = 4000;
bool merge_pays(int64_t w_child, int64_t w_parent, double zeros, double entries);

// merge = false: the same structure, every supernode its own.
Amalgamated amalgamate(const Symbolic &sym, bool merge);

}  // namespace fc
