// The device factor's supernodes: the reference's, with small neighbours in the tree merged.
//
// The reference's fundamental supernodes keep the exact fill pattern; on the device each of them is
// a front to assemble, a level's launches and an update matrix written and read once. Merging a
// supernode into its parent stores some explicit zeros and takes the child's update matrix and often
// a level away. On the 48^3 hex8 block the 36 407 supernodes become under 10 000, the tree 17 levels
// high at most instead of 93, the update matrices 1.4e9 entries instead of 5.75e9, for about 1 % more
// entries in L and half a per cent more operations.
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
