// Which activations a group of the network's passes runs in: the handle's own, which are there from
// its creation to its end, or a larger room that is made when a group first wants it.
#pragma once

#include <algorithm>
#include <climits>

namespace fc {

// A call takes the largest whole number of a vector's passes that there is room for. The larger room
// is never part of a captured graph (a later group may replace it), so a capture uses the handle's own,
// which no call frees. A size that found no memory is not tried again: the calls after it go on in what
// there is.
struct PassRoom {
  int own = 0;             // passes the handle's own activations hold
  int group = 0;           // passes the larger room holds, 0: none
  int refused = INT_MAX;   // the smallest size that found no memory
  struct Choice {
    int passes;      // how many run together (one of a vector's `per` where two do not fit)
    bool in_group;   // in the larger room
  };
  // Room for `want` passes, `per` a vector (want a multiple of per). grow(passes) replaces the larger
  // room, false (and none is left) when there is no memory.
  template <class Grow>
  Choice choose(int want, int per, bool capturing, Grow grow) {
    const int here = own >= per ? std::min(want, own / per * per) : 1;
    if (here >= want || capturing) return {here, false};
    if (refused <= want) want = (refused - 1) / per * per;
    if (want <= here) return {here, false};
    if (group >= want) return {want, true};
    for (; want > here; want -= per) {
      group = 0;
      if (grow(want)) {
        group = want;
        return {want, true};
      }
      refused = want;
    }
    return {here, false};
  }
};

}  // namespace fc
