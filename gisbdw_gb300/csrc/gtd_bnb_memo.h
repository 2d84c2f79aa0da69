// Which slots of the branch and bound's kept memo must be cleared before a
// solve (host only).
//
// A solve of graphs of at most 64 vertices marks its slots with its own number
// and takes a slot with another number for empty; a solve with a wider graph
// has no room for the number and needs its slots cleared before, and a later
// solve could take them for its own. Fresh memory counts like such slots. A
// solve uses the slots [0, used); those that may hold an entry without a
// number are kept as one range [lo, hi).
#pragma once

#include <cstddef>

namespace gtd {

struct MemoSlots {
  size_t lo = 0, hi = 0;

  void fresh(size_t cap) {
    lo = 0;
    hi = cap;
  }

  // The slots [*first, *first + count) to clear before a solve on [0, used);
  // `wide`: the solve leaves entries without a number. Never more than the
  // solve uses, whatever the memo has grown to.
  size_t clear_before(size_t used, bool wide, size_t* first) {
    if (wide) {
      lo = 0;
      hi = hi > used ? hi : used;
      *first = 0;
      return used;
    }
    const size_t end = hi < used ? hi : used;
    *first = lo;
    if (end <= lo)
      return 0;
    const size_t count = end - lo;
    lo = end;
    if (lo == hi)
      lo = hi = 0;
    return count;
  }
};

}  // namespace gtd
