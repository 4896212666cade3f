// The barrier between the CTAs of a cooperative grid: one word counts the arrivals of all barriers so far.  Waits
// are bounded; a CTA that gives up marks the word for good, unless the barrier completes first, so that all CTAs
// of a launch see the same end of its last barrier: either every one passes it or none does.
#pragma once

#include "chunks.cuh"

namespace hb {

constexpr unsigned kGaveUp = 0x80000000u;

// Word: add(1) that releases what was written before it, load() that acquires, swap(was, to), pause(turn).  want:
// arrivals when this barrier is complete.  (An arrival does not wait for the word's value: the first load says all.)
template <class Word>
HB_BOTH bool grid_barrier(Word& w, unsigned want, int turns) {
  w.add(1u);
  for (int it = 0; it < turns; ++it) {
    const unsigned seen = w.load();
    if (seen & kGaveUp) return false;
    if (seen >= want) return true;
    w.pause(it);
  }
  for (int it = 0; it < 65536; ++it) {  // (a swap fails once per arrival at most)
    const unsigned seen = w.load();
    if (seen & kGaveUp) return false;
    if (seen >= want) return true;
    if (w.swap(seen, seen | kGaveUp)) return false;
  }
  return false;
}

}  // namespace hb
