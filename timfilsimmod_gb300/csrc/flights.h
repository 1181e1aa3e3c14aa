// flights.h -- the launches of a service that may still run, and the slots
// (staging buffers, stream, completion event) that they hold. Host code without
// CUDA: tests/test_flights.py runs it alone.
#pragma once

#include <deque>

namespace tfs {

struct Flights {
  struct Flight {
    int slot, ctas;
  };
  std::deque<Flight> list;  // oldest first

  // CTAs in flight; flights whose slot has ended leave the list.
  template <typename Ended>
  int ctas(Ended ended) {
    int used = 0;
    for (auto it = list.begin(); it != list.end();) {
      if (ended(it->slot)) {
        it = list.erase(it);
      } else {
        used += it->ctas;
        ++it;
      }
    }
    return used;
  }

  // A slot of n that no flight holds; with fewer flights than slots there is one.
  // (Slots in turn, whatever still runs in them, would put a launch behind a
  // longer one and lose count of that one's CTAs.)
  int free_slot(int n) const {
    for (int i = 0; i < n; ++i) {
      bool held = false;
      for (const Flight &f : list) held = held || f.slot == i;
      if (!held) return i;
    }
    return -1;
  }

  void add(int slot, int ctas) { list.push_back({slot, ctas}); }
};

}  // namespace tfs
