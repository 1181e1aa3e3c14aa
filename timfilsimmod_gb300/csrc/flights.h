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

  // A launch of ctas CTAs behind every flight, in the given slot: wait(slot) for
  // each, launch(), record(slot), each 0 or an error that ends it. Only a launch
  // whose end is recorded replaces the flights; one that is not is synchronised.
  template <typename Wait, typename Launch, typename Record, typename Sync>
  int alone(int slot, int ctas, Wait wait, Launch launch, Record record, Sync sync) {
    int rc;
    for (const Flight &f : list)
      if ((rc = wait(f.slot)) != 0) return rc;
    if ((rc = launch()) != 0) return rc;
    if ((rc = record(slot)) != 0) {
      sync();
      return rc;
    }
    list.clear();
    add(slot, ctas);
    return 0;
  }
};

}  // namespace tfs
