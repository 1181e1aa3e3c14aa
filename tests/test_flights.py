"""The bookkeeping of a service's launches (csrc/flights.h) on the CPU: launches
that end out of order, more of them than slots."""
import ctypes
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = r'''
#include "flights.h"
using namespace tfs;
static Flights f;
static long now, ends[8];
static bool ended(int s) { return ends[s] <= now; }
extern "C" {
void reset() { f.list.clear(); now = 0; for (long &e : ends) e = 0; }
void wait_until(long t) { now = t; }
int ctas() { return f.ctas(ended); }
int flights() { return (int)f.list.size(); }
int fly(int n, int ctas, long end) {
  const int s = f.free_slot(n);
  if (s < 0) return s;
  ends[s] = end;
  f.add(s, ctas);
  return s;
}
// which call fails: 0 none, 1 the wait for a flight, 2 the launch, 3 the record
int alone(int n, int ctas, int fails, int *waits, int *synced) {
  *waits = *synced = 0;
  return f.alone(f.free_slot(n), ctas, [&](int) { ++*waits; return fails == 1 ? -1 : 0; },
                 [&] { return fails == 2 ? -2 : 0; },
                 [&](int s) { ends[s] = now + 50; return fails == 3 ? -3 : 0; },
                 [&] { *synced = 1; });
}
}
'''


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("flights")
    (d / "f.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-std=c++17",
                    "-I", os.path.join(ROOT, "timfilsimmod_gb300", "csrc"), str(d / "f.cpp"),
                    "-o", str(d / "f.so")], check=True, capture_output=True)
    return ctypes.CDLL(str(d / "f.so"))


def test_a_long_launch_beside_many_short_ones(lib):
    """A launch of 100 CTAs until t = 100, forty of 10 CTAs for 1 each, slots eight:
    the long one keeps its slot and its CTAs stay counted until it ends."""
    lib.reset()
    first = lib.fly(8, 100, 100)
    for t in range(1, 41):
        lib.wait_until(t)
        assert lib.ctas() == 100 and lib.flights() == 1
        assert lib.fly(8, 10, t + 1) != first
        assert lib.ctas() == 110
    lib.wait_until(99)
    assert lib.ctas() == 100
    lib.wait_until(100)
    assert lib.ctas() == 0 and lib.flights() == 0


def test_slots_are_of_one_launch_each(lib):
    lib.reset()
    assert sorted(lib.fly(8, 1, 10 + k) for k in range(8)) == list(range(8))
    assert lib.fly(8, 1, 5) == -1
    lib.wait_until(12)  # three have ended
    assert lib.ctas() == 5
    assert sorted(lib.fly(8, 1, 50) for _ in range(3)) == [0, 1, 2]


@pytest.mark.parametrize("fails", [0, 1, 2, 3])
def test_a_launch_on_all_ctas(lib, fails):
    """It replaces the flights it waits for, unless a step of it fails: then they
    stay, and a launch whose end is not recorded is waited for."""
    lib.reset()
    for k in range(3):
        lib.fly(8, 10, 20)
    waits, synced = ctypes.c_int(), ctypes.c_int()
    rc = lib.alone(8, 152, fails, ctypes.byref(waits), ctypes.byref(synced))
    assert rc == -fails and waits.value == (1 if fails == 1 else 3)
    assert synced.value == (fails == 3)
    assert lib.ctas() == (152 if fails == 0 else 30)
    lib.wait_until(20)
    assert lib.ctas() == (152 if fails == 0 else 0)
