"""Integer-pipe FP64 products (csrc/soft_mul.cuh), compiled for the host: the
bits of the FP64 multiplication wherever the function says so, and it says so
for every pair of normal numbers with a normal product."""
import os
import shutil
import subprocess
import tempfile

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "timfilsimmod_gb300", "csrc")
CODE = r"""
#include <cmath>
#include <cstdio>
#include "soft_mul.cuh"
static uint64_t st = 0x9e3779b97f4a7c15ull;
static uint64_t rnd() { st ^= st << 13; st ^= st >> 7; st ^= st << 17; return st; }
static double make(uint64_t u) { double x; memcpy(&x, &u, 8); return x; }
static uint64_t bits(double x) { uint64_t u; memcpy(&u, &x, 8); return u; }
int main() {
  long bad = 0, refused = 0, wrongly = 0, n = 0;
  const uint64_t sig[] = {0, 1, 2, 0xfffffffffffffull, 0xffffffffffffeull, 0x8000000000000ull,
                          0x7ffffffffffffull, 0x8000000000001ull, 0xfffff00000000ull, 0xffffffffull,
                          0x100000000ull, 0x6a09e667f3bcdull, 0x6a09e667f3bccull};
  auto check = [&](double a, double b) {
    bool ok = true;
    const double p = tfs::soft::mul(a, b, &ok), q = a * b;
    ++n;
    if (!ok) {
      ++refused;
      const bool normal = std::isnormal(a) && std::isnormal(b) && std::isnormal(q) &&
                          std::fabs(q) < 0x1p1023 && std::fabs(q) > 0x1p-1022;
      if (normal) ++wrongly;
    } else if (bits(p) != bits(q)) {
      if (bad++ < 5) std::printf("%a * %a = %a, got %a\n", a, b, q, p);
    }
  };
  for (uint64_t x : sig)
    for (uint64_t y : sig)
      for (int e = 0; e < 2048; e += (e < 4 || e > 2043) ? 1 : 37)
        for (int f = 0; f < 2048; f += (f < 4 || f > 2043) ? 1 : 41)
          check(make(((uint64_t)e << 52) | x), make((1ull << 63) | ((uint64_t)f << 52) | y));
  for (long i = 0; i < 20000000; ++i) {
    uint64_t a = rnd(), b = rnd();
    if (i & 1) {  // moderate exponents, and products close to a tie
      a = (a & 0x800fffffffffffffull) | ((1023ull + a % 40 - 20) << 52);
      b = (b & 0x800fffffffffffffull) | ((1023ull + b % 40 - 20) << 52);
      if (i & 2) a &= ~((1ull << (rnd() % 40)) - 1);
      if (i & 4) b &= ~((1ull << (rnd() % 40)) - 1);
    }
    check(make(a), make(b));
  }
  std::printf("%ld products, %ld refused\n", n, refused);
  return bad == 0 && wrongly == 0 ? 0 : 1;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_bits_of_the_product():
    with tempfile.TemporaryDirectory() as d:
        src = os.path.join(d, "t.cpp")
        with open(src, "w") as f:
            f.write(CODE)
        exe = os.path.join(d, "t")
        subprocess.run(["g++", "-O2", "-std=c++17", "-I", CSRC, src, "-o", exe], check=True)
        r = subprocess.run([exe], capture_output=True, text=True)
        assert r.returncode == 0, r.stdout
