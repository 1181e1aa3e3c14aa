"""The fixed-point far-field pair (csrc/fx_pair.cuh) keeps the exact zeros of
configurations in a plane, as FP64 pairs do. The header compiled for the host,
against the pair formula in long double. Tolerance: none."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = r'''
#include <math.h>
#include "fx_pair.cuh"
using namespace tfs::fx;
typedef long double Q;
// out: the sums (v_t, v_r) of n sources f = (F, T), forces of the unit 2^es;
// ref: in long double, at the positions the records hold
extern "C" void run(int fd, const double *x, const double *y, const double *f, int n, double a,
                    int Ex, int es, const int *below, double *out, double *ref) {
  const int lx = ilogb(0.74 * 2 * a);
  PairFx pc;
  const double b = ldexp(a, -lx), sq = 2 * b * b / 3;
  pc.shift = Ex - lx;
  pc.near_q = (float)(4 * b * b * (1 + 3.8147e-6) * ldexp(1.0, 58 - 2 * pc.shift));
  pc.s = limb_of((i64)rint(ldexp(sq, 61)));
  const Q s = 2 * (Q)a * a / 3;
  Acc v[6] = {};
  Q e[6] = {};
  u64 xw[3], yw[3];
  for (int k = 0; k < 3; ++k) xw[k] = (u64)llrint(ldexp(x[k], 61 - Ex));
  for (int j = 0; j < n; ++j) {
    const double *g = f + j * fd;
    Limb F[3], T[3];
    Q d[3], r2 = 0, dF = 0, dT = 0;
    for (int k = 0; k < 3; ++k) {
      yw[k] = (u64)llrint(ldexp(y[3 * j + k], 61 - Ex));
      F[k] = limb_of(llrint(ldexp(g[k], 62 - es + below[j])));
      if (fd == 6) T[k] = limb_of(llrint(ldexp(g[3 + k], 62 - es + below[j] - lx)));
      d[k] = ((Q)(i64)xw[k] - (Q)(i64)yw[k]) * ldexpl(1, Ex - 61);
      r2 += d[k] * d[k];
      dF += d[k] * g[k];
      if (fd == 6) dT += d[k] * g[3 + k];
    }
    if (fd == 6) PAIR6
    else PAIR3
    const Q r = sqrtl(r2), r3 = r * r2, r5 = r3 * r2;
    for (int k = 0; k < 3; ++k) {
      const int p = (k + 1) % 3, q = (k + 2) % 3;
      e[k] += (1 / r + s / r3) * g[k] + (1 / r3 - 3 * s / r5) * dF * d[k];
      e[3 + k] += (g[p] * d[q] - g[q] * d[p]) / r3;
      if (fd == 6) {
        e[k] += (g[3 + p] * d[q] - g[3 + q] * d[p]) / r3;
        e[3 + k] += -g[3 + k] / (2 * r3) + 1.5L * dT * d[k] / r5;
      }
    }
  }
  for (int k = 0; k < 6; ++k) {
    // words w3 w2 w1 w0 of the unit 2^-91, less n (2^62 + 2^31) of 2^-59
    __int128 t = ((__int128)v[k].w3 << 96) | ((__int128)v[k].w2 << 64) | ((u64)v[k].w1 << 32) | v[k].w0;
    t -= ((__int128)n * ((1ll << 62) + (1ll << 31))) << 32;
    const Q got = (Q)t * ldexpl(1, es - 91 - (k < 3 ? lx : 2 * lx));
    out[k] = (double)(got - e[k]);
    ref[k] = (double)e[k];
  }
}
'''


def build(tmp, below):
    arg = ", below[j]" if below else ""
    text = SOURCE.replace("PAIR6", "far_pair<6, 6>(v, xw, yw, F, T, pc%s);" % arg).replace(
        "PAIR3", "far_pair<6, 3>(v, xw, yw, F, T, pc%s);" % arg)
    src, so = tmp / "fx.cpp", tmp / "fx.so"
    src.write_text(text)
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-std=c++17",
                    "-I", os.path.join(ROOT, "timfilsimmod_gb300", "csrc"), str(src),
                    "-o", str(so)], check=True, capture_output=True)
    return ctypes.CDLL(str(so))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return build(tmp_path_factory.mktemp("fx"), False)


def run(lib, fd, x, y, f, ex, es, a=1.0, below=None):
    x, y, f = (np.ascontiguousarray(v, dtype=np.float64) for v in (x, y, f))
    below = np.ascontiguousarray(np.zeros(len(y)) if below is None else below, dtype=np.int32)
    err, ref = np.zeros(6), np.zeros(6)
    p = ctypes.c_void_p
    lib.run(fd, p(x.ctypes.data), p(y.ctypes.data), p(f.ctypes.data), len(y), ctypes.c_double(a), ex,
            es, p(below.ctypes.data), p(err.ctypes.data), p(ref.ctypes.data))
    return err, ref


def frame(*xs):
    big = max(np.abs(x).max() for x in xs)
    return max(int(np.floor(np.log2(1.7320509 * big))) + 1, 1)


@pytest.mark.parametrize("fd", [6, 3])
def test_a_plane_stays_a_plane(lib, fd):
    """Forces in the plane of the particles (and torques across it) turn nothing
    out of the plane and move nothing across it."""
    rng = np.random.default_rng(4)
    y = np.zeros((400, 3))
    y[:, :2] = 3.0 * np.stack(np.meshgrid(np.arange(20), np.arange(20)), -1).reshape(-1, 2)
    f = np.zeros((400, fd))
    f[:, :2] = rng.normal(size=2)  # alike: nothing averages out
    if fd == 6:
        f[:, 5] = 0.3
    err, ref = run(lib, fd, np.array([-2.5, -2.5, 0.0]), y, f, 7, 3)
    assert np.all(ref[2:5] == 0.0)
    assert np.all(err[2:5] == 0.0)
