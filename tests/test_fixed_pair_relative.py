"""The fixed-point far-field pair (csrc/fx_pair.cuh) keeps the relative accuracy
of an FP64 pair at every distance, for each coupling by itself, and the exact
zeros of configurations in a plane. The header compiled for the host, against
the pair formula in long double.

Tolerance: 2^-51 of the 2-norm of the pair's contribution, two last places of
FP64. An FP64 pair is a chain of some eight roundings of 2^-53. In fixed point
the factors of a coefficient and the coefficient itself are rounded to 2^-59 or
finer against at least 1/8 (1/r^3 in [1/8, 1) of its power of two), the unit
vector to 2^-62, and the reciprocal square root's series is cut at 2^-55: about
ten errors of 2^-55."""
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
    if (fd == 6) far_pair<6, 6>(v, xw, yw, F, T, pc, below[j]);
    else far_pair<6, 3>(v, xw, yw, F, T, pc, below[j]);
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


def build(tmp):
    src, so = tmp / "fx.cpp", tmp / "fx.so"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-std=c++17",
                    "-I", os.path.join(ROOT, "timfilsimmod_gb300", "csrc"), str(src),
                    "-o", str(so)], check=True, capture_output=True)
    return ctypes.CDLL(str(so))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return build(tmp_path_factory.mktemp("fx"))


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


@pytest.mark.parametrize("r", [2.0001, 2.9, 7.3, 50.0, 100.0, 300.0, 1000.0])
@pytest.mark.parametrize("fd,kind", [(6, "force"), (6, "torque"), (3, "force")])
def test_relative_error_of_a_pair(lib, r, fd, kind):
    """One source with a force or a torque alone: the velocity and the angular
    velocity each against their own size."""
    rng = np.random.default_rng(int(10 * r))
    for _ in range(200):
        u, g = rng.normal(size=3), rng.normal(size=3)
        u /= np.linalg.norm(u)
        g /= np.linalg.norm(g) * (1 + 1e-6)
        f = np.zeros((1, fd))
        f[0, :3 if kind == "force" else 6][-3:] = g
        x, y = 0.5 * r * u, -0.5 * r * u[None]
        err, ref = run(lib, fd, x, y, f, frame(x, y), 0)
        for part in (slice(0, 3), slice(3, 6)):
            assert np.linalg.norm(err[part]) <= 2.0 ** -51 * np.linalg.norm(ref[part])


@pytest.mark.parametrize("below", [1, 5, 9])
@pytest.mark.parametrize("r", [2.2, 100.0])
def test_a_source_below_the_largest(lib, r, below):
    """A source 2^below smaller than the sums' unit has all its places."""
    rng = np.random.default_rng(below)
    for _ in range(100):
        u, f = rng.normal(size=3), rng.normal(size=(1, 6))
        u /= np.linalg.norm(u)
        f *= 2.0 ** -below / np.linalg.norm(f) / (1 + 1e-6)
        x, y = 0.5 * r * u, -0.5 * r * u[None]
        err, ref = run(lib, 6, x, y, f, frame(x, y), 0, below=[below])
        for part in (slice(0, 3), slice(3, 6)):
            assert np.linalg.norm(err[part]) <= 2.0 ** -51 * np.linalg.norm(ref[part])


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
