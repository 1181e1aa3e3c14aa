"""The fixed-point far-field pair of FP64 products (csrc/fx_pair.cuh) on the
CPU: the header compiled for the host, against the pair formula in long double
and against FP64 sums.

Positions are rounded to 2^(Ex - 61) when a record is made (exact for FP64
coordinates above 2^-9 of the frame); the sums are compared at the rounded
ones.

Tolerances, in last places of the sums, 2^-59 of the largest force over lambda
(units of 1/(8 pi mu)). The coarsest coefficient, kappa/r, is rounded to one
last place, the others to half of one or finer; a component of a pair is four
products of a coefficient and a force that may be at its largest, each with
the errors of the two or three factors its coefficient is made of: at most 8
last places a pair. Over n pairs the roundings are independent: 8 sqrt(n). The
long double reference sums n terms with a relative error of 2^-64 each.
"""
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
static void exact(Q *v, const double *x, const double *y, const double *f, int fd) {
  Q d[3], r2 = 0, dF = 0, dT = 0;
  for (int k = 0; k < 3; ++k) { d[k] = (Q)x[k] - y[k]; r2 += d[k] * d[k]; }
  Q r = sqrtl(r2), r3 = r * r2, r5 = r3 * r2;
  Q s = SQ, A = 1 / r + s / r3, B = 1 / r3 - 3 * s / r5;
  for (int k = 0; k < 3; ++k) { dF += d[k] * f[k]; if (fd == 6) dT += d[k] * f[3 + k]; }
  for (int k = 0; k < 3; ++k) {
    int a = (k + 1) % 3, b = (k + 2) % 3;
    v[k] += A * f[k] + B * dF * d[k];
    v[3 + k] += (f[a] * d[b] - f[b] * d[a]) / r3;
    if (fd == 6) {
      v[k] += (f[3 + a] * d[b] - f[3 + b] * d[a]) / r3;
      v[3 + k] += -f[3 + k] / (2 * r3) + 1.5L * dT * d[k] / r5;
    }
  }
}
static Q read(const Acc &a, unsigned n) {
  // words w3 w2 w1 . w0, less n (2^62 + 2^31)
  __int128 top = ((__int128)a.w3 << 64) | (((u64)a.w2 << 32) | a.w1);
  top -= (__int128)n * ((1ll << 62) + (1ll << 31));
  return (Q)top + (Q)a.w0 / 4294967296.0L;
}
extern "C" int run(int fd, const double *x, const double *y, const double *f, int n, double a_t,
                   double a_s, int Ex, int es, double *out, double *ref, int *left_out) {
  const int lx = ilogb(0.74 * (a_t + a_s));
  PairFx pc;
  const double at = ldexp(a_t, -lx), as = ldexp(a_s, -lx), sq = (at * at + as * as) / 3.0;
  pc.shift = Ex - lx;
  pc.near_q = (float)((at + as) * (at + as) * (1 + 3.8147e-6) * ldexp(1.0, 58 - 2 * pc.shift));
  pc.s = limb_of((i64)rint(ldexp(sq, 61)));
  SQ = (Q)(a_t * a_t + a_s * a_s) / 3;
  Acc v[6] = {};
  Q e[6] = {};
  u64 xw[3], yw[3];
  Limb F[3], T[3];
  for (int k = 0; k < 3; ++k) xw[k] = (u64)llrint(ldexp(x[k], 61 - Ex));
  *left_out = 0;
  for (int j = 0; j < n; ++j) {
    const double *g = f + j * fd;
    for (int k = 0; k < 3; ++k) {
      yw[k] = (u64)llrint(ldexp(y[3 * j + k], 61 - Ex));
      F[k] = limb_of(llrint(ldexp(g[k], 62 - es)));
      if (fd == 6) T[k] = limb_of(llrint(ldexp(g[3 + k], 62 - es - lx)));
    }
    // the pair of the positions as the record holds them
    double xq[3], yq[3];
    for (int k = 0; k < 3; ++k) {
      xq[k] = ldexp((double)(i64)xw[k], Ex - 61);
      yq[k] = ldexp((double)(i64)yw[k], Ex - 61);
    }
    const bool near = fd == 6 ? far_pair<6, 6>(v, xw, yw, F, T, pc) : far_pair<6, 3>(v, xw, yw, F, T, pc);
    if (near) ++*left_out; else exact(e, xq, yq, g, fd);
  }
  for (int k = 0; k < 6; ++k) {
    out[k] = (double)(read(v[k], n) * ldexpl(1, es - 59 - (k < 3 ? lx : 2 * lx)) - e[k]);
    ref[k] = (double)e[k];
  }
  return 0;
}
'''


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("fx")
    src = d / "fx.cpp"
    src.write_text("static long double SQ;\n" + SOURCE)
    so = d / "fx.so"
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-std=c++17", "-x", "c++",
                    "-I", os.path.join(ROOT, "timfilsimmod_gb300", "csrc"), str(src),
                    "-o", str(so)], check=True, capture_output=True)
    return ctypes.CDLL(str(so))


def run(lib, fd, x, y, f, a_t=1.0, a_s=1.0):
    x, y, f = (np.ascontiguousarray(a, dtype=np.float64) for a in (x, y, f))
    lx = int(np.floor(np.log2(0.74 * (a_t + a_s))))
    big = max(np.abs(x).max(), np.abs(y).max())
    ex = max(int(np.floor(np.log2(1.7320509 * big))) + 1, lx + 1)
    fn = np.linalg.norm(f[:, :3], axis=1).max()
    if fd == 6:
        fn = max(fn, np.linalg.norm(f[:, 3:], axis=1).max() * 2.0 ** -lx)
    es = int(np.floor(np.log2(fn * (1 + 1e-6)))) + 1
    assert ex - lx <= 10
    err, ref, left = np.zeros(6), np.zeros(6), ctypes.c_int()
    p = ctypes.c_void_p
    lib.run(fd, p(x.ctypes.data), p(y.ctypes.data), p(f.ctypes.data), len(y),
            ctypes.c_double(a_t), ctypes.c_double(a_s), ex, es, p(err.ctypes.data),
            p(ref.ctypes.data), ctypes.byref(left))
    scale = np.array([2.0 ** (es - lx)] * 3 + [2.0 ** (es - 2 * lx)] * 3)
    return err / scale, ref / scale, left.value


def bound(n, ref):
    return 8 * np.sqrt(n) * 2.0 ** -59 + n * 2.0 ** -64 * np.abs(ref).max()


@pytest.mark.parametrize("fd", [6, 3])
@pytest.mark.parametrize("extent", [3.0, 60.0, 500.0])
@pytest.mark.parametrize("alike", [False, True])
def test_sum_error(lib, fd, extent, alike):
    rng = np.random.default_rng(7)
    n = 4000
    x = rng.uniform(-extent, extent, 3)
    y = rng.uniform(-extent, extent, (n, 3))
    y = y[np.linalg.norm(y - x, axis=1) > 2.001]
    f = rng.normal(size=(len(y), fd))
    if alike:
        f[:] = f[0]
    err, ref, left = run(lib, fd, x, y, f)
    assert left == 0
    assert np.abs(err).max() <= bound(len(y), ref)


@pytest.mark.parametrize("r", [2.0001, 2.2, 7.3, 150.0, 1000.0])
@pytest.mark.parametrize("axis", [0, 1, 2, None])
def test_single_pair(lib, r, axis):
    """One pair, along an axis (unit components at their limit) and not."""
    rng = np.random.default_rng(3)
    u = rng.normal(size=3) if axis is None else np.eye(3)[axis] * (-1) ** axis
    u /= np.linalg.norm(u)
    f = rng.normal(size=(1, 6))
    err, ref, left = run(lib, 6, 0.5 * r * u, -0.5 * r * u[None], f)
    assert left == 0
    assert np.abs(err).max() <= bound(1, ref)


@pytest.mark.parametrize("a_t,a_s", [(1.0, 1.3), (0.26, 0.24), (5.0, 5.0), (1.0, 0.1)])
def test_radii(lib, a_t, a_s):
    rng = np.random.default_rng(5)
    y = rng.uniform(-40 * a_t, 40 * a_t, (500, 3))
    y = y[np.linalg.norm(y, axis=1) > 1.001 * (a_t + a_s)]
    err, ref, left = run(lib, 6, np.zeros(3), y, rng.normal(size=(len(y), 6)), a_t, a_s)
    assert left == 0
    assert np.abs(err).max() <= bound(len(y), ref)


def test_contact_is_left_out(lib):
    """Coincident, overlapping and touching pairs add nothing and are reported."""
    y = np.array([[0.0, 0, 0], [0.3, 0.2, 0.1], [0, 0, 2.0], [0, 1e-9, 0], [0, 0, 2.001]])
    f = np.ones((5, 6))
    err, ref, left = run(lib, 6, np.zeros(3), y, f)
    assert left == 4
    assert np.abs(err).max() <= bound(1, ref)


def test_no_worse_than_fp64(lib):
    """Random forces on a ball of 3000 particles: the error of the fixed-point
    sum is below that of the FP64 sum in the same order."""
    rng = np.random.default_rng(11)
    y = rng.uniform(-50, 50, (3000, 3))
    tot_fx = tot_64 = 0.0
    for k in range(8):
        x = rng.uniform(-50, 50, 3)
        yy = y[np.linalg.norm(y - x, axis=1) > 2.001]
        f = rng.normal(size=(len(yy), 3))
        err, ref, _ = run(lib, 3, x, yy, f)
        es = int(np.floor(np.log2(np.linalg.norm(f, axis=1).max() * (1 + 1e-6)))) + 1
        d = x - yy
        r2 = (d * d).sum(1)
        rm1 = 1.0 / np.sqrt(r2)
        A = rm1 + (2.0 / 3.0) * rm1 / r2
        B = (rm1 / r2 - 2.0 * rm1 / r2 / r2) * (d * f).sum(1)
        v = np.zeros(3)
        for j in range(len(yy)):  # one addition after another, as the FP64 kernel
            v += A[j] * f[j] + B[j] * d[j]
        tot_fx += float((err[:3] ** 2).sum())
        tot_64 += float(((v / 2.0 ** es - ref[:3]) ** 2).sum())
    assert tot_fx <= tot_64
