"""FP32C pair sums and flow fields on packed FP32x2 instructions
(csrc/rpy_pair2.cuh, csrc/flow_kernels.cuh): odd source counts, chunks smaller
than a tile, single particles, against the CPU oracle.

Tolerance: 2e-5 of the 2-norm, the bar of every FP32C product (FP32 pairs:
each term to about 4e-7)."""
import numpy as np
import pytest

from oracle import Oracle

pytestmark = pytest.mark.gpu
TOL = 2e-5


def rel(a, b):
    a, b = np.asarray(a).ravel(), np.asarray(b).ravel()
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


def system(ns, nb, seed=0):
    rng = np.random.default_rng(seed)
    n = ns + nb
    m = int(np.ceil(n ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    x = 2.5 * (g - 0.5 * m) + rng.uniform(-0.2, 0.2, (n, 3))
    return x[:ns], rng.normal(size=(ns, 6)), x[ns:], rng.normal(size=(nb, 3))


@pytest.mark.parametrize("ns,nb", [(1, 1), (2, 1), (31, 33), (33, 32), (65, 255), (129, 257),
                                   (257, 127), (1025, 301)])
@pytest.mark.parametrize("variant", [0, 1, 2, 3, 4])
def test_products(ns, nb, variant):
    from timfilsimmod_gb300.mobility import RpyMobilitySolver

    xs, fs, xb, fb = system(ns, nb)
    s = RpyMobilitySolver(1, ns, 1, nb, "fp32c")
    for kind in range(6):
        s.set_queue_variant(kind, variant)
    s.set_state(xs, fs, xb, fb)
    o = Oracle(1.0, 1.0, 1.0)
    s.evaluate_segment_segment_mobility()
    s.evaluate_segment_blob_mobility()
    s.copy_segment_velocities_to_host()
    s.evaluate_blob_blob_mobility()
    s.copy_blob_velocities_to_host()
    s.wait_for_device()
    vs = o.msb(xs, xb, fb, o.mss(xs, fs))
    bb, bs = o.mbb(xb, fb).ravel(), o.mbs(xb, xs, fs).ravel()
    assert rel(s.v_segs_host, vs) <= TOL
    assert rel(s.v_blobs_host, bb) <= TOL
    s.apply_grand_mobility()
    s.copy_segment_velocities_to_host()
    s.copy_blob_velocities_to_host()
    s.wait_for_device()
    assert rel(s.v_segs_host, vs) <= TOL
    assert rel(s.v_blobs_host, bb + bs) <= TOL
    s.finalise()


def test_overlapping_and_touching():
    from timfilsimmod_gb300.mobility import RpyMobilitySolver

    rng = np.random.default_rng(2)
    xs = rng.uniform(-4, 4, (91, 3))
    xs[7] = xs[3]
    xs[9] = xs[8] + (2.0, 0.0, 0.0)
    fs = rng.normal(size=(91, 6))
    s = RpyMobilitySolver(1, 91, 1, 0, "fp32c")
    s.set_state(xs, fs, np.zeros((0, 3)), np.zeros((0, 3)))
    s.evaluate_segment_segment_mobility()
    s.copy_segment_velocities_to_host()
    s.wait_for_device()
    assert rel(s.v_segs_host, Oracle(1.0, 1.0, 1.0).mss(xs, fs)) <= TOL
    s.finalise()


@pytest.mark.parametrize("points", [1, 255, 257, 80000])
@pytest.mark.parametrize("nseg,nblob", [(1, 0), (63, 0), (65, 1), (257, 130), (1, 511)])
def test_flow(points, nseg, nblob):
    from timfilsimmod_gb300.flow_field import FlowFieldEvaluator

    rng = np.random.default_rng(points + nseg)
    xs, fs = rng.uniform(-20, 20, (nseg, 3)), rng.normal(size=(nseg, 6))
    xb, fb = rng.uniform(-20, 20, (nblob, 3)), rng.normal(size=(nblob, 3))
    xs[:, 2] += 25.0  # above the wall of the form without blobs
    p = rng.uniform(-30, 30, (points, 3)) + (0.0, 0.0, 31.0)
    ev = {k: FlowFieldEvaluator(1, nseg, 1, nblob, points, precision=k) for k in ("fp64", "fp32c")}
    v = {}
    for k, e in ev.items():  # the FP64 form has the oracle's parity (test_gpu_flow.py)
        e.read_positions_and_forces(p, xs, fs, xb, fb, np.zeros(3))
        v[k] = e.velocities().copy()
        e.wait()
        v[k] = e.v_flow_host.copy()
        e.close()
    assert rel(v["fp32c"], v["fp64"]) <= TOL
