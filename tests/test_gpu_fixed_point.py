"""FP64 products in fixed point (csrc/rpy_fx.cu) on the GPU: sizes at the edges
of tiles, blocks and chunks, and data the fixed-point form has to hand to the
FP64 pipe, against the CPU oracle.

Tolerance: 1e-12 of the largest component, the bar of every FP64 product (its
own error is a few 1e-16; the oracle's FP64 sums differ from it by 1e-14)."""
import numpy as np
import pytest

from oracle import Oracle

pytestmark = pytest.mark.gpu
TOL = 1e-12


def system(ns, nb, seed=0, spacing=2.5):
    rng = np.random.default_rng(seed)
    n = ns + nb
    m = int(np.ceil(n ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    x = spacing * (g - 0.5 * m) + rng.uniform(-0.2, 0.2, (n, 3))
    return x[:ns], rng.normal(size=(ns, 6)), x[ns:], rng.normal(size=(nb, 3))


def blocks(xs, fs, xb, fb, a_seg=1.0, a_blob=1.0, variant=None):
    from timfilsimmod_gb300.mobility import RpyMobilitySolver

    s = RpyMobilitySolver(1, len(xs), 1, len(xb), "fp64", a_seg=a_seg, a_blob=a_blob)
    if variant is not None:
        for kind in range(6):
            s.set_queue_variant(kind, variant)
    s.set_state(xs, fs, xb, fb)
    out = []
    s.evaluate_segment_segment_mobility()
    s.evaluate_segment_blob_mobility()
    s.copy_segment_velocities_to_host()
    s.evaluate_blob_blob_mobility()
    s.copy_blob_velocities_to_host()
    s.wait_for_device()
    out += [s.v_segs_host.copy(), s.v_blobs_host.copy()]
    s.evaluate_blob_segment_mobility()
    s.copy_blob_velocities_to_host()
    s.wait_for_device()
    out.append(s.v_blobs_host.copy())
    s.apply_grand_mobility()
    s.copy_segment_velocities_to_host()
    s.copy_blob_velocities_to_host()
    s.wait_for_device()
    out += [s.v_segs_host.copy(), s.v_blobs_host.copy()]
    s.finalise()
    return out


def expected(xs, fs, xb, fb, a_seg=1.0, a_blob=1.0):
    o = Oracle(1.0, a_seg, a_blob)
    vs = o.msb(xs, xb, fb, o.mss(xs, fs)).ravel()
    bb, bs = o.mbb(xb, fb).ravel(), o.mbs(xb, xs, fs).ravel()
    return [vs, bb, bs, vs, bb + bs]


def check(got, want):
    for g, w in zip(got, want):
        if w.size:
            assert np.max(np.abs(g - w)) <= TOL * np.max(np.abs(w))


@pytest.mark.parametrize("ns,nb", [(1, 1), (31, 33), (32, 64), (33, 31), (64, 127), (65, 129),
                                   (128, 32), (129, 1), (1345, 1344), (2049, 700)])
@pytest.mark.parametrize("variant", [0, 1, 2])
def test_sizes(ns, nb, variant):
    d = system(ns, nb)
    check(blocks(*d, variant=variant), expected(*d))


@pytest.mark.parametrize("ns,nb", [(40, 0), (0, 40)])
def test_one_kind(ns, nb):
    d = system(ns, nb)
    check(blocks(*d), expected(*d))


def test_variants_and_repeats_give_the_same_bits():
    d = system(700, 500)
    first = blocks(*d, variant=0)
    for v in (0, 1, 2):
        for a, b in zip(first, blocks(*d, variant=v)):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("shift", [0.0, 50.0, 1e4, -3e6])
def test_away_from_the_origin(shift):
    xs, fs, xb, fb = system(150, 90)
    d = (xs + shift, fs, xb + shift, fb)
    check(blocks(*d), expected(*d))


@pytest.mark.parametrize("spread", [1.0, 60.0, 1e4, 1e8])
def test_extents(spread):
    """Up to 2^10 lambda across in fixed point, beyond it on the FP64 pipe."""
    xs, fs, xb, fb = system(150, 90)
    d = (xs * spread, fs, xb * spread, fb)
    check(blocks(*d), expected(*d))


@pytest.mark.parametrize("scale", [1e-290, 1e-200, 1e-9, 1e9, 1e200])
def test_force_magnitudes(scale):
    xs, fs, xb, fb = system(100, 70)
    d = (xs, fs * scale, xb, fb * scale)
    check(blocks(*d), expected(*d))


def test_uneven_forces():
    """Tiles of very different magnitudes, and a tile without any force."""
    xs, fs, xb, fb = system(200, 160)
    fs[32:64] *= 1e-12
    fs[64:96] = 0.0
    fs[96:128] *= 1e7
    fb[:] = 0.0
    fb[40] = (0.0, 3.0, 0.0)
    check(blocks(xs, fs, xb, fb), expected(xs, fs, xb, fb))


def test_no_forces():
    xs, fs, xb, fb = system(50, 50)
    for v in blocks(xs, 0 * fs, xb, 0 * fb):
        assert np.all(v == 0.0)


@pytest.mark.parametrize("a_seg,a_blob", [(1.0, 0.6), (0.3, 1.0), (1.0, 0.05), (1e-3, 1e-3)])
def test_radii(a_seg, a_blob):
    xs, fs, xb, fb = system(120, 90)
    k = max(a_seg, a_blob)
    d = (xs * k, fs, xb * k, fb)
    check(blocks(*d, a_seg=a_seg, a_blob=a_blob), expected(*d, a_seg=a_seg, a_blob=a_blob))


def test_overlapping_and_touching():
    rng = np.random.default_rng(2)
    xs, xb = rng.uniform(-4, 4, (90, 3)), rng.uniform(-4, 4, (70, 3))
    xs[7] = xs[3]                       # coincident
    xs[9] = xs[8] + (2.0, 0.0, 0.0)     # touching
    xb[5] = xs[1]
    d = (xs, rng.normal(size=(90, 6)), xb, rng.normal(size=(70, 3)))
    check(blocks(*d), expected(*d))


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("where", ["force", "position"])
def test_not_finite(value, where):
    """As the FP64 sums: what the bad particle reaches is not finite."""
    xs, fs, xb, fb = system(80, 40)
    (fs if where == "force" else xs)[50, 1] = value
    got = blocks(xs, fs, xb, fb)
    assert not np.any(np.isfinite(got[0].reshape(-1, 6)[:, 1]))
    assert np.all(np.isfinite(got[1]))  # blob <- blob does not see it


def test_positions_written_on_the_device_without_notice():
    """Positions outside the frame of the last positions_updated."""
    import torch
    from timfilsimmod_gb300.mobility import RpyMobilitySolver

    xs, fs, xb, fb = system(100, 64)
    s = RpyMobilitySolver(1, 100, 1, 64, "fp64")
    view = torch.as_tensor(s.device_arrays()["x_segs"], device="cuda")
    s.set_state(xs, fs, xb, fb)
    s.evaluate_segment_segment_mobility()
    s.wait_for_device()
    view.mul_(3.0)
    torch.cuda.synchronize()
    s.evaluate_segment_segment_mobility()
    s.copy_segment_velocities_to_host()
    s.wait_for_device()
    want = Oracle(1.0, 1.0, 1.0).mss(3.0 * xs, fs).ravel()
    assert np.max(np.abs(s.v_segs_host - want)) <= TOL * np.max(np.abs(want))
    s.finalise()
