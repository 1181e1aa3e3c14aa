"""FP64 products in fixed point (csrc/rpy_fx.cu) on the GPU, where the size of a
result is far below that of the largest force over lambda."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def products(xs, fs, xb, fb):
    """M_ss f, M_sb f_b (alone), M_bs f, M_bb f_b."""
    from timfilsimmod_gb300.mobility import RpyMobilitySolver

    s = RpyMobilitySolver(1, len(xs), 1, len(xb), "fp64")
    out = []
    s.set_state(xs, fs, xb, fb)
    s.evaluate_segment_segment_mobility()
    s.copy_segment_velocities_to_host()
    s.evaluate_blob_segment_mobility()
    s.copy_blob_velocities_to_host()
    s.wait_for_device()
    out += [s.v_segs_host.reshape(-1, 6).copy(), s.v_blobs_host.reshape(-1, 3).copy()]
    s.set_state(xs, 0.0 * np.asarray(fs), xb, fb)
    s.evaluate_segment_segment_mobility()
    s.evaluate_segment_blob_mobility()
    s.copy_segment_velocities_to_host()
    s.evaluate_blob_blob_mobility()
    s.copy_blob_velocities_to_host()
    s.wait_for_device()
    out += [s.v_segs_host.reshape(-1, 6).copy(), s.v_blobs_host.reshape(-1, 3).copy()]
    s.finalise()
    return out


def test_a_plane_stays_a_plane():
    """Particles, forces and torques that keep to z = 0: no motion across it and no
    turn out of it, exactly."""
    rng = np.random.default_rng(8)
    g = np.stack(np.meshgrid(np.arange(40), np.arange(40)), -1).reshape(-1, 2) * 2.5
    x = np.zeros((1600, 3))
    x[:, :2] = g + rng.uniform(-0.6, 0.6, g.shape)  # some pairs overlap
    xs, xb = x[::2], x[1::2]
    fs, fb = np.zeros((len(xs), 6)), np.zeros((len(xb), 3))
    fs[:, :2], fs[:, 5], fb[:, :2] = rng.normal(size=2), 0.3, rng.normal(size=2)
    ss, bs, sb, bb = products(xs, fs, xb, fb)
    assert np.all(ss[:, 2:5] == 0.0) and np.all(sb[:, 2:5] == 0.0)
    assert np.all(bs[:, 2] == 0.0) and np.all(bb[:, 2] == 0.0)
    for v in (ss, bs, sb, bb):
        assert np.all(v[:, :2] != 0.0)
