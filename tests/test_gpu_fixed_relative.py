"""FP64 products in fixed point (csrc/rpy_fx.cu) on the GPU, where the size of a
result is far below that of the largest force over lambda."""
import numpy as np
import pytest

from oracle import Oracle

pytestmark = pytest.mark.gpu
Q = np.longdouble


def pair(x, y, f, t=None, a=1.0, mu=1.0):
    """Velocity and angular velocity at x of one source, far field, long double."""
    d = np.asarray(x, Q) - np.asarray(y, Q)
    f = np.asarray(f, Q)
    r2 = (d * d).sum(-1, keepdims=True)
    r, s = np.sqrt(r2), 2 * Q(a) * a / 3
    vt = (1 / r + s / r**3) * f + (1 / r**3 - 3 * s / r**5) * (d * f).sum(-1, keepdims=True) * d
    vr = np.cross(np.broadcast_to(f, d.shape), d) / r**3
    if t is not None:
        t = np.asarray(t, Q)
        vt = vt + np.cross(np.broadcast_to(t, d.shape), d) / r**3
        vr = vr - t / (2 * r**3) + Q(1.5) * (d * t).sum(-1, keepdims=True) * d / r**5
    k = 8 * Q("3.14159265358979323846264338327950288") * Q(mu)
    return vt / k, vr / k


def each_close(got, want, tol):
    """Every row of got within tol of its own size."""
    err = np.sqrt(((got - want) ** 2).sum(-1).astype(float))
    assert np.all(err <= tol * np.sqrt((want**2).sum(-1).astype(float)))


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


def line(n):
    """n particles from 2.5 to 900 radii off the origin, in all directions."""
    rng = np.random.default_rng(n)
    u = rng.normal(size=(n, 3))
    r = 2.5 * 360.0 ** np.linspace(0, 1, n)[:, None]
    return 0.5 * r * u / np.linalg.norm(u, axis=1, keepdims=True) - (0.3, 0.0, 0.1)


# Positions are held to 2^(Ex - 62) = 2^-52 in a frame of 2^10 radii: 2^-51.5 of 2.5 radii,
# times four in 1/r^3 and its direction; the pair 2^-51 and the result 2^-52 beside.
TOL = 2.0 ** -49


@pytest.mark.parametrize("kind", ["force", "torque"])
def test_one_loaded_segment(kind):
    """A column of the mobility: every other particle's velocity and angular
    velocity against its own size, in the same launch as the loaded one's."""
    xs, xb = line(70), line(50)[1:] + 0.4
    xs[40] = 0.0
    xb = xb[np.linalg.norm(xb, axis=1) > 2.01]
    fs = np.zeros((70, 6))
    fs[40, :3 if kind == "force" else 6][-3:] = (0.3, -1.0, 0.7)
    ss, bs, _, _ = products(xs, fs, xb, np.zeros((len(xb), 3)))
    far = np.linalg.norm(xs, axis=1) > 2.01
    vt, vr = pair(xs[far], xs[40], fs[40, :3], fs[40, 3:])
    each_close(ss[far, :3], vt, TOL)
    each_close(ss[far, 3:], vr, TOL)
    each_close(bs, pair(xb, xs[40], fs[40, :3], fs[40, 3:])[0], TOL)


def test_one_loaded_blob():
    xs, xb = line(70), line(50)
    xb[7] = 0.0
    fb = np.zeros((50, 3))
    fb[7] = (0.3, -1.0, 0.7)
    _, _, sb, bb = products(xs, np.zeros((70, 6)), xb, fb)
    far = np.linalg.norm(xs, axis=1) > 2.01
    vt, vr = pair(xs[far], xb[7], fb[7])
    each_close(sb[far, :3], vt, TOL)
    each_close(sb[far, 3:], vr, TOL)
    far = np.linalg.norm(xb, axis=1) > 2.01
    each_close(bb[far], pair(xb[far], xb[7], fb[7])[0], TOL)


def test_small_forces_beside_a_large_one():
    """One force at 800 radii, the others 2^-20 of it: each target against the
    terms it is the sum of."""
    rng = np.random.default_rng(9)
    xs = 4.0 * np.stack(np.meshgrid(*[np.arange(5.0)] * 3), -1).reshape(-1, 3)
    xs = np.vstack([xs + rng.uniform(-0.5, 0.5, xs.shape), [[460.0, 460.0, 460.0]]])
    fs = 2.0 ** -20 * rng.normal(size=(126, 6))
    fs[125] = rng.normal(size=6)
    ss, _, _, _ = products(xs, fs, np.array([[30.0, 0.0, 0.0]]), np.zeros((1, 3)))
    for i in range(125):
        o = np.arange(126) != i
        vt, vr = pair(xs[i], xs[o], fs[o, :3], fs[o, 3:])
        k = 8 * np.pi
        for got, v, own in ((ss[i, :3], vt, 4.0 / 3.0 * fs[i, :3] / k),
                            (ss[i, 3:], vr, fs[i, 3:] / k)):
            size = np.sqrt((v**2).sum(-1)).sum() + np.linalg.norm(own)
            assert np.linalg.norm((got - (v.sum(0) + own)).astype(float)) <= TOL * size


@pytest.mark.parametrize("length,force", [(1e14, 1e-264), (1e-14, 1e258), (1e14, 1e258),
                                          (1e-14, 1e-258), (1e5, 1e-238), (1e-5, 1e240)])
def test_exponents_of_lengths_and_forces(length, force):
    """Lengths and forces whose exponents add up; the bar of every FP64 product."""
    from timfilsimmod_gb300.mobility import RpyMobilitySolver

    rng = np.random.default_rng(1)
    x = 2.5 * np.stack(np.meshgrid(*[np.arange(4.0)] * 3), -1).reshape(-1, 3)
    f = rng.normal(size=(64, 6))
    f[:, 3:] *= length  # F L and T of a size
    s = RpyMobilitySolver(1, 64, 1, 0, "fp64", a_seg=length, a_blob=length)
    s.set_state(length * x, force * f, np.zeros((0, 3)), np.zeros((0, 3)))
    s.evaluate_segment_segment_mobility()
    s.copy_segment_velocities_to_host()
    s.wait_for_device()
    got = s.v_segs_host.reshape(-1, 6).copy()
    s.finalise()
    f[:, 3:] /= length
    want = Oracle(1.0, 1.0, 1.0).mss(x, f).reshape(-1, 6)
    got[:, :3] *= length
    got[:, 3:] *= length
    got[:, 3:] *= length
    got = got / force
    assert np.max(np.abs(got - want)) <= 1e-12 * np.max(np.abs(want))
