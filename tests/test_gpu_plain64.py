"""The FP64 products that keep the plain form (csrc/rpy_bb64.cu: the right-hand
side of the free-body solve, every product of an implicit step) give the sums of
the tile form, which a pinned variant keeps, bit for bit. Tolerance: none."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def sphere(n, radius):
    k = np.arange(n) + 0.5
    phi, z = np.pi * (1.0 + 5.0**0.5) * k, 1.0 - 2.0 * k / n
    s = np.sqrt(1.0 - z * z)
    return radius * np.stack([s * np.cos(phi), s * np.sin(phi), z], -1)


# targets around groups of 16 and 32, sources around stages of 32, tiles of 128
# and chunks of 256; segments near blobs and one another
@pytest.mark.parametrize("nfil,nseg,nb,gap", [(1, 2, 5, 3.0), (2, 16, 16, 3.0), (3, 11, 17, 1.5),
                                             (8, 16, 33, 3.0), (43, 3, 129, 2.0),
                                             (16, 16, 31, 3.0), (19, 27, 200, 1.5)])
def test_rhs_product(nfil, nseg, nb, gap):
    from timfilsimmod_gb300.mobility import RpyMobilitySolver

    rng = np.random.default_rng(nb)
    refs = sphere(nb, gap * max(1.0, (nb / 12.0) ** 0.5))
    ns = nfil * nseg
    xs = rng.uniform(-1, 1, size=(ns, 3)) * (np.abs(refs).max() + ns ** (1 / 3))
    fs = rng.normal(size=(ns, 6))
    out = []
    for variant in (0, 1, 2):
        s = RpyMobilitySolver(1, nfil, nseg, nb, precision="fp64")
        s.set_blob_references(refs)
        s.set_body_pose([0.1, -0.3, 0.7], [1.0, 0.0, 0.0, 0.0])
        s.set_linear_solver(1e-8)
        s.set_queue_variant(1, variant)
        s.x_segs_host[:], s.f_segs_host[:] = xs.ravel(), fs.ravel()
        s.copy_segment_positions_to_device()
        s.copy_segment_forces_to_device()
        s.compute_velocities(np.ones(6))
        out.append(np.concatenate([s.blob_forces().ravel(), s.body_velocities().ravel()]))
        s.finalise()
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])


@pytest.mark.parametrize("nfil,nseg", [(4, 10), (7, 19), (16, 16)])
def test_step_products(nfil, nseg):
    from timfilsimmod_gb300.geometry import elastic_swimmer
    from timfilsimmod_gb300.mobility import RpyMobilitySolver
    from timfilsimmod_gb300.stepper import ImplicitStepper

    blob_refs, fil_refs, fil_dirs, radius = elastic_swimmer(nfil, nseg, 2.2)
    rng = np.random.default_rng(nfil)
    u0 = 1e-3 * rng.normal(size=3 * nfil * nseg)
    out = []
    for variant in (0, 1, 2):
        s = RpyMobilitySolver(1, nfil, nseg, len(blob_refs), "fp64", end_force_magnitude=220)
        s.set_blob_references(blob_refs)
        s.set_linear_solver(1e-8)
        for kind in (2, 3):
            s.set_queue_variant(kind, variant)
        st = ImplicitStepper(s, nfil, nseg, fil_refs, fil_dirs, seg_sep=2.2, dt=1e-3, tol=1e-4,
                             end_force_magnitude=220, body_radius=radius)
        st.reset(u0)
        for nt in range(2):
            st.step(nt)
        g = st.state()
        out.append({k: np.array(g[k]) for k in ("x", "q", "body_x", "body_q", "tether")})
    for k in out[0]:
        assert np.array_equal(out[0][k], out[1][k]) and np.array_equal(out[0][k], out[2][k]), k


def test_autotuned_solver_keeps_the_plain_kernel():
    """Autotuning times the kernels of the fixed-point form; what it picks leaves
    the plain products alone."""
    torch = pytest.importorskip("torch")
    from torch.profiler import ProfilerActivity, profile

    from timfilsimmod_gb300.geometry import elastic_swimmer
    from timfilsimmod_gb300.mobility import RpyMobilitySolver
    from timfilsimmod_gb300.stepper import ImplicitStepper

    for nfil in range(5, 13):
        blob_refs, fil_refs, fil_dirs, radius = elastic_swimmer(nfil, 11, 2.2)
        s = RpyMobilitySolver(1, nfil, 11, len(blob_refs), "fp64", end_force_magnitude=220)
        s.set_blob_references(blob_refs)
        s.set_linear_solver(1e-8)
        st = ImplicitStepper(s, nfil, 11, fil_refs, fil_dirs, seg_sep=2.2, dt=1e-3, tol=1e-4,
                             end_force_magnitude=220, body_radius=radius)
        st.step(0)
        s.autotune(("fp64",), reps=1)
        for nt in (1, 2):  # (the first trace of a process may be empty)
            with profile(activities=[ProfilerActivity.CUDA]) as prof:
                st.step(nt)
                torch.cuda.synchronize()
        names = " ".join(e.name for e in prof.events())
        if "arnoldi" not in names:
            pytest.skip("no kernel trace")
        assert "rpy_plain64_kernel" in names and "rpy_fx_kernel" not in names, nfil
        st.close()
        s.finalise()


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
@pytest.mark.parametrize("nfil,nseg", [(4, 10), (19, 17)])
def test_a_broyden_loop_of_the_caller_gets_the_stepper_s_velocities(precision, nfil, nseg):
    """compute_velocities through the public call, as a program with a Broyden loop
    of its own makes it, and inside the library's implicit step."""
    from timfilsimmod_gb300.geometry import elastic_swimmer
    from timfilsimmod_gb300.mobility import RpyMobilitySolver
    from timfilsimmod_gb300.stepper import ImplicitStepper

    blob_refs, fil_refs, fil_dirs, radius = elastic_swimmer(nfil, nseg, 2.2)
    u0 = 1e-3 * np.random.default_rng(nfil).normal(size=3 * nfil * nseg)
    out = []
    for public in (False, True):
        s = RpyMobilitySolver(1, nfil, nseg, len(blob_refs), precision, end_force_magnitude=220)
        s.set_blob_references(blob_refs)
        s.set_linear_solver(1e-8)
        st = ImplicitStepper(s, nfil, nseg, fil_refs, fil_dirs, seg_sep=2.2, dt=1e-3, tol=1e-4,
                             end_force_magnitude=220, body_radius=radius)
        st.reset(u0)
        st.initial_guess(0)
        f = st.forces_and_torques(0)
        if public:
            g = st.state()
            s.set_body_pose(g["body_x"], g["body_q"])
            s.positions_updated()
            s.compute_velocities(f)
        else:
            st.compute_velocities(0)
        s.copy_segment_velocities_to_host()
        s.wait_for_device()
        out.append([s.v_segs_host.copy(), s.blob_forces().copy(), s.body_velocities().copy()])
        st.close()
        s.finalise()
    for a, b in zip(*out):
        assert np.any(a != 0.0) and np.array_equal(a, b)
