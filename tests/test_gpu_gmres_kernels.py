"""The Arnoldi kernels of the free-body GMRES (csrc/gmres.cu; FP32C: the
cooperative kernel of csrc/gmres_persistent.cu) against a dense FP64 solve, at slices of one blob and of many, and at Krylov spaces below and
above one group (16) and one pass (64) of columns.

Tolerances: the solve stops at 1e-10 of ||rhs||. Blob forces within 1e-8 (spaced
blobs: condition of order 10), the bar of the other FP64 solves; overlapping
ones are ill-conditioned, so there it is the residual that is checked, within
1e-8 (FP32C, refined to 1e-8: 2e-8). 27 000 blobs (slices longer than the rows kept in shared memory): the
residual that three columns leave is the estimate, within 1e-6."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def sphere(n, radius):
    k = np.arange(n) + 0.5
    phi, z = np.pi * (1.0 + 5.0**0.5) * k, 1.0 - 2.0 * k / n
    s = np.sqrt(1.0 - z * z)
    return radius * np.stack([s * np.cos(phi), s * np.sin(phi), z], -1)


def dense(refs):
    """[M_bb, -K; -K^T, 0] for unit spheres in unit viscosity."""
    nb = len(refs)
    d = refs[:, None] - refs[None]
    r2 = np.maximum((d * d).sum(-1), 1e-30)
    r = np.sqrt(r2)
    far = r > 2.0
    A = np.where(far, (1.0 + 2.0 / (3.0 * r2)) / r, 4.0 / 3.0 - 0.375 * r)
    B = np.where(far, (1.0 - 2.0 / r2) / (r2 * r), 0.125 / r)
    M = np.einsum("ij,kl->ikjl", A, np.eye(3)) + np.einsum("ij,ijk,ijl->ikjl", B, d, d)
    K = np.zeros((nb, 3, 6))  # U + Omega x d
    K[:, :, :3] = np.eye(3)
    for j, e in enumerate(np.eye(3)):
        K[:, :, 3 + j] = np.cross(e, refs)
    K = K.reshape(3 * nb, 6)
    return np.block([[M.reshape(3 * nb, 3 * nb) / (8 * np.pi), -K], [-K.T, np.zeros((6, 6))]])


def solver(refs, tol, cols, precision="fp64"):
    from timfilsimmod_gb300.mobility import RpyMobilitySolver

    s = RpyMobilitySolver(1, 2, 12, len(refs), precision=precision)
    s.set_blob_references(refs)
    s.set_body_pose([0.1, -0.3, 0.7], [1.0, 0.0, 0.0, 0.0])
    s.set_linear_solver(tol, cols)
    return s


@pytest.mark.parametrize("nb", [4, 31, 32, 33, 65, 300, 642])
def test_forces(nb):
    refs = sphere(nb, 3.0 * max(1.0, (nb / 12.0) ** 0.5))
    rhs = np.random.default_rng(nb).normal(size=3 * nb + 6)
    s = solver(refs, 1e-10, min(350, 3 * nb + 6))
    s.solve_linear_system(rhs)
    x = np.linalg.solve(dense(refs), rhs)[:3 * nb]
    assert np.linalg.norm(s.blob_forces().ravel() - x) <= 1e-8 * np.linalg.norm(x)
    s.finalise()


@pytest.mark.parametrize("gap", [1.0, 1.3, 2.0])
def test_many_columns(gap):
    refs = sphere(300, gap * 5.0)
    rhs = np.random.default_rng(7).normal(size=906)
    s = solver(refs, 1e-10, 350)
    iters = s.solve_linear_system(rhs)
    x = np.concatenate([s.blob_forces().ravel(), s.body_velocities().ravel()])
    s.finalise()
    assert iters > 16
    assert np.linalg.norm(rhs - dense(refs) @ x) <= 1e-8 * np.linalg.norm(rhs)


@pytest.mark.parametrize("nb,gap", [(3, 3.0), (65, 1.5), (257, 2.0), (642, 1.0), (642, 0.8)])
def test_cooperative_kernel(nb, gap):
    refs = sphere(nb, gap * max(1.0, (nb / 12.0) ** 0.5))
    rhs = np.random.default_rng(nb).normal(size=3 * nb + 6)
    s = solver(refs, 1e-8, min(350, 3 * nb + 6), "fp32c")
    s.set_persistent_gmres(True)
    s.set_refinement_vectors("fp64")  # FP32 vectors can't take these body rows
    s.solve_linear_system(rhs)
    x = np.concatenate([s.blob_forces().ravel(), s.body_velocities().ravel()])
    s.finalise()
    assert np.linalg.norm(rhs - dense(refs) @ x) <= 2e-8 * np.linalg.norm(rhs)


def test_long_slices():
    nb = 27000
    refs = sphere(nb, 3.0 * (nb / 12.0) ** 0.5)
    s = solver(refs, 1e-300, 3)
    lam0 = np.random.default_rng(3).normal(size=(nb, 3))

    def mbb(f):  # by the product entry point
        s.set_state(np.full((24, 3), 1e4) + np.arange(24)[:, None] * 5.0, np.zeros((24, 6)),
                    refs + np.array([0.1, -0.3, 0.7]), f)
        s.evaluate_blob_blob_mobility()
        s.copy_blob_velocities_to_host()
        s.wait_for_device()
        return s.v_blobs_host.reshape(-1, 3).copy()

    rhs = np.concatenate([mbb(lam0).ravel(), -lam0.sum(0), -np.cross(refs, lam0).sum(0)])
    s.set_state(np.full((24, 3), 1e4), np.zeros((24, 6)), refs, np.zeros((nb, 3)))
    assert s.solve_linear_system(rhs) == 3
    lam, vel = s.blob_forces().reshape(-1, 3), s.body_velocities().ravel()
    est = s.solve_info()["rel_residual"]
    v = mbb(lam)
    s.finalise()
    a = np.concatenate([(v - vel[:3] - np.cross(vel[3:], refs)).ravel(), -lam.sum(0),
                        -np.cross(refs, lam).sum(0)])
    assert abs(np.linalg.norm(rhs - a) / np.linalg.norm(rhs) - est) <= 1e-6
