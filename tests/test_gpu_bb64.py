"""The FP64 blob-blob product of the free-body GMRES (csrc/rpy_bb64.cu) gives
the sums of the tile kernel it stands for bit for bit: same splits, same order
of far and near pairs. Tolerance: none, the solutions are equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def sphere(n, radius):
    k = np.arange(n) + 0.5
    phi, z = np.pi * (1.0 + 5.0**0.5) * k, 1.0 - 2.0 * k / n
    s = np.sqrt(1.0 - z * z)
    return radius * np.stack([s * np.cos(phi), s * np.sin(phi), z], -1)


# gap: spacing of the blobs in radii (below 2 they overlap)
@pytest.mark.parametrize("nb,gap", [(2, 3.0), (31, 3.0), (33, 1.5), (64, 3.0), (127, 1.2),
                                    (128, 3.0), (129, 2.0), (300, 1.5), (642, 3.0), (1290, 3.0)])
def test_same_bits_as_the_tile_kernel(nb, gap):
    from timfilsimmod_gb300.mobility import RpyMobilitySolver

    rng = np.random.default_rng(nb)
    refs = sphere(nb, gap * max(1.0, (nb / 12.0) ** 0.5))
    xs = 3.0 * np.abs(refs).max() + 5.0 * rng.uniform(size=(24, 3)) * np.arange(1, 25)[:, None]
    fs = rng.normal(size=(24, 6))
    out = {}
    for variant in (0, 1):  # 0: rpy_bb64_kernel, 1: rpy_tile_kernel
        s = RpyMobilitySolver(1, 2, 12, nb, precision="fp64")
        s.set_blob_references(refs)
        s.set_body_pose([0.1, -0.3, 0.7], [1.0, 0.0, 0.0, 0.0])
        s.set_linear_solver(1e-8)
        s.set_tuning(2, variant)
        s.x_segs_host[:], s.f_segs_host[:] = xs.ravel(), fs.ravel()
        s.copy_segment_positions_to_device()
        s.copy_segment_forces_to_device()
        iters, _ = s.compute_velocities(np.ones(6))
        out[variant] = (iters, s.blob_forces(), s.body_velocities())
        s.finalise()
    assert out[0][0] == out[1][0] and out[0][0] > 0
    assert np.array_equal(out[0][1], out[1][1])
    assert np.array_equal(out[0][2], out[1][2])
