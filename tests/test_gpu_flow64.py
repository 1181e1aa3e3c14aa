"""FP64 flow fields with the pair products on the integer pipe (csrc/
flow_kernels.cuh, taken where the points fill the SMs) against the same points
alone, which run without.

Tolerance: 1e-12 of the largest component, the bar of the FP64 flow; only the
source splits' order may differ."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nseg,nblob", [(1, 0), (130, 0), (63, 5), (129, 257), (1, 1500)])
@pytest.mark.parametrize("zero", [False, True])
def test_same_as_alone(nseg, nblob, zero):
    from timfilsimmod_gb300.flow_field import FlowFieldEvaluator

    rng = np.random.default_rng(nseg + nblob)
    xs, fs = rng.uniform(-20, 20, (nseg, 3)), rng.normal(size=(nseg, 6))
    xb, fb = rng.uniform(-20, 20, (nblob, 3)), rng.normal(size=(nblob, 3))
    xs[:, 2] += 25.0  # above the wall of the form without blobs
    if zero:  # zeros in the products
        fs[::2, 1:5] = 0.0
        fb[::3] = 0.0
    many = rng.uniform(-30, 30, (80000, 3)) + (0.0, 0.0, 31.0)
    if nblob:
        many[5, :2] = xb[0, :2]  # two components of the separation zero
    few = many[:100]
    out = []
    for p in (many, few):
        e = FlowFieldEvaluator(1, nseg, 1, nblob, len(p), precision="fp64")
        e.read_positions_and_forces(p, xs, fs, xb, fb, np.zeros(3))
        e.velocities()
        e.wait()
        out.append(e.v_flow_host.reshape(-1, 3)[:100].copy())
        e.close()
    assert np.abs(out[0] - out[1]).max() <= 1e-12 * np.abs(out[1]).max()


@pytest.mark.parametrize("nseg,nblob", [(1, 0), (100, 0), (63, 5), (70, 57), (1, 126)])
def test_same_bits_with_one_split(nseg, nblob):
    """Fewer than 128 sources are one split whatever the points: the same points
    with and without the integer products, bit for bit."""
    from timfilsimmod_gb300.flow_field import FlowFieldEvaluator

    rng = np.random.default_rng(nseg + nblob)
    xs, fs = rng.uniform(-20, 20, (nseg, 3)), rng.normal(size=(nseg, 6))
    xb, fb = rng.uniform(-20, 20, (nblob, 3)), rng.normal(size=(nblob, 3))
    xs[:, 2] += 25.0
    fs[::2, 1:5] = 0.0
    many = rng.uniform(-30, 30, (80000, 3)) + (0.0, 0.0, 31.0)
    out = []
    for p in (many, many[:100]):
        e = FlowFieldEvaluator(1, nseg, 1, nblob, len(p), precision="fp64")
        e.read_positions_and_forces(p, xs, fs, xb, fb, np.zeros(3))
        e.velocities()
        e.wait()
        out.append(e.v_flow_host.reshape(-1, 3)[:100].copy())
        e.close()
    assert np.any(out[0] != 0.0) and np.array_equal(out[0], out[1])
