"""The fixed-point records of FP64 block products are held by the solvers that run
such products: not by FP32C solvers, nor in a server's budget."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
RECORDS = (9 * 8 + 4, 6 * 8 + 4)  # bytes a segment and a blob: words, exponent


def test_memory_of_a_solver():
    import torch
    from timfilsimmod_gb300.mobility import RpyMobilitySolver

    nseg, nblob = 200000, 30

    def used(precision):
        before = torch.cuda.mem_get_info()[0]
        s = RpyMobilitySolver(1, nseg, 1, nblob, precision)
        n = before - torch.cuda.mem_get_info()[0]
        s.finalise()
        return n

    used("fp64"), used("fp32c")  # what the first solver of a process loads
    extra = used("fp64") - used("fp32c")
    # blocks of 2 MB
    assert abs(extra - nseg * RECORDS[0]) <= 5 * (2 << 20)


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
def test_server_budget(precision):
    """What a blob more takes of a server's budget: its solver's doubles (vectors, 64
    partial sums, Krylov vectors and their scratch) and 200 bytes of records."""
    from timfilsimmod_gb300.geometry import elastic_swimmer
    from timfilsimmod_gb300.serving import StepServer

    blob_refs, fil_refs, fil_dirs, _ = elastic_swimmer(8, 20, 2.2)
    sv = StepServer(num_workers=1, precision=precision)
    n = [sv.request_bytes(blob_refs[:k], fil_refs, fil_dirs, 20) for k in (300, 400)]
    sv.close()

    def doubles(nb):
        rows, m = 3 * nb + 6, 350
        return 12 * nb + 64 * 3 * nb + rows * (m + 1) + 16 * rows + 57 * nb

    assert n[1] - n[0] == 8 * (doubles(400) - doubles(300)) + 200 * 100


@pytest.mark.parametrize("created", ["fp32c", "fp64"])
def test_precision_set_later(created):
    """A solver that becomes FP64 computes what one created so does, bit for bit."""
    from timfilsimmod_gb300.mobility import RpyMobilitySolver

    rng = np.random.default_rng(3)
    x = 3.0 * np.stack(np.meshgrid(*[np.arange(8.0)] * 3), -1).reshape(-1, 3)
    xs, xb, fs, fb = x[::2], x[1::2], rng.normal(size=(256, 6)), rng.normal(size=(256, 3))
    out = []
    for first in ("fp64", created):
        s = RpyMobilitySolver(1, 256, 1, 256, first)
        s.set_state(xs, fs, xb, fb)
        s.apply_grand_mobility()
        s.set_precision("fp32c")
        s.apply_grand_mobility()
        s.set_precision("fp64")
        s.apply_grand_mobility()
        s.copy_segment_velocities_to_host()
        s.copy_blob_velocities_to_host()
        s.wait_for_device()
        out.append(np.concatenate([s.v_segs_host, s.v_blobs_host]))
        s.finalise()
    assert np.any(out[0] != 0.0) and np.array_equal(out[0], out[1])
