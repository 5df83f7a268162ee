"""FP64 batches of more crystallites than a launch's grid has rows (65535): six like spins, whose
blocks of 20 go through the batched products.  One batch against batches forced by a memory budget,
bit for bit, and one of the orientations by itself."""
import numpy as np
import pytest

import blochlib_gb300 as bl
from helpers import gpu_fid, rel
from test_gpu_lengths import job_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps", [11, 18])  # one Dyson segment, two
def test_one_batch_beyond_65535_crystallites(steps):
    torch = pytest.importorskip("torch")
    count = 65568
    job, rows = job_of(6, steps)
    job = job.replace("npts: 60\n", "npts: 40\n")
    small = bl.Context(0, hbm_budget=32 << 30)
    if torch.cuda.mem_get_info()[0] < 150e9:
        pytest.skip("needs about 90 GB of device memory")
    many = np.tile(rows, (count // 3, 1))
    many[:, 3] /= count
    ctx = bl.Context(0, hbm_budget=140 << 30)
    one = gpu_fid(job, many, ctx=ctx)
    ctx.close()
    two = gpu_fid(job, many, ctx=small)
    np.testing.assert_array_equal(one, two)
    assert rel(one * count / (count // 3), gpu_fid(job, rows)) <= 1e-12
