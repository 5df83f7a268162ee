"""Floquet step of blocks above 8 with the eigenphases spread over the circle (couplings well above
the spinning rate), against the oracle: blocks on both sides of the sizes at which the sweeps start
in single precision (15, 20 and 35), short FIDs (single-precision sweeps in the mixed form) and FIDs
of more than 64 periods (FP64 sweeps in both).

FP64 to 1e-10 and the mixed form to 1e-6 relative L2, the engine's bars."""
import pytest

from helpers import gpu_fid, oracle_fid, rel
from test_gpu_lengths import job_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("npts", [48, 1120])
@pytest.mark.parametrize("nspin", [6, 7])
def test_spread_eigenphases_match_oracle(nspin, npts, precision):
    job, rows = job_of(nspin, 16, seed=7)
    job = job.replace("npts: 60\n", f"npts: {npts}\n")
    ref, _ = oracle_fid(job, rows)
    assert rel(gpu_fid(job, rows, precision=precision), ref) <= (1e-6 if precision else 1e-10)
