"""The FP64 form's FID terms (paired powers) at the edges of their tiles, against the oracle:
one and two periods, odd and even period counts, points short of a period, step counts that do not divide the
tile width.  Tolerance 1e-10 relative L2, the engine's FP64 bar; static and point-to-point
FIDs share the kernel."""
import numpy as np
import pytest

from helpers import gpu_fid, oracle_fid, rel

pytestmark = pytest.mark.gpu
SPIN = ("spin: numspin 2\nspin: T 1H 0\nspin: T 1H 1\nspin: C 0 3000 0.4 0 10 20 30\nspin: C 0 -2000 0.7 1 40 50 60\n"
        "spin: D 9000 0 1 70 80 0\nrho: Fx\ndet: Fp\n")
ROWS = np.array([[0.3, 1.1, 2.0, 0.5], [4.0, 0.7, 0.1, 1.5]])


@pytest.mark.parametrize("points", [1, 13, 14, 40, 41, 83, 131, 250])
def test_paired_powers_match_oracle(points):
    job = SPIN + f"npts: {points}\nsw: {13 * 9000.0!r}\nwr: 9000.0\nrotb: 54.7356\n"
    ref, _ = oracle_fid(job, ROWS)
    assert rel(gpu_fid(job, ROWS), ref) <= 1e-10
    assert rel(gpu_fid(job, ROWS, fave_method="direct"), ref) <= 1e-10


@pytest.mark.parametrize("points", [1, 63, 65, 128, 129, 700])
def test_static_terms_match_oracle(points):
    job = SPIN + f"npts: {points}\nsw: 40000.0\nwr: 0.0\nrotb: 54.7356\n"
    ref, _ = oracle_fid(job, ROWS)
    assert rel(gpu_fid(job, ROWS), ref) <= 1e-10


@pytest.mark.parametrize("points", [1, 2, 9, 10, 27, 50])
def test_point_to_point_terms_match_oracle(points):
    job = SPIN + f"npts: {points}\nsw: 0.0\nwr: 9000.0\nrotb: 54.7356\np2p: 9 4\nmaxtstep: 0.0\n"
    ref, _ = oracle_fid(job, ROWS)
    assert rel(gpu_fid(job, ROWS), ref) <= 1e-10
