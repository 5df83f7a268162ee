"""Segmented Dyson products: step counts at the edges of the 16-step segments, against the oracle.

FP64 to 1e-10 and the mixed form to 1e-6 relative L2, the engine's bars; small (3), large (10)
and rf-scheduled point-to-point blocks."""
import numpy as np
import pytest

from helpers import gpu_fid, oracle_fid, rel

pytestmark = pytest.mark.gpu


def job_of(nspin, n, extra=""):
    rng = np.random.default_rng(100 * nspin + n)
    lines = [f"numspin {nspin}"] + [f"T 1H {k}" for k in range(nspin)]
    for k in range(nspin):
        lines.append(f"C 0 {rng.uniform(500, 4000):.9g} {rng.uniform(0, 1):.9g} {k} "
                     + " ".join(f"{x:.9g}" for x in rng.uniform(0, 180, 3)))
        for j in range(k):
            lines.append(f"D {rng.uniform(-2e4, 2e4):.9g} {j} {k} " + " ".join(f"{x:.9g}" for x in rng.uniform(0, 180, 3)))
    wr = 1.0e4
    job = "".join(f"spin: {l}\n" for l in lines) + (
        f"npts: 60\nsw: {n * wr!r}\nwr: {wr!r}\nrotb: 54.7356\nrho: Fx\ndet: Fp\n" + extra)
    c = 3
    rows = np.stack([rng.uniform(0, 2 * np.pi, c), np.arccos(rng.uniform(-1, 1, c)), rng.uniform(0, 2 * np.pi, c),
                     rng.uniform(0.1, 1, c)], axis=1)
    return job, rows


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [15, 16, 17, 32, 33, 50])
@pytest.mark.parametrize("nspin", [3, 5])
def test_segment_edges_match_oracle(nspin, n, precision):
    job, rows = job_of(nspin, n)
    ref, _ = oracle_fid(job, rows)
    assert rel(gpu_fid(job, rows, precision=precision), ref) <= (1e-6 if precision else 1e-10)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("base,factor", [(16, 3), (17, 5), (33, 2)])
def test_segment_edges_point_to_point_match_oracle(base, factor, precision):
    job, rows = job_of(3, 10, f"p2p: {base} {factor}\nrfc: 3 1H 30000 90 0\n")
    ref, _ = oracle_fid(job, rows)
    assert rel(gpu_fid(job, rows, precision=precision), ref) <= (1e-6 if precision else 1e-10)
