"""Stages whose route depends on the steps per period or on the size of a step, against the oracle:
the correlation's transform lengths (2^a, 3 2^a, 5 2^a), the coefficients' Fourier series in runs of
16 steps, and the step polynomial's degrees.

FP64 to 1e-10 and the mixed form to 1e-6 relative L2, the engine's bars."""
import numpy as np
import pytest

from helpers import gpu_fid, oracle_fid, rel

pytestmark = pytest.mark.gpu


def job_of(nspin, n, rho="Fx", scale=1.0, seed=0):
    rng = np.random.default_rng(1000 * nspin + n + seed)
    lines = [f"numspin {nspin}"] + [f"T 1H {k}" for k in range(nspin)]
    for k in range(nspin):
        lines.append(f"C 0 {scale * rng.uniform(500, 4000):.9g} {rng.uniform(0, 1):.9g} {k} "
                     + " ".join(f"{x:.9g}" for x in rng.uniform(0, 180, 3)))
        for j in range(k):
            lines.append(f"D {scale * rng.uniform(-2e4, 2e4):.9g} {j} {k} "
                         + " ".join(f"{x:.9g}" for x in rng.uniform(0, 180, 3)))
    wr = 1.0e4
    job = "".join(f"spin: {l}\n" for l in lines) + (
        f"npts: 60\nsw: {n * wr!r}\nwr: {wr!r}\nrotb: 54.7356\nrho: {rho}\ndet: Fp\n")
    c = 3
    rows = np.stack([rng.uniform(0, 2 * np.pi, c), np.arccos(rng.uniform(-1, 1, c)), rng.uniform(0, 2 * np.pi, c),
                     rng.uniform(0.1, 1, c)], axis=1)
    return job, rows


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("rho", ["Fx", "Ix 0"])
@pytest.mark.parametrize("n", [5, 24, 25, 48, 49, 65, 80, 81, 96, 97, 129, 160, 161, 192, 193, 320, 384])
def test_transform_lengths_match_oracle(n, rho, precision):
    job, rows = job_of(3, n, rho)
    ref, _ = oracle_fid(job, rows)
    assert rel(gpu_fid(job, rows, precision=precision), ref) <= (1e-6 if precision else 1e-10)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("nspin", [4, 5, 6])
@pytest.mark.parametrize("scale", [1e-3, 0.03, 0.1, 0.3, 1.0])
def test_step_degrees_match_oracle(nspin, scale, precision):
    job, rows = job_of(nspin, 20, scale=scale)
    ref, _ = oracle_fid(job, rows)
    assert rel(gpu_fid(job, rows, precision=precision), ref) <= (1e-6 if precision else 1e-10)
