"""Floquet step of period propagators with equal eigenvalues: methyl groups (three equal dipole
tensors), uncoupled spins beside a coupled pair, blocks of 3 to 35, against the oracle.  The last
form (more than 64 rotor periods in the mixed form) takes the FP64 sweeps there too.

FP64 to 1e-10 and the mixed form to 1e-6 relative L2, the engine's bars."""
import numpy as np
import pytest

from helpers import gpu_fid, oracle_fid, rel

pytestmark = pytest.mark.gpu


def _group(spins, a, alpha, beta):
    return [f"D {a} {i} {j} {alpha} {beta} 0" for i in spins for j in spins if i < j]


# spins, couplings, orientations
SYSTEMS = {
    "ch3": (3, _group((0, 1, 2), 9000, 30, 50), 600),
    "pair_of_four": (4, _group((0, 1), 9000, 30, 50), 600),
    "ch3_and_one": (4, _group((0, 1, 2), 9000, 30, 50) + ["D 300 0 3 70 20 0"], 600),
    "five_equal": (5, _group(range(5), 4000, 30, 50), 200),
    "two_ch3": (6, _group((0, 1, 2), 9000, 30, 50) + _group((3, 4, 5), 9000, 80, 110), 60),
    "two_ch3_and_one": (7, _group((0, 1, 2), 9000, 30, 50) + _group((3, 4, 5), 9000, 80, 110) + ["D 400 0 6 10 80 0"], 24),
}


@pytest.mark.parametrize("form", ["fp64", "point_to_point", "mixed_beyond_64_periods"])
@pytest.mark.parametrize("name", sorted(SYSTEMS))
def test_equal_eigenphases_match_oracle(name, form):
    nspin, couplings, count = SYSTEMS[name]
    rng = np.random.default_rng(nspin)
    lines = [f"numspin {nspin}"] + [f"T 1H {k}" for k in range(nspin)] + couplings
    n, wr = 24, 1.0e4
    mixed = form.startswith("mixed")
    job = "".join(f"spin: {l}\n" for l in lines) + (
        f"npts: {65 * n if mixed else 40}\nsw: {n * wr!r}\nwr: {wr!r}\nrotb: 54.7356\nrho: Ix 0\ndet: Fp\n")
    if form == "point_to_point":
        job += "p2p: 24 7\n"
    rows = np.stack([rng.uniform(0, 2 * np.pi, count), np.arccos(rng.uniform(-1, 1, count)),
                     rng.uniform(0, 2 * np.pi, count), rng.uniform(0.1, 1, count)], axis=1)
    ref, _ = oracle_fid(job, rows)
    assert rel(gpu_fid(job, rows, precision=int(mixed)), ref) <= (1e-6 if mixed else 1e-10)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("coupling", [1e-34, 1e-37, 1e-40])
@pytest.mark.parametrize("nspin", [4, 6])
def test_couplings_below_the_single_precision_range(nspin, coupling, precision):
    """A pair with a coupling near and below the smallest normal FP32 number, equal shifts, beside a
    strongly coupled pair: the element's reciprocal overflows in FP32."""
    lines = [f"numspin {nspin}"] + [f"T 1H {k}" for k in range(nspin)]
    lines += ["D 5000 0 1 30 50 0", f"D {coupling!r} 2 3 70 20 0"] + [f"D 900 1 {k} 10 80 0" for k in range(4, nspin)]
    n, wr = 24, 1.0e4
    job = "".join(f"spin: {l}\n" for l in lines) + (
        f"npts: 40\nsw: {n * wr!r}\nwr: {wr!r}\nrotb: 54.7356\nrho: Ix 0\ndet: Fp\n")
    rows = np.array([[0.3, 1.1, 0.2, 1.0], [2.0, 0.4, 1.5, 0.5], [4.1, 2.2, 5.0, 0.7]])
    ref, _ = oracle_fid(job, rows)
    assert rel(gpu_fid(job, rows, precision=precision), ref) <= (1e-6 if precision else 1e-10)
