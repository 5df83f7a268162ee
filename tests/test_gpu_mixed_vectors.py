"""Mixed form: bits of the small blocks' Floquet vectors.  Pairs of protons over 52 rotor periods,
mixed against FP64: the mean over 100 random systems is 1.40e-7 when I + W and I - W are rounded once
and V takes no rotation by K's rounding, 1.60e-7 with such rotations and 1.96e-7 with W rounded first
as well; the bound lies between the first two."""
import numpy as np
import pytest

import perf.cases as cases
from helpers import rel

pytestmark = pytest.mark.gpu


def test_small_block_vectors_keep_single_precision():
    steps = 14
    case = dict(kind="mas", iso="1H 1H", powder=10, steps=steps, points=52 * steps, wr=20e3, mixed=True, rho="Ix 0",
                det="Fp")
    errors = []
    for seed in range(100):
        s = cases.prepare(case, seed)["jobs"][0]
        f64, mixed = (cases.bl.oneFID(s["system"], case["points"], cases._sweep(case), case["wr"], cases.MAGIC,
                                      precision=p).FID(s["pw"], s["ro"], s["det"]) for p in (0, 1))
        errors.append(rel(mixed, f64))
    assert np.mean(errors) <= 1.5e-7
