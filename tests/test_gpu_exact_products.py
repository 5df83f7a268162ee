"""Products by exact digit slices (blocks above 74, both forms) against dense 64-bit propagation,
at the edges of the Dyson segments: blocks of 84 and 126 leave K and column remainders in every
tile.  Tolerances are the engine's bars: 1e-10 (FP64) and 1e-6 (mixed form) relative L2."""
import numpy as np
import pytest

import perf.cases as cases
from helpers import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("steps,rho", [(12, "Fx"), (17, "Ix 0"), (33, "Fx")])
def test_blocks_of_84_and_126_match_dense_propagation(steps, rho, mixed):
    case = dict(kind="mas", iso=" ".join(["1H"] * 9), powder=1, steps=steps, points=40, wr=20e3, mixed=mixed, rho=rho,
                det="Fp")
    want = cases.exact(case, 5)
    assert want is not None
    got = np.asarray(cases.run(cases.prepare(case, 5)))
    assert rel(got, want) <= (1e-6 if mixed else 1e-10)
