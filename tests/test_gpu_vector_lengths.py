"""FP64 form, blocks of 84 and 126: short FIDs against dense 64-bit propagation, where nothing but the
rounding of the products and of the Floquet vectors is left.  The reference itself is up to 8e-15
from 80-bit propagation here; vectors whose length grows in the sweeps add 1.2e-14 (1.1e-14 to
2e-14 from the reference), without that the engine is 1e-15 from 80-bit propagation."""
import numpy as np
import pytest

import perf.cases as cases
from helpers import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("powder,steps,points,rho", [(1, 24, 96, "Fx"), (2, 15, 60, "Ix 0")])
@pytest.mark.parametrize("seed", [0, 1, 2])
def test_short_fids_to_fp64_rounding(seed, powder, steps, points, rho):
    case = dict(kind="mas", iso=" ".join(["1H"] * 9), powder=powder, steps=steps, points=points, wr=20e3, mixed=False,
                rho=rho, det="Fp")
    want = cases.exact(case, seed)
    assert want is not None
    assert rel(np.asarray(cases.run(cases.prepare(case, seed))), want) <= 1e-14
