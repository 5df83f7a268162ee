"""Mixed form: factors that every FID term shares (the correlation's 1/M, the 2/n scale, the powder
weights) against the FP64 form, at steps per period whose correlation length is 2^a, 3 2^a and
5 2^a.  A shared factor kept in single precision is off by up to 2^-24 and moves the whole FID by
that, so the FID's amplitude along the FP64 FID has to be right to 2^-24."""
import numpy as np
import pytest

import perf.cases as cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nspin,powder", [(3, 64), (4, 11), (5, 3)])
@pytest.mark.parametrize("steps", [12, 20, 24, 40, 48, 64, 80, 90, 96])
def test_amplitude_of_the_mixed_form(steps, nspin, powder):
    case = dict(kind="mas", iso=" ".join(["1H"] * nspin), powder=powder, steps=steps, points=4 * steps, wr=20e3,
                mixed=True, rho="Fx", det="Fp")
    state = cases.prepare(case, steps)["jobs"][0]
    fid = {}
    for precision in (0, 1):
        drv = cases.bl.oneFID(state["system"], case["points"], cases._sweep(case), case["wr"], cases.MAGIC,
                              precision=precision)
        fid[precision] = drv.FID(state["pw"], state["ro"], state["det"])
    ref = fid[0]
    assert abs(np.vdot(ref, fid[1]).real / np.vdot(ref, ref).real - 1.0) <= 2.0 ** -24
