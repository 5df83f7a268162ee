"""FP64 form, blocks of 20 to 35 on the digit-slice products: the FID is linear in the detection
operator, also where that is near the ends of the FP64 range."""
import numpy as np
import pytest

import blochlib_gb300 as bl
from helpers import parse_job, rel
from test_gpu_lengths import job_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("power", [-1005, -985, -60, 60, 985])
@pytest.mark.parametrize("nspin", [6, 7])
def test_fid_is_linear_in_the_detection_operator(nspin, power):
    job, rows = job_of(nspin, 18, rho="Ix 0")
    lines, _ = parse_job(job)
    system = bl.SolidSys(lines)
    pw = bl.powder.from_arrays(theta=rows[:, 1], phi=rows[:, 0], gamma=rows[:, 2], weight=rows[:, 3])
    drv = bl.oneFID(system, 60, 18e4, 1e4, 54.7356)
    ro, det = system.op("Ix 0"), system.op("Fp")
    ref = drv.FID(pw, ro, det)
    got = drv.FID(pw, ro, np.ldexp(det.real, power) + 0j)
    got = np.ldexp(got.real, -power) + 1j * np.ldexp(got.imag, -power)
    assert rel(got, ref) <= 1e-12
