"""A serving pool of just the planned bytes holds the request: eleven like spins, whose index tables
(FID elements, operators by element) exceed the planner's fixed allowance, one orientation."""
import time

import numpy as np
import pytest

import blochlib_gb300 as bl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
def test_pool_of_the_planned_bytes_holds_eleven_spins(precision):
    n, wr, points = 11, 2.0e4, 11
    rng = np.random.default_rng(11)
    lines = [f"numspin {n}"] + [f"T 1H {k}" for k in range(n)]
    lines += [f"D {rng.uniform(-3e3, 3e3):.6g} {i} {j} {rng.uniform(0, 180):.6g} {rng.uniform(0, 180):.6g} 0"
              for i in range(n) for j in range(i)]
    system = bl.SolidSys(lines)
    pw = bl.powder.from_arrays(theta=[0.8], phi=[1.1], gamma=[0.3], weight=[1.0])
    job = dict(ro=system.op("Fx"), det=system.op("Fp"), npts=points, sw=11 * wr, wr=wr, rotb=54.7356, precision=precision)
    planned, _ = bl.job_bytes(system, pw, job["ro"], job["det"], points, job["sw"], wr, job["rotb"], precision=precision)
    if planned > 60 << 30:
        pytest.skip("planned for more than 60 GB")
    srv = bl.Server(0, lanes=1, pool_bytes=(planned + 1023) & ~1023)
    t = srv.submit(system, pw, **job)
    t0 = time.time()
    while True:
        state, fid, _, _ = srv.result(t)
        if state >= srv.DONE:
            break
        assert time.time() - t0 < 300
        time.sleep(0.01)
    assert state == srv.DONE
    dim = 2 ** n
    # Tr(Fp Fx) of every step over the reference's integer n / 2
    np.testing.assert_allclose(fid[0], n * dim / 2 * 11 / (11 // 2), rtol=1e-6)
    srv.close()
