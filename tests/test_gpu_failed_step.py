"""A step whose tolerance solve ends in an error leaves max|u| as it was: the
next device-CFL step takes its dt from the last completed step's velocity.

The residual overflows because of a sink of 1e30, which a dt of 0.5 uses up (its
strength falls to 1e-6 of it in 0.02; device-CFL steps need the list empty).
Tolerance 0 for dt: the same expression in FP32 on the same maximum.
"""
import numpy as np
import pytest

from ubootgl_gb300 import _lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "fp16"])
def test_dt_after_a_failed_solve(lib, precision):
    from ubootgl_gb300.simulation import Simulation
    W, H = 130, 66
    rng = np.random.default_rng(1)
    s = Simulation(np.ones((H, W), np.float32), 1.0, 1e-4)
    s.set_options(solver_mode=L.SOLVE_TOLERANCE, tol=1e-4, precision=precision)
    s.set("vx", (1.0 + 0.1 * rng.standard_normal((H, W - 1))).astype(np.float32))
    s.step_cfl(0.5)
    umax = max(np.abs(s.get(n)).max() for n in ("vx", "vy"))
    s.add_sink(0.5, 0.25, 1e30)
    with pytest.raises(L.UbgError):
        s.step(0.5)
    s.step_cfl(0.5)
    assert s.last_dt() == np.float32(0.5) * np.float32(s.h) / umax
    s.close()
