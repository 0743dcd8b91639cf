"""Grids whose coarse levels are at the limits of the one-block coarse solve
(the tolerance hierarchy's is larger than the reference's: 20 warps, 2560
groups of four cells): a tolerance step runs and reaches its tolerance.

27x583, 50x1162: tops of 14x292, levels of 2052 groups.  32x640, 34x624: tops
of 17x321 (too many rows) and 18x313.  24x640: 13x321, one row more than 20
warps hold.  257x40: 129 columns, one more than a warp's.
"""
import numpy as np
import pytest

from ubootgl_gb300 import _lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "fp16", "bf16"])
@pytest.mark.parametrize("W,H", [(27, 583), (26, 582), (50, 1162), (32, 640), (34, 624), (24, 640),
                                 (257, 40)])
def test_step(lib, W, H, precision):
    from ubootgl_gb300.simulation import Simulation
    rng = np.random.default_rng(W + H)
    flag = np.ones((H, W), np.float32)
    flag[H // 3:H // 3 + 4, 5:W // 2] = 0.0
    s = Simulation(flag, 1.0, 1e-4)
    s.set_options(solver_mode=L.SOLVE_TOLERANCE, tol=1e-4, max_vcycles=200, precision=precision)
    s.set("vx", (1.0 + 0.1 * rng.standard_normal((H, W - 1))).astype(np.float32))
    s.step_cfl(0.5)
    assert s.solver_stats()[1] <= 1e-4
    assert all(np.isfinite(s.get(n)).all() for n in ("vx", "vy", "p"))
    s.close()
