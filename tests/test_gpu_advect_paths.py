"""The advection takes one of three ways per tile: every stencil in the staged
windows and clear of the domain's edge, every stencil in the windows, or any
trace.  Each against the restatement, at grids with tall and with low tiles
and remainders in both directions, for fields whose fastest face travels from
a fraction of a cell to many cells (1.28 cells is where a tile changes over),
and for fields with single infinite, huge and undefined values.

Tolerance 0: the restatement's expressions on the same values (two NaNs
count as equal).
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def check(W, H, cells, odd=()):
    from ubootgl_gb300.simulation import Simulation
    rng = np.random.default_rng(W + H)
    flag = np.ones((H, W), np.float32)
    for _ in range(20):
        x, y = rng.integers(4, W), rng.integers(4, H)
        flag[y:y + 5, x:x + 9] = 0.0
    v = {"vx": rng.uniform(-1, 1, (H, W - 1)).astype(np.float32),
         "vy": rng.uniform(-1, 1, (H - 1, W)).astype(np.float32)}
    for k, a in enumerate(odd):
        v["vx"][H // 2, (k + 1) * W // 5] = a
        v["vy"][(k + 1) * H // 5, W // 2] = a
    sim, ref = Simulation(flag, 1.0, 1e-4), O.PortSim(flag, 1.0, 1e-4)
    dt = np.float32(cells * ref.h)
    for s in (sim, ref):
        for n in v:
            s.set(n, v[n])
            s.set(n + "_back", v[n])
    sim.dt = float(dt)
    ref.set_dt(dt)
    sim.advect()
    ref.stage("advect")
    for n in ("vx", "vy"):
        a, b = sim.get(n), ref.get(n)
        same = (a == b) | (np.isnan(a) & np.isnan(b))
        assert same.all(), (W, H, cells, n, np.argwhere(~same)[:4].tolist())
    sim.close()


# 608 tiles of 64 x 16 and more are advected in tall tiles
SIZES = [(8, 8), (67, 13), (130, 66), (193, 41), (1217, 521), (2049, 307)]


@pytest.mark.parametrize("W,H", SIZES)
@pytest.mark.parametrize("cells", [0.5, 1.27, 1.29, 40.0])
def test_reach(lib, W, H, cells):
    check(W, H, cells)
    check(W, H, -cells)


@pytest.mark.parametrize("W,H", [(130, 66), (2049, 307)])
@pytest.mark.parametrize("odd", [(np.inf,), (-np.inf, np.nan), (1e30, 1e38), (1e-40,)])
def test_odd_values(lib, W, H, odd):
    check(W, H, 0.5, odd)
    check(W, H, 0.0, odd)
