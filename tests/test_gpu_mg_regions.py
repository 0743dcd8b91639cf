"""The multigrid's register-held regions (k_tile, k_coarse) at the sizes where
they can go wrong: one column or row less, equal and more than a region and
than the overlapping regions' strides (112 x 48, 112 x 16), levels that
enter the one-block coarse solve at its limits (128 x 64), elongated levels
that it does not take, and magnitudes outside the range in which the packed
scaling is used.

Against the CPU restatement, tolerance 0: both evaluate the same IEEE
operations in the same order.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

SIZES = [(8, 8), (9, 70), (127, 31), (128, 64), (129, 65), (128, 63), (112, 161), (239, 113),
         (240, 48), (241, 112), (256, 128), (257, 130), (353, 33), (400, 20), (1201, 60),
         (2000, 24)]


def arrays(W, H, scale, seed):
    """Random flags (edge cells and isolated cells among them), p and f."""
    rng = np.random.default_rng(seed)
    flag = (rng.random((H, W)) < 0.8).astype(np.float32)
    flag[H // 4:3 * H // 4, W // 4:3 * W // 4] = 1.0  # and an all-fluid part
    p = (scale * rng.standard_normal((H, W))).astype(np.float32)
    f = (scale * W * rng.standard_normal((H, W))).astype(np.float32)
    return flag, p, f


@pytest.mark.parametrize("zgbc", [True, False])
@pytest.mark.parametrize("W,H", SIZES)
def test_solve_bit_exact(lib, W, H, zgbc):
    from ubootgl_gb300.simulation import MG
    flag, p, f = arrays(W, H, 1.0, W * 1000 + H)
    h = float(np.float32(1.0 / (W - 1)))
    mg = MG(flag)
    a = b = p
    for _ in range(2):
        a = mg.solve(a.copy(), f, flag, h, zgbc)
        b = O.port_mg_solve(b, f, flag, h, zgbc, coarse_flag=flag)
        assert np.array_equal(a, b), np.abs(a.astype(np.float64) - b).max()


@pytest.mark.parametrize("scale", [1e25, 1e-25, 1e-38])
@pytest.mark.parametrize("W,H", [(129, 65), (300, 100)])
def test_solve_magnitudes_bit_exact(lib, W, H, scale):
    from ubootgl_gb300.simulation import MG
    flag, p, f = arrays(W, H, scale, 5)
    h = float(np.float32(1.0 / (W - 1)))
    a = MG(flag).solve(p.copy(), f, flag, h, True)
    b = O.port_mg_solve(p, f, flag, h, True, coarse_flag=flag)
    assert np.isfinite(b).all()
    assert np.array_equal(a, b)


@pytest.mark.parametrize("tile", ["128x64", "128x32"])
def test_region_choice_bit_exact(lib, tile):
    """Both regions on every level: the autotuner's trials run all of them, so
    a step after it compares what it chose; the level sizes are such that the
    default takes the other one on at least one level."""
    from ubootgl_gb300.simulation import Simulation
    W, H = (1300, 200) if tile == "128x32" else (700, 300)
    flag, _, _ = arrays(W, H, 1.0, 3)
    sim, ref = Simulation(flag), O.PortSim(flag)
    rng = np.random.default_rng(4)
    vx = rng.standard_normal((H, W - 1)).astype(np.float32)
    vy = rng.standard_normal((H - 1, W)).astype(np.float32)
    rep = sim.autotune()
    assert {lv["pre"] for lv in rep["levels"]} <= {"default", "128x64", "128x32"}
    for s in (sim, ref):
        s.set("vx", vx)
        s.set("vy", vy)
    for _ in range(2):
        sim.step(1e-4)
        ref.step(np.float32(1e-4))
    for n in ("vx", "vy", "p"):
        assert np.array_equal(sim.get(n), ref.get(n)), n
    sim.close()
