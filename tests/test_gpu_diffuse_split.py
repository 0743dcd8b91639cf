"""Below 3000 blocks (256 x 4 faces) a block of the diffusion sweep takes one
velocity component, from there on both: a block less, the limit and a block more,
as a stage and in a step.

Tolerance 0: the restatement's expressions on the same values.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H", [11995, 11996, 11999, 12001])
def test_both_sides_of_the_limit(lib, H):
    from ubootgl_gb300.simulation import Simulation
    W = 20
    rng = np.random.default_rng(H)
    flag = (rng.random((H, W)) < 0.9).astype(np.float32)
    v = {"vx": rng.standard_normal((H, W - 1)).astype(np.float32),
         "vy": rng.standard_normal((H - 1, W)).astype(np.float32)}
    v.update(vx_back=v["vx"], vy_back=v["vy"])
    sim, ref = Simulation(flag, 1.0, 1e-2), O.PortSim(flag, 1.0, 1e-2)
    dt = np.float32(1e-3)
    for s in (sim, ref):
        for n, a in v.items():
            s.set(n, a)
    sim.dt = float(dt)
    ref.set_dt(dt)
    sim.diffuse()
    ref.stage("diffuse")
    for n in ("vx", "vy"):
        assert np.array_equal(sim.get(n), ref.get(n)), n
    sim.step(float(dt))
    ref.step(dt)
    for n in ("vx", "vy", "p"):
        assert np.array_equal(sim.get(n), ref.get(n)), n
    sim.close()
