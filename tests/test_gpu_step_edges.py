"""The step's kernels set the boundary values themselves; the stages called one
by one do it in launches of their own (setVBCs, setPBC).  Both ways give the
same bits for every combination of the four boundary types, at sizes where the
last columns and rows fall differently into the kernels' tiles (4 faces per
thread, 64 x 16 per block), with the two buffers' edges different at the
start, and over several steps.

Tolerance 0: the same expressions on the same values.
"""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TYPES = ["INFLOW", "OUTFLOW", "OUTFLOW_ZERO_PRESSURE", "NOSLIP"]
FIELDS = ("vx", "vy", "vx_back", "vy_back", "p", "f")


def pair(W, H, seed, **options):
    from ubootgl_gb300.simulation import Simulation
    rng = np.random.default_rng(seed)
    flag = (rng.random((H, W)) < 0.9).astype(np.float32)
    shape = {"vx": (H, W - 1), "vy": (H - 1, W), "p": (H, W)}
    shape.update(vx_back=shape["vx"], vy_back=shape["vy"])
    start = {n: rng.standard_normal(s).astype(np.float32) for n, s in shape.items()}
    sims = [Simulation(flag, 1.0, 1e-2) for _ in range(2)]
    for s in sims:
        if options:
            s.set_options(**options)
        for n, a in start.items():
            s.set(n, a)
    return sims


def stages(s, dt):
    s.dt = dt
    s.diffuse()
    s.advect()
    s.setVBCs()
    s.project()
    s.setVBCs()


def check(a, b, steps, what):
    dt = 0.3 / a.width
    for k in range(steps):
        a.step(dt)
        stages(b, dt)
        for n in FIELDS:
            x, y = a.get(n), b.get(n)
            assert np.array_equal(x, y), (what, k, n, np.argwhere(x != y)[:4].tolist())


def test_every_combination(lib):
    a, b = pair(14, 11, 1)
    start = {n: a.get(n) for n in FIELDS}
    for bcs in itertools.product(TYPES, repeat=4):
        for s in (a, b):
            s.set_bcs(*bcs)
            for n, v in start.items():
                s.set(n, v)
        check(a, b, 1, bcs)


@pytest.mark.parametrize("W,H", [(8, 8), (9, 10), (65, 17), (66, 19), (67, 18), (68, 33), (129, 34),
                                 (257, 20)])
def test_sizes(lib, W, H):
    for i, bcs in enumerate([("INFLOW", "OUTFLOW_ZERO_PRESSURE", "NOSLIP", "NOSLIP"),
                             ("NOSLIP", "INFLOW", "INFLOW", "OUTFLOW"),
                             ("OUTFLOW", "NOSLIP", "OUTFLOW_ZERO_PRESSURE", "INFLOW")]):
        a, b = pair(W, H, 10 * W + i)
        for s in (a, b):
            s.set_bcs(*bcs)
        check(a, b, 3, bcs)
        a.close()
        b.close()


@pytest.mark.parametrize("options", [{"advect": "bilinear"}, {"use_graph": False},
                                     {"precision": "fp16"}])
def test_options(lib, options):
    a, b = pair(70, 41, 5, **options)
    for s in (a, b):
        s.set_bcs("INFLOW", "OUTFLOW", "INFLOW", "NOSLIP")
    check(a, b, 2, options)
