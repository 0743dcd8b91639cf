"""Fused batches where their launches differ from a single simulation's: the
multigrid region is chosen by the blocks of all members together (the short one
below 304 short blocks, whatever a level's width), and the fused kernels set
every member's own boundary values.

Tolerance 0: the same expressions on the same values, against the restatement
and against each member stepped alone.
"""
import itertools

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

FIELDS = ("vx", "vy", "vx_back", "vy_back", "p")


def start(W, H, seed):
    rng = np.random.default_rng(seed)
    flag = (rng.random((H, W)) < 0.9).astype(np.float32)
    flag[H // 4:3 * H // 4, W // 4:3 * W // 4] = 1.0
    v = {"vx": rng.standard_normal((H, W - 1)).astype(np.float32),
         "vy": rng.standard_normal((H - 1, W)).astype(np.float32),
         "p": rng.standard_normal((H, W)).astype(np.float32)}
    v.update(vx_back=v["vx"], vy_back=v["vy"])
    return flag, v


def short_blocks(W, H):
    def regions(c, n):
        return 1 if c <= n else (c - 16 + n - 17) // (n - 16)
    return regions(W, 128) * regions(H, 32)


# one level 0 of 1200 columns and more in the short region (the tall one
# alone), narrower levels 0 and 1 in the tall region (the short one alone)
@pytest.mark.parametrize("sizes,tall", [
    ([(1300, 201), (1201, 97)], (False, False)),
    ([(450 + 7 * i, 255 + i) for i in range(6)], (True, False)),
    ([(480 + 7 * i, 255 + 3 * i) for i in range(14)], (True, True))])
def test_region_by_blocks(lib, sizes, tall):
    from ubootgl_gb300.simulation import Batch, Simulation
    for l in range(2):
        assert (sum(short_blocks(W >> l, H >> l) for W, H in sizes) >= 304) == tall[l]
    sims, refs = [], []
    for i, (W, H) in enumerate(sizes):
        flag, v = start(W, H, i)
        sims.append(Simulation(flag, 1.0, 1e-4))
        refs.append(O.PortSim(flag, 1.0, 1e-4))
        for s in (sims[-1], refs[-1]):
            for n, a in v.items():
                s.set(n, a)
    batch = Batch(sims)
    for _ in range(2):
        batch.step(cfl=0.5)
        batch.sync()
        for s, r in zip(sims, refs):
            r.step(np.float32(s.last_dt()))
    for s, r in zip(sims, refs):
        for n in ("vx", "vy", "p"):
            assert np.array_equal(s.get(n), r.get(n)), (s.width, s.height, n)
    batch.close()
    for s in sims:
        s.close()


def test_every_boundary_combination(lib):
    from ubootgl_gb300.simulation import Batch, Simulation
    types = ["INFLOW", "OUTFLOW", "OUTFLOW_ZERO_PRESSURE", "NOSLIP"]
    combos = list(itertools.product(types, repeat=4))

    def make(i):
        flag, v = start(34 + i % 9, 25 + i % 5, i)
        s = Simulation(flag, 1.0, 1e-2)
        s.set_bcs(*combos[i])
        for n, a in v.items():
            s.set(n, a if not n.endswith("_back") else 0.5 * a)
        return s

    members = [make(i) for i in range(len(combos))]
    batch = Batch(members)
    for _ in range(3):
        batch.step(cfl=0.5)
    batch.sync()
    for i, m in enumerate(members):
        s = make(i)
        for _ in range(3):
            s.step_cfl(0.5)
        for n in FIELDS:
            assert np.array_equal(s.get(n), m.get(n)), (combos[i], n)
        s.close()
    batch.close()
    for m in members:
        m.close()
