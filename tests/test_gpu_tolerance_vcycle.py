"""One V-cycle of the tolerance solver's hierarchy (k_tile and k_coarse with
edges that follow their inner neighbours, FP32 and 16-bit coarse levels)
against its numpy restatement, at the sizes where it can go wrong: every
remainder of the width modulo 4 (the place of column w-1 in a lane) and of the
height modulo 8 (row h-1 as a warp's or a lane's first row), one region and
several, in both directions, of the tall and of the short region, levels of 1 to
20 warps in the one-block solve, and ones that do not fit it.

Tolerance 0: the same operations in the same order, rounded to 16 bits at the
same places (two NaNs count as equal).
"""
import numpy as np
import pytest

from oracle import tolerance as T
from ubootgl_gb300 import _lib as L

pytestmark = pytest.mark.gpu

PREC = {"fp32": L.FP32, "fp16": L.MIXED_FP16, "bf16": L.MIXED_BF16}

SIZES = ([(W, 8 + (W * 5) % 23) for W in range(8, 40)] +
         [(W, 97 + k) for k, W in enumerate((126, 127, 128, 129, 130, 131, 132, 133))] +
         # tops of 65x33, 64x32, 64x64, 33x121 (16 warps), 18x229 (FP32: smaller ones)
         [(128, 64), (129, 65), (127, 63), (126, 127), (65, 240), (34, 456)] +
         # 14x292 (2052 groups), 17x160 and 17x161 (20 warps and more), 13x320
         [(27, 583), (33, 319), (33, 320), (25, 639)] +
         # several regions; the tall region; elongated tails
         [(241, 113), (353, 33), (500, 131), (257, 225), (1203, 130), (1300, 209), (2400, 60),
          (2049, 40), (40, 1500)])


def inputs(W, H, seed):
    rng = np.random.default_rng(seed)
    flag = (rng.random((H, W)) < 0.85).astype(np.float32)
    flag[H // 4:3 * H // 4, W // 4:3 * W // 4] = 1.0  # an all-fluid part
    flag[H // 2:H // 2 + max(2, H // 8), 2:max(4, W // 6)] = 0.0  # and a solid one
    r = rng.standard_normal((H, W)).astype(np.float32)
    r[1:-1, 1:-1] *= flag[1:-1, 1:-1]
    r[0] = r[-1] = r[:, 0] = r[:, -1] = 0.0
    return flag, r


def vcycle(lib, flag, r, h, precision, rmax):
    H, W = r.shape
    z = np.empty_like(r)
    L.check(lib.ubg_selftest_vcycle(L.fptr(flag), L.fptr(r), W, H, h, PREC[precision], rmax,
                                    L.fptr(z)))
    return z


def check(lib, W, H, precision, less=1.0):
    flag, r = inputs(W, H, 1000 * W + H)
    h, rmax = float(np.float32(1.0 / (W - 1))), float(np.abs(r).max() * less)
    a = vcycle(lib, flag, r, h, precision, rmax)
    b = T.vcycle(flag, r, h, precision, rmax)
    same = (a == b) | (np.isnan(a) & np.isnan(b))
    assert same.all(), (int((~same).sum()), np.argwhere(~same)[:6].tolist())


@pytest.mark.parametrize("precision", list(PREC))
@pytest.mark.parametrize("W,H", SIZES)
def test_bit_exact(lib, W, H, precision):
    check(lib, W, H, precision)


@pytest.mark.parametrize("W,H,less", [(1300, 209, 17), (500, 131, 16), (257, 225, 15)])
def test_overflow_in_the_sweeps(lib, W, H, less):
    """A scale 2^less too large: FP16 values overflow, some within the sweeps
    of a region that starts with finite ones; solid cells stay 0."""
    check(lib, W, H, "fp16", 2.0 ** -less)
