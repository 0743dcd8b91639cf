"""numpy restatement of one preconditioning V-cycle of the tolerance solver
(the hierarchy of `ext_*` in k_mg.cu) -- TEST INFRASTRUCTURE ONLY.

Every level's arrays in plain numpy, the library's operations in its order, in
FP32, the levels above the coarse end rounded to FP16 or BF16 where the library
stores them so.  A cell's neighbours are selected by their flags, edges are
copied after each sweep: nothing of the kernels' layout is in it.
"""
import numpy as np

f32 = np.float32


def round_to(precision):
    """The rounding of stored values: FP32, FP16 or BF16 (to nearest even)."""
    if precision == "fp32":
        return lambda a: a
    if precision == "fp16":
        return lambda a: a.astype(np.float16).astype(f32)

    def bf16(a):
        u = np.ascontiguousarray(a, f32).view(np.uint32)
        r = ((u + np.uint32(0x7fff) + ((u >> 16) & 1)) & np.uint32(0xffff0000)).view(f32)
        return np.where(np.isnan(a), a, r)
    return bf16


def shapes(W, H):
    out = [(W, H)]
    while True:
        w, h = out[-1]
        nw, nh = w // 2 + 1, h // 2 + 1
        if nw < 5 or nh < 5 or nw >= w or nh >= h:
            return out
        out.append((nw, nh))


def coarsen(flag):
    """Fluid if any of the nine fine cells is; edge cells fluid."""
    H, W = flag.shape
    w, h = W // 2 + 1, H // 2 + 1
    c = np.ones((h, w), bool)
    X, Y = np.arange(1, w - 1), np.arange(1, h - 1)
    a = np.zeros((h - 2, w - 2), bool)
    for dy in (-1, 0, 1):
        for dx in (-1, 0, 1):
            a |= flag[np.ix_(2 * Y + dy, 2 * X + dx)]
    c[1:-1, 1:-1] = a
    return c


def copy_edges(e):
    e[1:-1, 0] = e[1:-1, 1]
    e[1:-1, -1] = e[1:-1, -2]
    e[0] = e[1]
    e[-1] = e[-2]


class Level:
    def __init__(self, flag, h, rnd):
        self.flag, self.rnd, self.h = flag, rnd, f32(h)
        self.ihsq = f32(1.0) / self.h / self.h
        H, W = flag.shape
        self.n = (flag[1:-1, :-2].astype(int) + flag[1:-1, 2:] + flag[:-2, 1:-1] + flag[2:, 1:-1])
        self.red = (np.add.outer(np.arange(1, H - 1), np.arange(1, W - 1)) & 1) == 1
        self.e = np.zeros((H, W), f32)
        self.f = np.zeros((H, W), f32)

    def neighbours(self, other):
        """West, east, south, north values; `other` where the flag is not set."""
        e, g = self.e, self.flag
        for a, b in ((np.s_[1:-1, :-2],) * 2, (np.s_[1:-1, 2:],) * 2, (np.s_[:-2, 1:-1],) * 2,
                     (np.s_[2:, 1:-1],) * 2):
            yield np.where(g[b], e[a], other)

    def half(self, red):
        v = f32(0.0)
        for t in self.neighbours(f32(0.0)):
            v = v + t
        v = v + self.f[1:-1, 1:-1] * self.h * self.h
        q = np.zeros_like(v)
        for k in (1, 2, 4):
            q = np.where(self.n == k, v * f32(1.0 / k), q)
        q = np.where(self.n == 3, v / f32(3.0), q)
        q = np.where(self.flag[1:-1, 1:-1], self.rnd(q), f32(0.0))
        inner = self.e[1:-1, 1:-1]
        inner[...] = np.where(self.red == red, q, inner)

    def sweeps(self, n):
        for _ in range(n):
            self.half(True)
            self.half(False)
            copy_edges(self.e)

    def residual(self):
        c = self.e[1:-1, 1:-1]
        v = f32(0.0)
        for t in self.neighbours(c):
            v = v + t
        v = v + f32(-4.0) * c
        r = np.zeros_like(self.e)
        r[1:-1, 1:-1] = np.where(self.flag[1:-1, 1:-1],
                                 self.rnd(self.f[1:-1, 1:-1] + v * self.ihsq), f32(0.0))
        return r

    def restricted(self, shape, rfac):
        r = self.residual()
        h, w = shape
        X, Y = 2 * np.arange(1, w - 1), 2 * np.arange(1, h - 1)
        at = lambda dy, dx: r[np.ix_(Y + dy, X + dx)]  # noqa: E731
        one = lambda dy: (at(dy, -1) + f32(2) * at(dy, 0)) + at(dy, 1)  # noqa: E731
        two = (f32(2) * at(0, -1) + f32(4) * at(0, 0)) + f32(2) * at(0, 1)
        out = np.zeros(shape, f32)
        out[1:-1, 1:-1] = ((one(-1) + two) + one(1)) * rfac
        return out

    def correct(self, c, scale=None):
        """p += prolongate(c.e) on the interior fluid cells, then the edges."""
        H, W = self.flag.shape
        y, x = np.mgrid[1:H - 1, 1:W - 1]
        X, Y = x >> 1, y >> 1
        X1, Y1 = np.minimum(X + 1, c.e.shape[1] - 1), np.minimum(Y + 1, c.e.shape[0] - 1)
        e, g = c.e, c.flag.astype(int)
        E00, E10, E01, E11 = e[Y, X], e[Y, X1], e[Y1, X], e[Y1, X1]
        G00, G10, G01, G11 = g[Y, X], g[Y, X1], g[Y1, X], g[Y1, X1]
        d = np.array([f32(np.float64(f32(k)) + 0.0001) for k in range(5)], f32)
        xo, yo = (x & 1) == 1, (y & 1) == 1
        u = np.where(xo & ~yo, (E00 + E10) / d[G00 + G10], E00)
        u = np.where(~xo & yo, (E00 + E01) / d[G00 + G01], u)
        u = np.where(xo & yo, (((E00 + E11) + E10) + E01) / d[G00 + G11 + G10 + G01], u)
        if scale is not None:
            u = u * scale
        p = self.e[1:-1, 1:-1]
        p[...] = np.where(self.flag[1:-1, 1:-1], self.rnd(p + u), p)
        copy_edges(self.e)


def vcycle(flag, r, h, precision="fp32", rmax=None, ncoarse=16):
    """z = M r (H x W float32): level 0 in FP32, the coarse levels FP32 or, in
    the h^2-scaled form, 16-bit down to the first one of at most 4096 cells,
    whose result alone is rounded (its inside and the levels below are FP32).
    rmax: the largest |r|, which sets the 16-bit levels' scale."""
    with np.errstate(all="ignore"):
        return _vcycle(flag, r, h, precision, rmax, ncoarse)


def _vcycle(flag, r, h, precision, rmax, ncoarse):
    H, W = r.shape
    sh = shapes(W, H)
    scaled = precision != "fp32"
    rnd, exact = round_to(precision), round_to("fp32")
    last = len(sh) - 1
    top = next((l for l in range(1, last + 1) if sh[l][0] * sh[l][1] <= 4096), last)
    lv, g, hh = [], np.asarray(flag) != 0, f32(h)
    for l in range(len(sh)):
        lv.append(Level(g, f32(1.0) if scaled and l else hh, rnd if 1 <= l < top else exact))
        g, hh = coarsen(g), f32(2.0) * hh
    lv[0].f[...] = r
    rfac0, back = f32(1.0 / 16.0), None
    if scaled:
        h1sq = (f32(2.0) * f32(h)) * (f32(2.0) * f32(h))
        kexp = 0
        if precision == "fp16":
            n = float(max(sh[1]))
            kexp = max(0, int(np.ceil(np.log2(0.5 * n * n))) - 14)
        m = f32(np.abs(r).max() if rmax is None else rmax) * h1sq
        ex = int(np.frexp(m)[1])
        rfac0 = rfac0 * (f32(2.0 ** (-ex - kexp)) * h1sq)
        back = f32(2.0 ** (ex + kexp))
    rfac = f32(0.25) if scaled else f32(1.0 / 16.0)
    for l in range(last):
        lv[l].sweeps(3)
        f = lv[l].restricted(lv[l + 1].f.shape, rfac0 if l == 0 else rfac)
        lv[l + 1].f[...] = rnd(f) if l + 1 <= top else f
    lv[last].sweeps(ncoarse)
    for l in range(last - 1, -1, -1):
        if l + 1 == top:
            lv[top].e[...] = rnd(lv[top].e)
        lv[l].correct(lv[l + 1], back if l == 0 else None)
        lv[l].sweeps(3)
    return lv[0].e
