"""The workloads the library's speed is measured on, through its public entry points.

A case is a dict of plain values; `kind` names the entry point:

* step    one simulation, `steps` device-CFL steps (Simulation.step_cfl), then
          its vx, vy and p read in place on the device;
* io      host in, host out: every frame uploads its velocity from pinned
          memory, steps, and reads the result back (ubg_io_*);
* tol     steps whose projection is solved to a relative residual `tol`;
* batch   several uneven simulations advanced together (Batch.step);
* serve   requests of several steps each on the sessions of a Server;
* mg      the pressure solver alone on device arrays (ubg_mg_solve_device).

Work on the device is ordered with PyTorch's current stream on both sides, as
in a program that hands the fields to PyTorch.  `exact` is the same arithmetic
in 64 bits in plain PyTorch.
"""
import ctypes as C
import math

import torch
import torch.nn.functional as F

from ubootgl_gb300 import _lib as L
from ubootgl_gb300.simulation import MG, Batch, Server, Simulation

CFL, PWIDTH, MU = 0.5, 1.0, 1e-4


def listed():
    def step(W, H, steps, advect="bicubic"):
        return {"name": "step_%dx%d" % (W, H), "kind": "step", "W": W, "H": H, "steps": steps,
                "advect": advect}

    return [
        # a small interactive session: the smallest size that is served, a
        # request of several steps; launches and coarse levels decide
        step(256, 128, 10),
        # an odd grid, with the option of bilinear advection
        step(389, 211, 8, "bilinear"),
        # the reference's own comparison grid
        step(1024, 512, 4),
        # a ragged grid of ordinary size
        step(2045, 1021, 2),
        # the headline grid, and the largest that is run
        step(4096, 2048, 2),
        step(8192, 4096, 1),
        # the headline grid fed from and read back to host memory each step
        {"name": "io_4096x2048", "kind": "io", "W": 4096, "H": 2048, "steps": 2},
        # projections solved to a tolerance: FP32, and 16-bit coarse levels
        {"name": "tol_fp32_1024x512", "kind": "tol", "W": 1024, "H": 512, "steps": 1,
         "precision": "fp32", "tol": 1e-6},
        {"name": "tol_fp16_4096x2048", "kind": "tol", "W": 4096, "H": 2048, "steps": 1,
         "precision": "fp16", "tol": 1e-5},
        # uneven instances advanced together
        {"name": "batch_20", "kind": "batch", "n": 20, "wmin": 128, "wmax": 2048, "steps": 2},
        # requests of 1 to 20 steps on resident sessions
        {"name": "serve_16", "kind": "serve", "n": 16, "wmin": 256, "wmax": 2048},
        # the solver alone, several V-cycles on device arrays
        {"name": "mg_1025x513", "kind": "mg", "W": 1025, "H": 513, "cycles": 4, "zgbc": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "io", "tol", "batch", "serve", "mg"])
    if kind in ("batch", "serve"):
        c = {"kind": kind, "n": rng.randint(4, 16), "wmin": 128 if kind == "batch" else 256,
             "wmax": _log_int(rng, 512, 2048)}
        if kind == "batch":
            c["steps"] = rng.randint(1, 4)
        return c
    top = {"step": 8192, "io": 4096, "tol": 2048, "mg": 4096}[kind]
    W = _log_int(rng, 96, top)
    H = max(24, int(W * rng.uniform(0.3, 0.6)))
    c = {"kind": kind, "W": W, "H": H}
    if kind == "mg":
        c.update(cycles=rng.randint(1, 4), zgbc=rng.random() < 0.75)
        return c
    c["steps"] = max(1, min(rng.randint(1, 12), 16777216 // (W * H)))
    if kind == "step":
        c["advect"] = "bilinear" if rng.random() < 0.25 else "bicubic"
    if kind == "tol":
        c["steps"] = min(c["steps"], 2)
        c.update(precision=rng.choice(["fp32", "fp16"]), tol=rng.choice([1e-5, 1e-6]))
    return c


# ------------------------------------------------------------------ inputs
def _instance(W, H, seed, u_in=1.0):
    """A channel with solid top and bottom rows and seeded discs (8 to 15 %
    solid), and a stream along it with smoothed noise: (flag, vx, vy) on the
    GPU, float32."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    cpu = torch.Generator().manual_seed(seed + 1)
    flag = torch.ones(H, W, device="cuda")
    flag[0] = 0.0
    flag[-1] = 0.0
    yy = torch.arange(H, device="cuda", dtype=torch.float32)[:, None]
    xx = torch.arange(W, device="cuda", dtype=torch.float32)[None, :]
    rnd = lambda: float(torch.rand((), generator=cpu))  # noqa: E731
    want, area = (0.08 + 0.07 * rnd()) * W * H, 0.0
    while area < want:
        r = (0.02 + 0.04 * rnd()) * min(W, 2 * H)
        cx, cy = W * (0.1 + 0.8 * rnd()), H * rnd()
        x0, x1 = max(1, int(cx - r) - 1), min(W - 1, int(cx + r) + 2)
        y0, y1 = max(0, int(cy - r) - 1), min(H, int(cy + r) + 2)
        area += 0.85 * math.pi * r * r
        d2 = (xx[:, x0:x1] - cx) ** 2 + (yy[y0:y1] - cy) ** 2
        flag[y0:y1, x0:x1] *= (d2 > r * r).float()

    def noise(h, w):
        c = torch.randn(1, 1, h // 8 + 2, w // 8 + 2, generator=g, device="cuda")
        n = F.interpolate(c, size=(h, w), mode="bicubic", align_corners=True)[0, 0]
        return n / n.std().clamp_min(1e-9)

    vx = 1.0 + 0.1 * noise(H, W - 1)
    vy = 0.1 * noise(H - 1, W)
    vx[:, 0] = u_in
    vx *= flag[:, :-1] * flag[:, 1:]
    vy *= flag[:-1] * flag[1:]
    vy[0] = 0.0
    return flag, vx, vy


def _members(case, seed):
    """(W, H, seed, inflow, steps) of every member of a batch or server; the
    sizes and the steps are the case's own."""
    g = torch.Generator().manual_seed(17 * case["n"] + case["wmax"])
    out = []
    for i in range(case["n"]):
        r = [float(v) for v in torch.rand(3, generator=g)]
        w = case["wmin"] * (case["wmax"] / case["wmin"]) ** r[0]
        W = max(case["wmin"], min(case["wmax"], 32 * round(w / 32)))
        k = case["steps"] if case["kind"] == "batch" else 1 + int(r[2] * 19.999)
        out.append((W, W // 2, seed * 1000 + 7 * i, 0.5 + r[1], k))
    return out


class _View:
    """A field of the library on the device, for torch.as_tensor; the tensor
    keeps the view, and the view the owner of the memory."""

    def __init__(self, owner, ptr, pitch, w, h):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (h, w), "strides": (pitch * 4, 4),
                                         "typestr": "<f4", "data": (ptr, False), "version": 3}


class _Fields:
    """Device views of a simulation's fields: the buffers rotate from step to
    step, so the pointer is asked for each time; tensors are kept by it."""

    def __init__(self, owner, handle):
        self.owner, self.lib, self.handle, self.made = owner, owner._lib, handle, {}
        self.ptr, self.pitch, self.w, self.h = C.c_void_p(), C.c_int(), C.c_int(), C.c_int()

    def __call__(self, name):
        L.check(self.lib.ubg_field_device(self.handle, L.FIELDS[name], C.byref(self.ptr),
                                          C.byref(self.pitch), C.byref(self.w), C.byref(self.h)))
        key = (name, self.ptr.value)
        if key not in self.made:
            self.made[key] = torch.as_tensor(
                _View(self.owner, self.ptr.value, self.pitch.value, self.w.value, self.h.value),
                device="cuda")
        return self.made[key]

    def all(self):
        return [self(n) for n in ("vx", "vy", "p")]


def _stream(call, handle):
    p = C.c_void_p()
    L.check(call(handle, C.byref(p)))
    return torch.cuda.ExternalStream(p.value)


def _simulation(W, H, seed, u_in=1.0, **options):
    flag, vx, vy = _instance(W, H, seed, u_in)
    sim = Simulation(flag.cpu().numpy(), PWIDTH, MU)
    if options:
        sim.set_options(**options)
    fields = _Fields(sim, sim._h)
    for back in ("", "_back"):  # the inflow is held in both buffers
        fields("vx" + back).copy_(vx)
        fields("vy" + back).copy_(vy)
    torch.cuda.synchronize()
    return sim, fields


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("step", "tol"):
        if kind == "step":
            opt = {"advect": "bilinear"} if case["advect"] == "bilinear" else {}
        else:
            opt = {"solver_mode": L.SOLVE_TOLERANCE, "tol": case["tol"],
                   "precision": case["precision"]}
        sim, fields = _simulation(case["W"], case["H"], seed, **opt)
        return {"kind": kind, "steps": case["steps"], "sim": sim, "fields": fields,
                "stream": _stream(sim._lib.ubg_stream, sim._h)}
    if kind == "io":
        W, H = case["W"], case["H"]
        flag, vx, vy = _instance(W, H, seed)
        sim = Simulation(flag.cpu().numpy(), PWIDTH, MU)
        frames = []
        for k in range(case["steps"]):
            bufs = [torch.empty(s, pin_memory=True) for s in ((H, W - 1), (H - 1, W)) * 2]
            bufs[0].copy_(vx)
            bufs[1].copy_(vy * (1.0 - 0.1 * k))
            frames.append(bufs)
        torch.cuda.synchronize()
        return {"kind": kind, "sim": sim, "frames": frames}
    if kind == "batch":
        members = [_simulation(*m[:4]) for m in _members(case, seed)]
        batch = Batch([m[0] for m in members])
        return {"kind": kind, "steps": case["steps"], "batch": batch, "members": members,
                "stream": _stream(batch._lib.ubg_batch_stream, batch._h)}
    if kind == "serve":
        srv = Server(8 << 30, max_active=16)
        sessions = []
        for W, H, s, u, k in _members(case, seed):
            flag, vx, vy = (t.cpu().numpy() for t in _instance(W, H, s, u))
            sid = srv.open(flag, vx, vy, PWIDTH, MU)
            h = C.c_void_p()
            L.check(srv._lib.ubg_server_session_sim(srv._h, sid, C.byref(h)))
            sessions.append((sid, k, _Fields(srv, h)))
        return {"kind": kind, "server": srv, "sessions": sessions}
    if kind == "mg":
        W, H = case["W"], case["H"]
        flag, vx, vy = _instance(W, H, seed)
        f = torch.zeros(H, W, device="cuda")
        h = PWIDTH / (W - 1)
        f[1:-1, 1:-1] = -(vx[1:-1, 1:] - vx[1:-1, :-1] + vy[1:, 1:-1] - vy[:-1, 1:-1]) / h
        mg = MG(flag.cpu().numpy())
        torch.cuda.synchronize()
        return {"kind": kind, "mg": mg, "p": torch.zeros(H, W, device="cuda"), "f": f,
                "flag": flag.to(torch.uint8), "h": h, "cycles": case["cycles"],
                "zgbc": int(case["zgbc"]), "stream": torch.cuda.Stream()}
    raise ValueError(kind)


# --------------------------------------------------------------------- run
def run(s):
    kind = s["kind"]
    if kind == "io":
        sim = s["sim"]
        at = lambda t: C.cast(t.data_ptr(), C.POINTER(C.c_float))  # noqa: E731
        for ix, iy, ox, oy in s["frames"]:
            L.check(sim._lib.ubg_io_upload_async(sim._h, at(ix), at(iy)))
            sim.step_cfl(CFL)
            L.check(sim._lib.ubg_io_download_async(sim._h, at(ox), at(oy)))
        L.check(sim._lib.ubg_io_wait(sim._h))
        return [[b[2], b[3]] for b in s["frames"]]
    if kind == "serve":
        for sid, k, _ in s["sessions"]:
            s["server"].submit(sid, k, CFL)
        s["server"].drain()
        return [f.all() for _, _, f in s["sessions"]]
    here = torch.cuda.current_stream()
    s["stream"].wait_stream(here)
    if kind == "mg":
        p, f, flag, mg = s["p"], s["f"], s["flag"], s["mg"]
        W = p.shape[1]
        for _ in range(s["cycles"]):
            L.check(mg._lib.ubg_mg_solve_device(
                mg._h, p.data_ptr(), W, f.data_ptr(), W, flag.data_ptr(), W, s["h"], s["zgbc"],
                s["stream"].cuda_stream))
        here.wait_stream(s["stream"])
        return p
    if kind == "batch":
        for _ in range(s["steps"]):
            s["batch"].step(cfl=CFL)
        here.wait_stream(s["stream"])
        return [f.all() for _, f in s["members"]]
    for _ in range(s["steps"]):
        s["sim"].step_cfl(CFL)
    here.wait_stream(s["stream"])
    return s["fields"].all()


# -------------------------------------------------------------------- work
def work(case):
    """One step reads vx, vy, p and the flag and writes vx, vy and p.  Its
    arithmetic per cell: two diffusion sweeps of two components (32), three
    16-point samples for each of two faces (420), two V(3,3) cycles (165), the
    rest (15).  A tolerance solve does not say how many cycles it needs: it
    cannot do with less than the two of the fixed step.  The solver alone
    reads p, f and the flag and writes p."""
    kind = case["kind"]
    if kind == "mg":
        n = case["W"] * case["H"]
        return {"bytes": 13.0 * n, "flops": 83.0 * n * case["cycles"]}
    if kind in ("batch", "serve"):
        n = sum(W * H * k for W, H, _, _, k in _members(case, 1))
    else:
        n = case["W"] * case["H"] * case["steps"]
    flops = 632.0 if case.get("advect") != "bilinear" else 282.0
    return {"bytes": (41.0 if kind == "io" else 25.0) * n, "flops": flops * n}


# ------------------------------------------------------- the same in 64 bits
class _Mg64:
    """V(3,3) cycles of red-black Gauss-Seidel on flags (H, W)."""

    def __init__(self, flag):
        self.flag = [flag.double()]
        while min(self.flag[-1].shape) // 2 > 3:
            f = self.flag[-1]
            h, w = f.shape[0] // 2, f.shape[1] // 2
            c = torch.ones(h, w, dtype=torch.float64, device=f.device)
            c[1:-1, 1:-1] = (self._weigh(f, h, w) / 16.0 > 0.2).double()
            self.flag.append(c)
        self.mask = []
        for f in self.flag:
            h, w = f.shape
            odd = (torch.arange(h, device=f.device)[:, None] +
                   torch.arange(w, device=f.device)[None, :]) % 2 == 1
            self.mask.append(odd[1:-1, 1:-1])

    @staticmethod
    def _weigh(r, h, w):
        s = lambda dy, dx: r[2 + dy:2 * h - 3 + dy:2, 2 + dx:2 * w - 3 + dx:2]  # noqa: E731
        return (s(-1, -1) + s(-1, 1) + s(1, -1) + s(1, 1) + 4.0 * s(0, 0) +
                2.0 * (s(-1, 0) + s(1, 0) + s(0, -1) + s(0, 1)))

    @staticmethod
    def _around(a):
        return a[1:-1, :-2], a[1:-1, 2:], a[:-2, 1:-1], a[2:, 1:-1]

    def sweep(self, p, f, level, hh):
        flag, odd = self.flag[level], self.mask[level]
        n = sum(self._around(flag))
        keep = flag[1:-1, 1:-1] * (n > 0)
        n = n.clamp_min(1.0)
        for red in (odd, ~odd):
            v = sum(a * b for a, b in zip(self._around(p), self._around(flag)))
            v = keep * (v + f[1:-1, 1:-1] * hh * hh) / n
            p[1:-1, 1:-1] = torch.where(red, v, p[1:-1, 1:-1])

    @staticmethod
    def edges(p):
        p[1:-1, 0], p[1:-1, -1] = p[1:-1, 1].clone(), p[1:-1, -2].clone()
        p[0, 1:-1], p[-1, 1:-1] = p[1, 1:-1].clone(), p[-2, 1:-1].clone()

    def residual(self, p, f, level, hh):
        flag, c = self.flag[level], p[1:-1, 1:-1]
        v = sum((a - c) * b for a, b in zip(self._around(p), self._around(flag)))
        r = torch.zeros_like(p)
        r[1:-1, 1:-1] = (f[1:-1, 1:-1] + v / (hh * hh)) * flag[1:-1, 1:-1]
        return r

    def prolongate(self, ec, level, h, w):
        fc = self.flag[level + 1]
        e = torch.zeros(h, w, dtype=torch.float64, device=ec.device)
        for oy in (0, 1):
            for ox in (0, 1):
                y0, x0 = (1 if oy else 2), (1 if ox else 2)
                ys, xs = range(y0, h - 1 - oy, 2), range(x0, w - 1 - ox, 2)
                if not len(ys) or not len(xs):
                    continue
                s = lambda a, dy, dx: a[y0 // 2 + dy:y0 // 2 + dy + len(ys),  # noqa: E731
                                        x0 // 2 + dx:x0 // 2 + dx + len(xs)]
                at = [(dy, dx) for dy in range(oy + 1) for dx in range(ox + 1)]
                v = sum(s(ec, *d) for d in at)
                if oy or ox:
                    v = v / (sum(s(fc, *d) for d in at) + 0.0001)
                e[y0:h - 1 - oy:2, x0:w - 1 - ox:2] = v
        return e * self.flag[level]

    def cycle(self, p, f, hh, zgbc, level=0):
        h, w = p.shape
        if level == len(self.flag) - 2:
            for _ in range(5):
                self.sweep(p, f, level, hh)
            return
        bc = zgbc and level == 0

        def sweeps():
            for _ in range(3):
                self.sweep(p, f, level, hh)
                if bc:
                    self.edges(p)

        sweeps()
        r = self.residual(p, f, level, hh)
        hc, wc = h // 2, w // 2
        rc = torch.zeros(hc, wc, dtype=torch.float64, device=p.device)
        rc[1:-1, 1:-1] = self._weigh(r, hc, wc) / 16.0
        ec = torch.zeros_like(rc)
        self.cycle(ec, rc, hh * (w - 1.0) / (wc - 1.0), False, level + 1)
        p[1:-1, 1:-1] += self.prolongate(ec, level, h, w)[1:-1, 1:-1]
        if bc:
            self.edges(p)
        sweeps()


class _Sim64:
    """The fluid step: inflow in the west, outflow with zero pressure in the
    east, no slip in the north and south."""

    def __init__(self, flag, vx, vy, bilinear=False):
        self.flag, self.vx, self.vy = flag.double(), vx.double(), vy.double()
        self.H, self.W = flag.shape
        self.h, self.bilinear = PWIDTH / (self.W - 1.0), bilinear
        self.p = torch.zeros_like(self.flag)
        self.mg = _Mg64(flag)
        F_, W = self.flag, self.W
        self.mx, self.my = F_[:, :-1] * F_[:, 1:], F_[:-1] * F_[1:]
        # faces the back-trace covers: chunks of 8 from x = 1 that start
        # before width - 8 and hold a fluid pair
        self.ax = self._chunks(self.mx, W - 1)
        below = torch.zeros_like(F_)
        below[1:] = F_[1:] * F_[:-1]
        self.ay = self._chunks(torch.cat([below[:, 1:], below[:, :1] * 0], 1), W)[:-1]

    @staticmethod
    def _chunks(pair, width):
        """pair[y, x - 1]: whether lane x of a chunk is fluid."""
        h = pair.shape[0]
        out = torch.zeros(h, width, dtype=torch.bool, device=pair.device)
        n = len(range(1, width - 8, 8))
        if n:
            live = (pair[:, :8 * n].reshape(h, n, 8) > 0).any(2)
            out[:, 1:1 + 8 * n] = live.repeat_interleave(8, 1)
        return out

    @staticmethod
    def _out(a):
        return a.clamp_min(0.0)

    def vbc(self):
        vx, vy = self.vx, self.vy
        vx[:, -1] = self._out(vx[:, -2])
        vx[0], vx[-1] = -vx[1], -vx[-2]
        vy[:, -1] = self._out(vy[:, -2])
        vy[0], vy[-1] = 0.0, 0.0

    def diffuse(self, dt):
        a = dt * MU * (self.W - 1.0) / PWIDTH
        fl = self.flag
        old = None
        self.vbc()
        for _ in range(2):
            v, n = self.vx, self.vx.clone()
            c = v[1:-1, 1:-1]
            t = v[1:-1, 2:] * fl[1:-1, 2:-1] * fl[1:-1, 3:]
            t = t + v[1:-1, :-2] * fl[1:-1, 1:-2] * fl[1:-1, :-3]
            for s in (2, 0):
                f = fl[s:s + self.H - 2, 1:-2] * fl[s:s + self.H - 2, :-3]
                t = t + v[s:s + self.H - 2, 1:-1] * f - (1.0 - f) * c
            n[1:-1, 1:-1] = self.mx[1:-1, 1:-1] * (c + a * t) / (1.0 + 4.0 * a)
            v, m = self.vy, self.vy.clone()
            c = v[1:-1, 1:-1]
            t = v[:-2, 1:-1] * fl[1:-2, 1:-1] * fl[:-3, 1:-1]
            t = t + v[2:, 1:-1] * fl[2:-1, 1:-1] * fl[3:, 1:-1]
            for s in (2, 0):
                f = fl[1:-2, s:s + self.W - 2] * fl[2:-1, s:s + self.W - 2]
                t = t + v[1:-1, s:s + self.W - 2] * f - (1.0 - f) * c
            m[1:-1, 1:-1] = self.my[1:-1, 1:-1] * (c + a * t) / (1.0 + 4.0 * a)
            self.vx, self.vy = n, m
            self.vbc()
            old = old or (self.vx, self.vy)
        return old

    def sample(self, g, cx, cy):
        gh, gw = g.shape
        flat = g.reshape(-1)
        if self.bilinear:
            cx, cy = cx.clamp(0.0, gw - 1.1), cy.clamp(0.0, gh - 1.1)
        else:
            cx, cy = cx.clamp_max(gw - 3.0).clamp_min(3.0), cy.clamp_max(gh - 3.0).clamp_min(3.0)
        ix, iy = cx.long(), cy.long()
        sx, sy = cx - ix, cy - iy
        at = iy * gw + ix
        if self.bilinear:
            a = flat[at] + (flat[at + 1] - flat[at]) * sx
            b = flat[at + gw] + (flat[at + gw + 1] - flat[at + gw]) * sx
            return a + (b - a) * sy

        def weights(t):
            return (t * (-0.5 + t * (1.0 - 0.5 * t)), 1.0 + t * t * (-2.5 + 1.5 * t),
                    t * (0.5 + t * (2.0 - 1.5 * t)), t * t * (-0.5 + 0.5 * t))

        wx, wy, out = weights(sx), weights(sy), 0.0
        for j in range(4):
            out = out + wx[j] * sum(wy[i] * flat[at + (i - 1) * gw + j - 1] for i in range(4))
        return out

    def advect(self, dt, old, rows=256):
        """In strips of rows, to bound the memory of the temporaries."""
        vx, vy, dh = self.vx, self.vy, dt / self.h
        H, W, dev = self.H, self.W, vx.device
        nx, ny = old[0].clone(), old[1].clone()
        xs = torch.arange(W, dtype=torch.float64, device=dev)
        for y0 in range(1, H - 1, rows):
            y1 = min(H - 1, y0 + rows)
            y = torch.arange(y0, y1, dtype=torch.float64, device=dev)[:, None]

            def trace(px, py, u, v):
                mx, my = px - u * 0.5 * dh, py - v * 0.5 * dh
                u2 = self.sample(vx, mx - 0.5, my)
                v2 = self.sample(vy, mx, my - 0.5)
                return px - u2 * dh, py - v2 * dh

            u = vx[y0:y1, 1:-1]
            v = 0.25 * (vy[y0:y1, 1:-2] + vy[y0 - 1:y1 - 1, 1:-2] + vy[y0:y1, 2:-1] +
                        vy[y0 - 1:y1 - 1, 2:-1])
            ex, ey = trace(xs[1:W - 2] + 0.5, y, u, v)
            r = self.sample(vx, ex - 0.5, ey) * self.mx[y0:y1, 1:-1]
            nx[y0:y1, 1:-1] = torch.where(self.ax[y0:y1, 1:-1], r, nx[y0:y1, 1:-1])
            # the average of the vy faces at x = W-2 reads one element on in
            # the flat array, the first of the next row
            east = torch.cat([vx, torch.cat([vx[1:, :1], vx[-1:, :1]], 0)], 1)
            v = vy[y0:y1, 1:-1]
            u = 0.25 * (east[y0:y1, 1:W - 1] + east[y0 - 1:y1 - 1, 1:W - 1] +
                        east[y0:y1, 2:W] + east[y0 - 1:y1 - 1, 2:W])
            ex, ey = trace(xs[1:W - 1], y + 0.5, u, v)
            r = self.sample(vy, ex, ey - 0.5) * self.my[y0:y1, 1:-1]
            ny[y0:y1, 1:-1] = torch.where(self.ay[y0:y1, 1:-1], r, ny[y0:y1, 1:-1])
        # edges: those of the diffused field
        nx[0], nx[-1], nx[:, 0], nx[:, -1] = vx[0], vx[-1], vx[:, 0], vx[:, -1]
        self.vx, self.vy = nx, ny

    def gradient(self):
        p, ih = self.p, 1.0 / self.h
        self.vx[1:-1, 1:-1] -= self.mx[1:-1, 1:-1] * ih * (p[1:-1, 2:-1] - p[1:-1, 1:-2])
        self.vy[1:-1, 1:-1] -= self.my[1:-1, 1:-1] * ih * (p[2:-1, 1:-1] - p[1:-2, 1:-1])

    def solve(self, f):
        """The projection's exact solution: conjugate gradients on the
        zero-gradient system, the sum of f taken up at the outflow."""
        fl = self.flag[1:-1, 1:-1]
        inner = F.pad(fl, (1, 1, 1, 1))
        nb = self.mg._around(inner)
        op = lambda x: sum((x - a) * b for a, b in  # noqa: E731
                           zip(self.mg._around(F.pad(x, (1, 1, 1, 1))), nb)) * fl
        b = f[1:-1, 1:-1] * fl
        col = fl[:, -1:]
        b[:, -1:] -= b.sum() / col.sum().clamp_min(1.0) * col
        b = b * self.h * self.h
        x = torch.zeros_like(b)
        d = sum(nb).clamp_min(1.0)
        r, z = b.clone(), b / d
        q, rz, stop = z.clone(), (b * z).sum(), 1e-22 * (b * b).sum()
        for k in range(20000):
            s = op(q)
            al = rz / (q * s).sum()
            x += al * q
            r -= al * s
            if k % 50 == 49 and bool((r * r).sum() < stop):
                break
            z = r / d
            new = (r * z).sum()
            q, rz = z + (new / rz) * q, new
        self.p = F.pad(x, (1, 1, 1, 1))

    def step(self, tolerance=False):
        top = max(float(self.vx.abs().max()), float(self.vy.abs().max()), 1e-7)
        dt = CFL * self.h / top
        old = self.diffuse(dt)
        self.advect(dt, old)
        self.vbc()
        f = torch.zeros_like(self.p)
        f[1:-1, 1:-1] = -(self.vx[1:-1, 1:] - self.vx[1:-1, :-1] + self.vy[1:, 1:-1] -
                          self.vy[:-1, 1:-1]) / self.h
        if tolerance:
            self.solve(f)
        else:
            for _ in range(2):
                self.mg.cycle(self.p, f, self.h, True)
            p = self.p
            p[:, 0], p[:, -1] = p[:, 1].clone(), -p[:, -2]
            p[0], p[-1] = p[1].clone(), p[-2].clone()
        self.gradient()
        self.vbc()


def _steps64(W, H, seed, u_in, steps, **how):
    s = _Sim64(*_instance(W, H, seed, u_in), **how)
    for _ in range(steps):
        s.step()
    return [s.vx, s.vy, s.p]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("batch", "serve"):
        return [_steps64(*m) for m in _members(case, seed)]
    W, H = case["W"], case["H"]
    if kind == "step":
        return _steps64(W, H, seed, 1.0, case["steps"], bilinear=case["advect"] == "bilinear")
    flag, vx, vy = _instance(W, H, seed)
    if kind == "mg":
        f = torch.zeros(H, W, device="cuda")
        h = PWIDTH / (W - 1)
        f[1:-1, 1:-1] = -(vx[1:-1, 1:] - vx[1:-1, :-1] + vy[1:, 1:-1] - vy[:-1, 1:-1]) / h
        mg, p = _Mg64(flag), torch.zeros(H, W, dtype=torch.float64, device="cuda")
        for _ in range(case["cycles"]):
            mg.cycle(p, f.double(), h, case["zgbc"])
        return p
    s, out = _Sim64(flag, vx, vy), []
    if kind == "io":
        for k in range(case["steps"]):
            s.vx, s.vy = vx.double(), (vy * (1.0 - 0.1 * k)).double()
            s.step()
            out.append([s.vx.clone(), s.vy.clone()])
        return out
    if W * H > 600000:
        return None  # unpreconditioned conjugate gradients take too long
    for _ in range(case["steps"]):
        s.step(tolerance=True)
    return [s.vx, s.vy, None]  # p is known up to a constant on each region
