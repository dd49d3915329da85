"""Timing cases of the channel-DNS engine, through its public entry points.

A case is a dict of plain values:
  kind   "run"     upload a state, `steps` RK3 steps, download it (Engine.upload / .step, lh_download_state)
         "host"    lh_step_host: host buffers up, `steps` steps, down, in place (the Fortran drop-in call)
         "batch"   `steps` steps of a Batch of the instances in `members` ("16*32x32x153 ..."), all states down
         "solve"   lh_lusolu_noalloc on the caller's device arrays, velocity grid `grid_id`
         "sample"  a sampling window: `samples` times (spectra, stats and pressure snapshot of the state, then
                   `steps` steps), then the accumulators
  Nx, Nz, ny, tanh (the tanh(2) y grid instead of the polynomial one), re_tau,
  cfl (the CFL rule at 0.7) or a fixed dt, flowrate (constant flow rate instead
  of constant pressure gradient), steps.

`exact` restates the time step in plain torch float64 from the equations: RK3
with implicit viscous terms, 3/2-rule pseudo-spectral products, staggered
second-order differences in y, pressure projection.
"""
import ctypes
import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "final-single-block-_b200"))

MPGX, ALP, BET, CFL = -3.0675e-3, 1.0, 2.0, 0.7


def _case(name, kind, Nx, Nz, ny, steps, **more):
    c = dict(name=name, kind=kind, Nx=Nx, Nz=Nz, ny=ny, steps=steps, tanh=False, re_tau=180.0, cfl=False, dt=5e-4,
             flowrate=False)
    c.update(more)
    return c


def listed():
    return [
        # one step behind the Fortran driver of a minimal channel: launches and latency
        _case("host_16x16x97", "host", 16, 16, 97, 1, dt=1e-3),
        # the reference's own input deck (32^2 modes, CFL time step), 100 steps
        _case("run_32x32x153", "run", 32, 32, 153, 100, cfl=True),
        # a mid-size channel of the request grid
        _case("run_64x64x153", "run", 64, 64, 153, 40),
        # the headline plain workload
        _case("run_128x128x153", "run", 128, 128, 153, 25),
        # the two large request sizes, on the stretched tanh grid
        _case("run_192x192x257", "run", 192, 192, 257, 10, tanh=True, re_tau=550.0, dt=2.5e-4),
        _case("run_256x256x257", "run", 256, 256, 257, 10, tanh=True, re_tau=550.0, dt=2.5e-4),
        # a ragged one: unequal mode counts off the usual powers of two, odd rows, constant flow rate
        _case("run_72x48x101", "run", 72, 48, 101, 40, flowrate=True, dt=1e-3),
        # the drop-in call at the headline size: PCIe both ways every step
        _case("host_128x128x153", "host", 128, 128, 153, 1),
        # a parameter sweep of 64 small channels in shared launches
        dict(name="batch_64x32x32x153", kind="batch", members="64*32x32x153", tanh=False, steps=20),
        # the mixed batch: small, mid, headline and one large instance
        dict(name="batch_uneven", kind="batch", members="16*32x32x153 8*64x64x153 4*128x128x153 1*256x256x257",
             tanh=True, steps=4),
        # a Helmholtz solve inside a caller's own device loop
        dict(name="solve_128x128x153", kind="solve", Nx=128, Nz=128, ny=153, grid_id=2, substep=2, dt=5e-4, re_tau=180.0,
             tanh=False),
        # a statistics window of a rectangular box
        _case("sample_96x64x129", "sample", 96, 64, 129, 4, samples=4),
    ]


_SIZES = [16, 24, 32, 36, 48, 64, 72, 96, 108, 128, 144, 192, 216, 256]
_MOST = 256 * 256 * 257 * 10  # grid points x steps of the largest listed case


def _unnamed(*a, **more):
    c = _case("", *a, **more)
    del c["name"]
    return c


def draw(rng):
    kind = rng.choice(["run"] * 6 + ["host", "host", "batch", "batch", "solve", "sample"])
    Nx = rng.choice(_SIZES)
    Nz = Nx if rng.random() < 0.5 else rng.choice([n for n in _SIZES if Nx // 2 <= n <= 2 * Nx])
    ny = int(round(math.exp(rng.uniform(math.log(33), math.log(257)))))
    tanh, flowrate = rng.random() < 0.3, rng.random() < 0.2
    re_tau, dt = round(rng.uniform(100, 400), 3), round(rng.uniform(2e-4, 5e-4), 6)
    if kind == "solve":
        return dict(kind="solve", Nx=min(Nx, 128), Nz=min(Nz, 128), ny=min(ny, 200), grid_id=rng.choice([1, 2]),
                    substep=rng.choice([1, 2, 3]), dt=dt, re_tau=re_tau, tanh=tanh)
    if kind == "batch":
        m = []
        for _ in range(rng.choice([1, 2, 3])):
            n = rng.choice([16, 24, 32, 48, 64])
            m.append("%d*%dx%dx%d" % (rng.randint(2, 12), n, n, rng.randint(33, 193)))
        return dict(kind="batch", members=" ".join(m), tanh=tanh, steps=rng.randint(4, 12))
    points = Nx * Nz * ny
    if kind == "host":
        return _unnamed("host", Nx, Nz, ny, 1, tanh=tanh, re_tau=re_tau, dt=dt, flowrate=flowrate)
    steps = max(2, min(40, int(_MOST * rng.uniform(0.1, 0.6) / points)))
    if kind == "sample":
        Nx, Nz = min(Nx, 128), min(Nz, 128)
        return _unnamed("sample", Nx, Nz, ny, 2, tanh=tanh, re_tau=re_tau, dt=dt, samples=3)
    cfl = rng.random() < 0.25
    if cfl:
        re_tau = min(re_tau, 200.0)
    return _unnamed("run", Nx, Nz, ny, steps, tanh=tanh, re_tau=re_tau, dt=dt, cfl=cfl, flowrate=flowrate)


# ---- inputs ----------------------------------------------------------------
def _re(re_tau):
    return re_tau / math.sqrt(-MPGX)


def _y_grid(ny, tanh):
    """yu, yv and dtheta/dy of both grids: v faces 0..ny-1, u centres around them."""
    n, q = ny - 1, (ny - 1) / 2.0
    tv, tu = np.arange(n + 1) - q, np.arange(n + 2) - 0.5 - q
    if tanh:
        g, t = 2.0, math.tanh(2.0)
        y = lambda s: np.tanh(g * s / q) / t  # noqa: E731
        d = lambda s: q * t / (g * (1.0 - np.tanh(g * s / q) ** 2))  # noqa: E731
    else:
        m, r = 5, 10.0
        b = (r - 1) / (q * (1 - q ** (m - 1) + r * ((1 - q) * q ** (m - 1) - (1 - q) ** m)))
        a = (1 - b * q ** m) / q
        y = lambda s: a * s + b * s ** m  # noqa: E731
        d = lambda s: 1.0 / (a + m * b * s ** (m - 1))  # noqa: E731
    return y(tu), y(tv), d(tu), d(tv)


def _wavenumbers(Nx, Nz):
    kx = ALP * np.arange(Nx // 2 + 1)
    kz = BET * np.where(np.arange(Nz) < Nz // 2, np.arange(Nz), np.arange(Nz) - Nz)
    return kx, kz


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _initial(Nx, Nz, ny, tanh, re, seed):
    """Perturbed laminar u1, u2, u3 and a zero p, [column, row] on the GPU: one
    complex Gaussian coefficient per mode, 0.05 exp(-(kx^2+kz^2)/16) (1-y^2)^2."""
    dev = _device()
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed * 2654435761 % (1 << 62))
    yu, yv, _, _ = _y_grid(ny, tanh)
    kx, kz = _wavenumbers(Nx, Nz)
    env = torch.as_tensor(0.05 * np.exp(-(kx[None, :] ** 2 + kz[:, None] ** 2) / 16.0), device=dev)
    out = []
    for y in (yu, yv, yu):
        g = torch.randn(Nz, Nx // 2 + 1, 2, generator=gen, device=dev, dtype=torch.float64)
        a = env * torch.view_as_complex(g)
        a[0, 0] = 0.0  # the mean mode carries the mean profile
        a[Nz // 2 + 1:, 0] = torch.conj(a[1:Nz // 2, 0].flip(0))  # real in physical space
        a[Nz // 2, 0] = a[Nz // 2, 0].real.clone()
        prof = torch.as_tensor((1.0 - np.clip(y, -1, 1) ** 2) ** 2, device=dev)
        out.append(a.reshape(-1, 1) * prof[None, :])
    out[0][0] += torch.as_tensor(0.5 * re * MPGX * (yu ** 2 - 1.0), device=dev)
    gw = (yu[0] - yv[0]) / (yu[1] - yv[0])
    for u in (out[0], out[2]):
        u[:, 0] = gw * u[:, 1]
        u[:, -1] = gw * u[:, -2]
    out[1][:, 0] = 0.0
    out[1][:, -1] = 0.0
    out.append(torch.zeros(out[0].shape[0], ny - 1, dtype=torch.complex128, device=dev))
    return out


def _pinned(x):
    h = torch.empty(x.shape, dtype=x.dtype, pin_memory=torch.cuda.is_available())
    h.copy_(x)
    return h


def _ptr(t):
    return ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_double))


def _desc(c):
    from lh_b200 import Desc
    return Desc(Nx=c["Nx"], Nz=c["Nz"], ny=c["ny"], Re=_re(c["re_tau"]), alp=ALP, bet=BET, mpgx=MPGX,
                flag_ctpress=0 if c.get("flowrate") else 1, grid_type=1 if c["tanh"] else 0, gamma=2.0,
                dt_mode=0 if c.get("cfl") else 1, CFL=CFL, dt=c["dt"])


def _members(case, seed):
    """The batch's instances as case dicts, Re_tau and dt of each from the seed."""
    r, out = random.Random(seed), []
    for k, part in enumerate(case["members"].split()):
        count, size = part.split("*")
        Nx, Nz, ny = (int(v) for v in size.split("x"))
        for _ in range(int(count)):
            out.append(dict(Nx=Nx, Nz=Nz, ny=ny, tanh=case["tanh"], re_tau=r.uniform(100, 400), dt=r.uniform(2e-4, 5e-4),
                            cls=k, seed=r.randrange(1 << 40)))
    return out


def prepare(case, seed):
    from lh_b200 import Batch, Engine
    kind = case["kind"]
    if kind == "batch":
        b, mem = Batch(), _members(case, seed)
        for m in mem:
            ic = [x.cpu().numpy() for x in _initial(m["Nx"], m["Nz"], m["ny"], m["tanh"], _re(m["re_tau"]), m["seed"])]
            m["slot"] = b.add(_desc(m), *ic)
        outs = {}
        for k in sorted({m["cls"] for m in mem}):
            own = [m for m in mem if m["cls"] == k]
            nc, ny = (own[0]["Nx"] // 2 + 1) * own[0]["Nz"], own[0]["ny"]
            outs[k] = [_pinned(torch.zeros(len(own), nc, rows, dtype=torch.complex128)) for rows in (ny + 1, ny, ny + 1, ny - 1)]
        where = []
        for k in outs:
            for i, m in enumerate(m for m in mem if m["cls"] == k):
                where.append((m["slot"], [_ptr(x[i]) for x in outs[k]]))
        return dict(kind=kind, batch=b, where=where, out=[x for k in sorted(outs) for x in outs[k]], steps=case["steps"])
    e = Engine(_desc(case))
    if kind == "solve":
        rows = case["ny"] + (1 if case["grid_id"] == 2 else 0)
        nc = (case["Nx"] // 2 + 1) * case["Nz"]
        rhs = _solve_rhs(rows, nc, seed)
        u = torch.zeros_like(rhs)
        torch.cuda.synchronize()
        stream = torch.cuda.ExternalStream(e.stream())
        return dict(kind=kind, engine=e, rhs=rhs, u=u, args=(case["grid_id"], case["substep"], case["dt"]), stream=stream)
    ic = [_pinned(x) for x in _initial(case["Nx"], case["Nz"], case["ny"], case["tanh"], _re(case["re_tau"]), seed)]
    out = ic if kind == "host" else [_pinned(torch.zeros(x.shape, dtype=x.dtype)) for x in ic]
    return dict(kind=kind, engine=e, ic=[x.numpy() for x in ic], keep=ic, out=out, ptr=[_ptr(x) for x in out],
                steps=case["steps"], samples=case.get("samples", 0))


def _solve_rhs(rows, nc, seed):
    gen = torch.Generator(device=_device())
    gen.manual_seed(seed)
    return torch.view_as_complex(torch.randn(rows, nc, 2, generator=gen, device=_device(), dtype=torch.float64))


def run(s):
    kind = s["kind"]
    if kind == "batch":
        b = s["batch"]
        b.step(s["steps"])
        for slot, p in s["where"]:
            if b.L.lh_batch_download(b.h, slot, *p) != 0:
                raise RuntimeError(b.L.lh_batch_last_error(b.h).decode())
        return s["out"]
    e = s["engine"]
    if kind == "solve":
        rc = e.L.lh_lusolu_noalloc(e.h, *s["args"], s["rhs"].data_ptr(), s["u"].data_ptr())
        if rc != 0:
            raise RuntimeError(e.L.lh_last_error(e.h).decode())
        torch.cuda.current_stream().wait_stream(s["stream"])
        return s["u"]
    if kind == "host":
        e.step_host(s["ic"], s["steps"])
        return s["out"]
    e.upload(*s["ic"])
    if kind == "sample":
        e.spectra_reset()
        e.stats_reset()
        for _ in range(s["samples"]):
            e.pressure_snapshot()
            e.spectra_accumulate()
            e.stats_accumulate()
            e.step(s["steps"])
        return {"stats": e.stats()[0], "spectra": e.spectra()[0]}
    e.step(s["steps"])
    if e.L.lh_download_state(e.h, *s["ptr"]) != 0:
        raise RuntimeError(e.L.lh_last_error(e.h).decode())
    return s["out"]


# ---- what a pass cannot do without -------------------------------------------
def _step_work(Nx, Nz, ny):
    """Bytes and float64 operations of one RK3 step of one instance: per substep
    u, w, v, p and the nonlinear terms read and written once by the column
    solves and u, w, v read and the nonlinear terms written once by the
    transforms (20 fields); transforms at 5 n log2 n, products, solves."""
    nxh, Mx, Mz = Nx // 2 + 1, 3 * Nx // 2, 3 * Nz // 2
    field = 16.0 * nxh * Nz * ny
    ffts = 9 * nxh * 5 * Mz * math.log2(Mz) + 6 * Mz * 5 * Mx * math.log2(Mx) + 6 * Mx * Mz
    return 3 * 20 * field, 3 * ny * (ffts + 200.0 * nxh * Nz)


def work(case):
    if case["kind"] == "solve":
        n = (case["Nx"] // 2 + 1) * case["Nz"] * (case["ny"] + (1 if case["grid_id"] == 2 else 0))
        return {"bytes": 32.0 * n, "flops": 24.0 * n}
    if case["kind"] == "batch":
        members, passes = _members(case, 0), case["steps"]
    else:
        members, passes = [case], case["steps"] * max(1, case.get("samples", 0))
    b = f = 0.0
    for m in members:
        sb, sf = _step_work(m["Nx"], m["Nz"], m["ny"])
        state = 4 * 16.0 * (m["Nx"] // 2 + 1) * m["Nz"] * m["ny"]
        b += passes * sb + (1 if case["kind"] == "batch" else 2) * state
        f += passes * sf
    return {"bytes": b, "flops": f}


# ---- the same in plain torch ---------------------------------------------------
class _Channel:
    """Instances of one size side by side, fields [instance, row, kz, kx]."""

    RK = [(4 / 15, 4 / 15, 8 / 15, 0.0, 8 / 15), (1 / 15, 1 / 15, 5 / 12, -17 / 60, 2 / 15), (1 / 6, 1 / 6, 3 / 4, -5 / 12, 1 / 3)]

    def __init__(self, Nx, Nz, ny, tanh, re, dt, cfl, flowrate, states):
        self.Nx, self.Nz, self.Mx, self.Mz, self.ny = Nx, Nz, 3 * Nx // 2, 3 * Nz // 2, ny
        self.nyu, self.cfl, self.flowrate = ny - 1, cfl, flowrate
        dev = self.dev = states[0][0].device
        t = lambda a: torch.as_tensor(np.asarray(a, np.float64), device=dev)  # noqa: E731
        self.yu, self.yv, self.thu, self.thv = (t(a) for a in _y_grid(ny, tanh))
        kx, kz = _wavenumbers(Nx, Nz)
        self.kx, self.kz = t(kx), t(kz)[:, None]
        self.k2 = -(self.kx ** 2 + self.kz ** 2)
        self.mask = torch.ones(Nz, 1, dtype=torch.float64, device=dev)
        self.mask[Nz // 2] = 0.0  # no derivative on the kz = -Nz/2 row
        col = lambda v: t(v).reshape(-1, 1, 1, 1)  # noqa: E731
        self.re, self.dt = col(re), col(dt)
        self.mpgx = torch.full_like(self.re, MPGX)
        yu, yv = self.yu, self.yv
        self.gw = (-(yv[0] - yu[0]) / (yv[0] - yu[1]), (yu[-1] - yv[-1]) / (yv[-1] - yu[-2]))
        self.gwbc = (yu[0] - yv[0]) / (yu[1] - yv[0])
        self.dtv = self.re / (-self.k2[0, Nx // 2] + (BET * (Nz // 2 - 1)) ** 2 + 4.0 / (yv[1] - yv[0]) ** 2)
        shape = lambda f: torch.stack([s[f] for s in states]).transpose(1, 2).reshape(len(states), -1, Nz, Nx // 2 + 1).contiguous()  # noqa: E731
        self.u1, self.u2, self.u3, self.p = (shape(f) for f in range(4))
        self.nu = [torch.zeros_like(self.p), torch.zeros_like(self.p[:, 1:]), torch.zeros_like(self.p)]
        self.factors = {}
        # d2/dy2 at the interior rows of both grids
        self.d2 = []
        for y in (yu, yv):
            a, b = y[1:-1] - y[:-2], y[2:] - y[1:-1]
            self.d2.append((2 / (a * (a + b)), -2 / (a * b), 2 / (b * (a + b))))
        self.qt = self.flow(self.u1[:, :, 0, 0].real)
        self.poisson = self.poisson_factors()

    def flow(self, u):
        return (u[:, 1:self.nyu + 1] * (self.yv[1:] - self.yv[:-1])).sum(1)

    # tridiagonal systems a1 x(j-1) + a2 x(j) + a3 x(j+1): factors, then solves, along dim 1
    @staticmethod
    def factor(a1, a2, a3):
        inv, up = [], []
        for j in range(len(a2)):
            inv.append(1.0 / (a2[j] if j == 0 else a2[j] - a1[j] * up[-1]))
            up.append(a3[j] * inv[-1])
        return a1, inv, up

    @staticmethod
    def solve(f, r):
        a1, inv, up = f
        x = list(r.unbind(1))
        x[0] = x[0] * inv[0]
        for j in range(1, len(x)):
            x[j] = (x[j] - a1[j] * x[j - 1]) * inv[j]
        for j in range(len(x) - 2, -1, -1):
            x[j] = x[j] - up[j] * x[j + 1]
        return torch.stack(x, 1)

    def poisson_factors(self):
        th, tv, n = self.thu, self.thv, self.nyu
        a1, a2, a3 = [], [], []
        for j in range(1, n + 1):
            lo = th[j] * tv[j - 1] if j > 1 else 0.0 * th[j]
            hi = th[j] * tv[j] if j < n else 0.0 * th[j]
            a1.append(lo)
            a2.append(-(lo + hi) + self.k2)
            a3.append(torch.ones_like(self.k2) * hi)
        a2[0] = a2[0].clone()
        a2[0][0, 0] = 1.0 / (self.yu[2] - self.yu[1]) ** 2  # gauge of the mean mode
        a3[0] = a3[0].clone()
        a3[0][0, 0] = 0.0
        return self.factor(a1, a2, a3)

    def helmholtz(self, grid, beta):
        d1, d2, d3 = self.d2[grid]
        b, one = beta[:, 0], torch.ones_like(beta[:, 0])
        g1, g2 = self.gw if grid == 0 else (0.0, 0.0)
        a1 = [0.0 * one] + [-b * v for v in d1] + [g2 * one]
        a2 = [one] + [1.0 - b * (v + self.k2) for v in d2] + [one]
        a3 = [g1 * one] + [-b * v for v in d3] + [0.0 * one]
        return self.factor(a1, a2, a3)

    def phys(self, f):
        h, Nz = self.Nz // 2, self.Nz
        z = torch.zeros(*f.shape[:2], self.Mz, f.shape[3], dtype=f.dtype, device=self.dev)
        z[:, :, :h] = f[:, :, :h]
        z[:, :, self.Mz - h:] = f[:, :, Nz - h:]
        z = torch.fft.ifft(z, dim=2, norm="forward")
        z[..., 0] = z[..., 0].real.clone()
        return torch.fft.irfft(z, n=self.Mx, dim=3, norm="forward")

    def modes(self, x):
        h = self.Nz // 2
        f = torch.fft.fft(torch.fft.rfft(x, dim=3, norm="forward")[..., :self.Nx // 2 + 1], dim=2, norm="forward")
        return torch.cat([f[:, :, :h], f[:, :, self.Mz - h:]], 2)

    def centre(self, v):
        """v faces to u centres 1..nyu."""
        d = (self.yv[1:] - self.yv[:-1]).reshape(-1, 1, 1)
        w = (self.yu[1:-1] - self.yv[:-1]).reshape(-1, 1, 1)
        return (w * v[:, 1:] + (d - w) * v[:, :-1]) / d

    def face(self, u):
        """u centres to v faces 0..nyu."""
        d = (self.yu[1:] - self.yu[:-1]).reshape(-1, 1, 1)
        w = (self.yv - self.yu[:-1]).reshape(-1, 1, 1)
        return (w * u[:, 1:] + (d - w) * u[:, :-1]) / d

    def substep(self, k):
        a, b, g, c, d = self.RK[k]
        r = lambda v: v.reshape(-1, 1, 1)  # noqa: E731
        n, ikx, ikz = self.nyu, 1j * self.kx, 1j * self.kz
        u1, u2, u3, p = self.u1, self.u2, self.u3, self.p
        # products on the dealiased grid: centres, then faces 1..nyu
        x1, x3, x2 = self.phys(u1[:, 1:-1]), self.phys(u3[:, 1:-1]), self.phys(self.centre(u2))
        if k == 0 and self.cfl:
            wall = [torch.view_as_real(u[:, 0]).abs().amax((1, 2, 3)) for u in (u1, u3)]
            m = [torch.maximum(w, x[:, :n - 1].abs().amax((1, 2, 3))) for w, x in zip(wall, (x1, x3))]
            dtc = torch.minimum(1 / (ALP * (self.Nx // 2) * m[0]), 1 / (BET * (self.Nz // 2) * m[1]))
            self.dt = torch.minimum(2.5 * self.dtv, CFL * dtc.reshape(-1, 1, 1, 1))
            self.factors = {}
        uu, uw, vv, ww = self.modes(x1 * x1), self.modes(x1 * x3), self.modes(x2 * x2), self.modes(x3 * x3)
        del x1, x2, x3
        y2 = self.phys(u2[:, 1:])
        uv = self.modes(self.phys(self.face(u1)[:, 1:]) * y2)
        wv = self.modes(self.phys(self.face(u3)[:, 1:]) * y2)
        del y2
        nil = torch.zeros_like(uv[:, :1])
        dy = lambda f: torch.diff(torch.cat([nil, f], 1), dim=1) * r(self.thu[1:-1])  # noqa: E731
        nu = [self.mask * (ikx * uu + ikz * uw) + dy(uv),
              self.mask * (ikx * uv + ikz * wv)[:, :-1] + torch.diff(vv, dim=1) * r(self.thv[1:-1]),
              self.mask * (ikx * uw + ikz * ww) + dy(wv)]
        del uu, uw, vv, ww, uv, wv
        lap = lambda f, q: r(q[0]) * f[:, :-2] + (self.k2 + r(q[1])) * f[:, 1:-1] + r(q[2]) * f[:, 2:]  # noqa: E731
        dt, du = self.dt, self.d2[0]
        du1 = a / self.re * lap(u1, du) - c * self.nu[0] - d * ikx * p - g * nu[0]
        du1[:, :, 0, 0] -= (d * self.mpgx)[:, :, 0, 0]
        du3 = a / self.re * lap(u3, du) - c * self.nu[2] - d * ikz * p - g * nu[2]
        du2 = a / self.re * lap(u2, self.d2[1]) - c * self.nu[1] - d * r(self.thv[1:-1]) * torch.diff(p, dim=1) - g * nu[1]
        self.nu = nu
        beta = b * dt / self.re
        if k not in self.factors:
            self.factors[k] = (self.helmholtz(0, beta), self.helmholtz(1, beta))
        fu, fv = self.factors[k]
        pad = lambda u, q: torch.cat([0 * u[:, :1], u[:, 1:-1] + dt * q, 0 * u[:, :1]], 1)  # noqa: E731
        u1, u3, u2 = self.solve(fu, pad(u1, du1)), self.solve(fu, pad(u3, du3)), self.solve(fv, pad(u2, du2))
        del du1, du2, du3
        if self.flowrate:
            zero = ([v[:, :1, :1] if v.dim() else v for v in x] for x in fu)  # the mean mode's factors
            e = torch.ones(u1.shape[0], n + 2, 1, 1, dtype=torch.float64, device=self.dev) * (-d * dt)
            e[:, 0] = 0.0
            e[:, -1] = 0.0
            e = self.solve(tuple(zero), e)[:, :, 0, 0]
            q1 = (e[:, :n] * (self.yv[1:] - self.yv[:-1])).sum(1)
            s = (self.qt - self.flow(u1[:, :, 0, 0].real)) / q1
            self.mpgx = self.mpgx + s.reshape(-1, 1, 1, 1)
            u1[:, :, 0, 0] += s[:, None] * e
        div = ikx * u1[:, 1:-1] + ikz * u3[:, 1:-1] + r(self.thu[1:-1]) * torch.diff(u2, dim=1)
        h = dt * (a + b)
        psi = div / h
        psi[:, 0, 0, 0] = 0.0
        psi = self.solve(self.poisson, psi)
        self.p = p + psi
        for u, ik in ((u1, ikx), (u3, ikz)):
            u[:, 1:-1] -= h * ik * psi
            u[:, 0] = self.gwbc * u[:, 1]
            u[:, -1] = self.gwbc * u[:, -2]
        u2[:, 1:-1] -= h * r(self.thv[1:-1]) * torch.diff(psi, dim=1)
        u2[:, 0] = 0.0
        u2[:, -1] = 0.0
        self.u1, self.u2, self.u3 = u1, u2, u3

    def step(self, steps):
        for _ in range(steps):
            for k in range(3):
                self.substep(k)

    def fields(self):
        """u1, u2, u3, p as [instance, column, row]."""
        return [f.flatten(2).transpose(1, 2).contiguous() for f in (self.u1, self.u2, self.u3, self.p)]

    def spectra(self):
        sq = lambda f: torch.view_as_real(f).square().sum(-1)  # noqa: E731
        yu, yv = self.yu, self.yv
        i = self.centre(self.u2)
        lo = (yu[0] - yu[1]) / (yv[0] - yu[1]) * (self.u2[:, :1] - i[:, :1]) + i[:, :1]
        hi = (yu[-1] - yu[-2]) / (yv[-1] - yu[-2]) * (self.u2[:, -1:] - i[:, -1:]) + i[:, -1:]
        i = torch.cat([lo, i, hi], 1)
        uv = self.u1.real * i.real + self.u1.imag * i.imag
        out = dict(spU=sq(self.u1), spV=sq(self.u2), spW=sq(self.u3), spUV=uv, spP=sq(self.p))
        return {k: v[0].flatten(1).transpose(0, 1) for k, v in out.items()}

    def stats(self):
        """The thirteen plane sums: physical values on planes 1..nyu, the
        coefficients themselves on the wall planes, p's coefficients, omega_x."""
        n, out = self.nyu, torch.zeros(13, self.nyu + 2, dtype=torch.float64, device=self.dev)
        s = lambda x: x.sum((-2, -1))[0]  # noqa: E731
        raw = lambda f: torch.view_as_real(f).flatten(2)[0]  # noqa: E731
        yu, yv = self.yu, self.yv
        a, w, vc = self.phys(self.u1[:, 1:-1]), self.phys(self.u3[:, 1:-1]), self.phys(self.centre(self.u2))
        v, wf = self.phys(self.u2[:, 1:]), self.phys(self.face(self.u3)[:, 1:])
        for q, x in enumerate((a, a * a, v, v * v, w, w * w, a * vc, a * w, v * wf)):
            out[q, 1:n + 1] = s(x)
        i = self.centre(self.u2)
        lo = (yu[0] - yu[1]) / (yv[0] - yu[1]) * (self.u2[:, 0] - i[:, 0]) + i[:, 0]
        hi = (yu[-1] - yu[-2]) / (yv[-1] - yu[-2]) * (self.u2[:, -1] - i[:, -1]) + i[:, -1]
        f0 = self.face(self.u3)[:, 0]
        nil = torch.zeros_like(f0)
        for j, a, v, w, vc, wf in ((0, self.u1[:, 0], self.u2[:, 0], self.u3[:, 0], lo, f0),
                                   (n + 1, self.u1[:, -1], nil, self.u3[:, -1], hi, nil)):
            a, v, w, vc, wf = (torch.view_as_real(x)[0].flatten() for x in (a, v, w, vc, wf))
            for q, x in enumerate((a, a * a, v, v * v, w, w * w, a * vc, a * w, v * wf)):
                out[q, j] = x.sum()
        p = raw(self.p).flatten(1)
        out[9, 1:n + 1], out[10, 1:n + 1] = p.sum(1), p.square().sum(1)
        o = -1j * self.kz * self.u2 + torch.diff(self.u3, dim=1) * self.thv.reshape(-1, 1, 1)
        o = torch.fft.ifft(o, dim=2, norm="forward")
        o[..., 0] = o[..., 0].real.clone()
        o = torch.fft.irfft(o, n=self.Nx, dim=3, norm="forward")
        out[11, :n + 1], out[12, :n + 1] = s(o), s(o * o)
        return out


def exact(case, seed):
    if case["kind"] == "solve":
        nxh, Nz = case["Nx"] // 2 + 1, case["Nz"]
        nil = [torch.zeros(nxh * Nz, r, dtype=torch.complex128, device=_device()) for r in (case["ny"] + 1, case["ny"], case["ny"] + 1, case["ny"] - 1)]
        ch = _Channel(case["Nx"], Nz, case["ny"], case["tanh"], [_re(case["re_tau"])], [case["dt"]], False, False, [nil])
        rows = case["ny"] + (1 if case["grid_id"] == 2 else 0)
        rhs = _solve_rhs(rows, nxh * Nz, seed).reshape(1, rows, Nz, nxh)
        f = ch.helmholtz(0 if case["grid_id"] == 2 else 1, ch.RK[case["substep"] - 1][1] * ch.dt / ch.re)
        return ch.solve(f, rhs).reshape(rows, nxh * Nz)
    if case["kind"] == "batch":
        out = []
        mem = _members(case, seed)
        for k in sorted({m["cls"] for m in mem}):
            own = [m for m in mem if m["cls"] == k]
            m = own[0]
            re = [_re(x["re_tau"]) for x in own]
            states = [_initial(m["Nx"], m["Nz"], m["ny"], m["tanh"], r, x["seed"]) for r, x in zip(re, own)]
            ch = _Channel(m["Nx"], m["Nz"], m["ny"], m["tanh"], re, [x["dt"] for x in own], False, False, states)
            ch.step(case["steps"])
            out += ch.fields()
        return out
    re = _re(case["re_tau"])
    state = _initial(case["Nx"], case["Nz"], case["ny"], case["tanh"], re, seed)
    ch = _Channel(case["Nx"], case["Nz"], case["ny"], case["tanh"], [re], [case["dt"]], case["cfl"], case["flowrate"], [state])
    if case["kind"] == "sample":
        st, sp = 0.0, {}
        for _ in range(case["samples"]):
            for k, v in ch.spectra().items():
                sp[k] = sp.get(k, 0.0) + v
            st = st + ch.stats()
            ch.step(case["steps"])
        return {"stats": st, "spectra": {k: v.contiguous() for k, v in sp.items()}}
    ch.step(case["steps"])
    return [f[0] for f in ch.fields()]
