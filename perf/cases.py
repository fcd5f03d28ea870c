"""Performance cases of the channel-flow LES library.

A pass of a stepping case is what a run does between two records of its
history: a block of RK3 steps, the statistics of the last one and a snapshot
of the state read back into pinned host memory.  The three forms (FP64,
mixed, mixed with the learned closure) run over the grids of the tests, the
benchmark channels and the training run, from launch-bound to
bandwidth-bound; the six reference-named stage entry points (the Fortran
host's loop) run the Smagorinsky closure and the Deardorff closure with shear
production.  The operator entry points and the training of the network are
cases of their own.

`exact` is the same computation in plain torch at 64 bits, on the level-by-
level form of the stage (no code of the library).
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DEV = "cuda:0"
XL, YL, ZL = 2 * math.pi, math.pi, 2.0
UTAU, EMIN, FORCING = math.sqrt(0.016), 1e-6, 0.016
GRID = (16, 32, 64, 96, 128, 192, 256, 384, 512)  # nnx, nny the library takes
NIN, NOUT, HID = 11, 6, 64


def host():
    name = "les_gpu_host"
    if name not in sys.modules:
        spec = importlib.util.spec_from_file_location(name, os.path.join(ROOT, "paes-channelflow_b200", "les_gpu.py"))
        sys.modules[name] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(sys.modules[name])
    return sys.modules[name]


def step_case(name, form, nx, ny, nz, steps, re_tau, floor=False):
    return {"name": name, "kind": "step", "form": form, "nx": nx, "ny": ny, "nz": nz, "steps": steps,
            "re_tau": re_tau, "tke_floor": floor}


def listed():
    return [
        # the smallest grid of the tests: launches and latency
        step_case("step fp64 32x32x16", "fp64", 32, 32, 16, 8, 180.0),
        # the two FP64 drop-in channels that are checked against the reference
        step_case("step fp64 64x64x64", "fp64", 64, 64, 64, 8, 180.0),
        step_case("step fp64 128x128x96", "fp64", 128, 128, 96, 8, 395.0),
        # the mixed-precision validation channel
        step_case("step mixed 256x256x128", "mixed", 256, 256, 128, 8, 590.0),
        # the production grid of the benchmark in its three forms
        step_case("step fp64 512x512x256", "fp64", 512, 512, 256, 8, 590.0),
        step_case("step mixed 512x512x256", "mixed", 512, 512, 256, 8, 590.0),
        step_case("step learned 512x512x256", "learned", 512, 512, 256, 8, 590.0),
        # the learned closure off the benchmark grid, nz odd
        step_case("step learned 256x192x99", "learned", 256, 192, 99, 4, 395.0),
        # late in a run without shear production: the TKE has decayed to its
        # floor, so its padded field is clipped on every level (in 64 bits: in
        # 32 a TKE that small is mostly rounding)
        step_case("step fp64 384x192x101 floor", "fp64", 384, 192, 101, 8, 395.0, True),
        # the Fortran host's loop over the six stage routines
        {"name": "split smag 96x128x45", "kind": "split", "imodel": 4, "production": False, "nx": 96, "ny": 128,
         "nz": 45, "steps": 4, "re_tau": 180.0},
        # dealiasing and derivatives for callers that keep their own state
        {"name": "operators f64 256x128x24", "kind": "ops", "bits": 64, "nx": 256, "ny": 128, "planes": 24},
        # an epoch's slice of closure training at the trained batch size
        {"name": "train 65536", "kind": "train", "batch": 65536, "steps": 16},
    ]


def draw(rng):
    kind = rng.choice(("fp64", "fp64", "mixed", "mixed", "learned", "learned", "split", "ops", "train"))
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if kind == "ops":
        return {"kind": "ops", "bits": rng.choice((32, 64)), "nx": rng.choice(GRID), "ny": rng.choice(GRID),
                "planes": log(1, 64)}
    if kind == "train":
        return {"kind": "train", "batch": log(1000, 131072), "steps": rng.choice((4, 8, 16))}
    if kind == "split":
        return {"kind": "split", "imodel": rng.choice((3, 4)), "production": rng.random() < 0.5,
                "nx": rng.choice(GRID[1:7]), "ny": rng.choice(GRID[1:7]), "nz": log(8, 96), "steps": 4,
                "re_tau": rng.choice((180.0, 395.0))}
    if kind == "learned":  # grids at least as fine as the closure's training data
        c = step_case("", kind, rng.choice(GRID[5:]), rng.choice(GRID[5:]), log(96, 256), 4, rng.choice((395.0, 590.0)))
    else:
        c = step_case("", kind, rng.choice(GRID[1:]), rng.choice(GRID[1:]), log(8, 256), 8,
                      rng.choice((180.0, 395.0, 590.0)), kind == "fp64" and rng.random() < 0.3)
    del c["name"]
    return c


def work(case):
    if case["kind"] == "ops":
        nx, ny, n, rb = case["nx"], case["ny"], case["planes"], case["bits"] // 8
        s, l = nx * ny * n, 9 * nx * ny * n // 4
        lg = 2.5 * math.log2(1.5 * math.sqrt(nx * ny))
        # expand, compress, deal of the small planes, both derivatives of the padded ones
        return {"bytes": (6 * s + 6 * l) * rb, "flops": lg * (8 * s + 12 * l)}
    if case["kind"] == "train":
        n, per = case["batch"], 2 * (16 * HID + 2 * HID * HID + HID * 16)
        return {"bytes": n * (32 + 32) * (case["steps"] + 2) + n * 32, "flops": n * per * (3 * (case["steps"] + 1) + 1)}
    pts = case["nx"] * case["ny"] * case["nz"]
    rb = 8 if case.get("form", "fp64") == "fp64" else 4
    # per point and step: three stages reading u, v, w, e and the old
    # tendencies and writing them back, the pressure solve's four 64-bit values
    per = 480 if rb == 8 else 288
    net = 3 * 18560 if case.get("form") == "learned" else 0
    return {"bytes": pts * (per * case["steps"] + 4 * rb), "flops": pts * case["steps"] * (12700.0 + net)}


# ------------------------------------------------------------------ inputs
def z0_of(case):
    return math.exp(-0.4 * 5.0) / case["re_tau"]


def turbulence(nz, ny, nx, g):
    """A smooth random field of unit variance, periodic in all directions: the
    inertial-range decay of a developed flow, damped towards the grid's
    cut-off as a sub-grid model damps it."""
    a = torch.fft.rfftn(torch.randn((nz, ny, nx), generator=g, device=DEV, dtype=torch.float32))
    k = lambda n, length: torch.fft.fftfreq(n, 1.0 / n, device=DEV).mul_(2 * math.pi / length).square_()
    k2 = k(nz, ZL)[:, None, None] + k(ny, YL)[None, :, None] + k(nx, XL)[None, None, : nx // 2 + 1]
    cut = math.pi / max(XL / nx, YL / ny, ZL / nz)
    a *= (1.0 + k2 / 9.0) ** (-11.0 / 12.0) * torch.exp(-4.0 * k2 / cut**2)
    a[0, 0, 0] = 0.0
    a = torch.fft.irfftn(a, s=(nz, ny, nx)).double()
    return a / a.std()


def initial(case, seed):
    """u, v, w, e on the GPU at the form's own real width: the benchmark
    channels' parabolic mean at the bulk velocity of Re_tau, solenoidal
    turbulence of a channel's intensity, and a sub-grid energy of a fraction
    of u_tau^2 or, late in a run, decayed to its floor over most of the
    domain."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    g = torch.Generator(device=DEV).manual_seed(seed)
    dz = ZL / nz
    eta = (torch.arange(nz, device=DEV, dtype=torch.float64) + 0.5) * dz - 1.0
    bulk = UTAU * ((math.log(case["re_tau"]) - 1.0) / 0.4 + 5.0)
    u, v, w = (UTAU * a * turbulence(nz, ny, nx, g) for a in (2.0, 1.0, 1.0))
    w[-1] = 0.0
    p = poisson(dx(u) + dy(v) + torch.diff(w, dim=0, prepend=torch.zeros_like(w[:1])) / dz, dz)
    u -= dx(p)
    v -= dy(p)
    w[:-1] -= (p[1:] - p[:-1]) / dz
    del p
    u += (1.5 * bulk * (1.0 - eta * eta))[:, None, None]
    t = turbulence(nz, ny, nx, g)
    e = EMIN * torch.exp(torch.clamp(2 * t - 1, min=0.0)) if case.get("tke_floor") else 0.3 * UTAU**2 * torch.exp(0.5 * t)
    real = torch.float64 if case.get("form", "fp64") == "fp64" else torch.float32
    return [a.to(real) for a in (u, v, w, e)]


def time_step(case, fields):
    """The advective CFL time step (0.5) of the initial field."""
    u, v, w = (float(a.abs().max()) for a in fields[:3])
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    return 0.5 / max(u * 1.5 * nx / XL, v * 1.5 * ny / YL, w * nz / ZL, 0.25 * nz)


def weights():
    z = np.load(os.path.join(ROOT, "paes-channelflow_b200", "weights", "sgs_c4.npz"))
    return z["params"], z["norm"]


def batches(case, seed):
    """Normalised features and targets as the training run makes them: unit
    gradient directions, capped wall distances, heavy-tailed stresses."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    n = case["batch"]
    made = []
    for _ in range(3):
        x = torch.zeros((n, 16), device=DEV)
        d = torch.randn((n, 9), generator=g, device=DEV)
        x[:, :9] = 3 * d / d.norm(dim=1, keepdim=True)
        x[:, 9:11] = 1.7 * (2 * torch.rand((n, 2), generator=g, device=DEV) - 1)
        t = torch.zeros((n, 8), device=DEV)
        t[:, :NOUT] = torch.randn((n, NOUT), generator=g, device=DEV) ** 3 / 4 + 0.3 * x[:, :NOUT] * x[:, 3:9]
        made.append((x.to(torch.bfloat16), t))
    p = []
    for rows, cols in ((HID, NIN), (HID, HID), (HID, HID), (NOUT, HID)):
        p += [torch.randn(rows * cols, generator=g, device=DEV) / math.sqrt(cols), torch.zeros(rows, device=DEV)]
    return made, torch.cat(p).cpu().numpy()


def prepare(case, seed):
    P = host()
    kind = case["kind"]
    if kind == "ops":
        g = torch.Generator(device=DEV).manual_seed(seed)
        real = torch.float64 if case["bits"] == 64 else torch.float32
        mk = lambda *s: torch.randn(s, generator=g, device=DEV, dtype=real)
        n, nx, ny = case["planes"], case["nx"], case["ny"]
        return {"case": case, "P": P, "small": mk(n, ny, nx), "large": mk(n, 3 * ny // 2, 3 * nx // 2)}
    if kind == "train":
        made, params = batches(case, seed)
        return {"case": case, "P": P, "data": made, "net": P.Mlp(params)}
    fields = initial(case, seed)
    form = case.get("form", "fp64")
    cfg = P.channel_config(case["nx"], case["ny"], case["nz"], dt=time_step(case, fields), re_tau=case["re_tau"],
                           imodel=case["imodel"] if kind == "split" else P.SGS_LEARNED if form == "learned"
                           else P.SGS_DEARDORFF,
                           tke_production=int(case.get("production", False)),
                           precision=P.PREC_FP64 if form == "fp64" else P.PREC_MIXED)
    h = P.LesGpu(cfg)
    state = {"case": case, "P": P, "h": h}
    if form == "learned":
        state["net"] = P.Mlp(*weights())
        h.set_mlp(state["net"], case["re_tau"])
    state["out"] = [torch.empty(a.shape, dtype=a.dtype, pin_memory=True) for a in fields]
    for a, b in zip(state["out"], fields):
        a.copy_(b)
    h.upload(*state["out"])
    return state


# ------------------------------------------------------------------- a pass
def run(state):
    case, P = state["case"], state["P"]
    if case["kind"] == "ops":
        s, l = state["small"], state["large"]
        return {"expand": P.expand(s), "compress": P.compress(l), "deal": P.deal(s), "xderiv": P.xderiv(l, XL),
                "yderiv": P.yderiv(l, YL)}
    if case["kind"] == "train":
        net, data = state["net"], state["data"]
        for i in range(case["steps"]):
            net.adam_step(*data[i % 2], lr=1e-3)
        loss, grad = net.loss_grad(*data[2])
        return {"loss": loss, "grad": grad, "out": net.forward(data[2][0]), "params": net.get_params()[0]}
    h, n = state["h"], case["steps"]
    for i in range(n):
        last = i == n - 1
        if case["kind"] == "split":
            for stage in (1, 2, 3):
                h.stage_split(i + 1, last, stage)
        else:
            h.step(it=i + 1, mnout=last)
    profiles, scalars = h.stats()
    h.download_into(*state["out"])
    real = np.float64 if state["out"][0].dtype == torch.float64 else np.float32
    out = dict(zip("uvwe", state["out"]), profiles=profiles.astype(real))
    if real is np.float64:  # in 32 bits the mean tendencies are the rounding left of cancelling fluxes
        out["scalars"] = scalars
    return out


# ------------------------------------------------- the same in 64 bits, torch
def wave(n, length):
    k = torch.fft.fftfreq(n, 1.0 / n, device=DEV, dtype=torch.float64) * (2 * math.pi / length)
    k[n // 2] = 0.0
    return k


def dx(a, length=XL):
    n = a.shape[-1]
    return torch.fft.irfft(torch.fft.rfft(a) * (1j * wave(n, length)[: n // 2 + 1]), n=n)


def dy(a, length=YL):
    n = a.shape[-2]
    return torch.fft.ifft(torch.fft.fft(a, dim=-2) * (1j * wave(n, length))[:, None], dim=-2).real


def resize(a, ny, nx):
    """Planes on another grid with the modes both grids have, Nyquist removed."""
    my, mx = a.shape[-2:]
    z = torch.fft.rfft2(a, norm="forward")
    o = torch.zeros(a.shape[:-2] + (ny, nx // 2 + 1), dtype=z.dtype, device=DEV)
    hy, hx = min(ny, my) // 2, min(nx, mx) // 2
    o[..., :hy, :hx] = z[..., :hy, :hx]
    o[..., ny - hy + 1:, :hx] = z[..., my - hy + 1:, :hx]
    return torch.fft.irfft2(o, s=(ny, nx), norm="forward")


def poisson(rhs, dz):
    """Solution p of the staggered pressure equation for each mode (unit
    off-diagonals, Neumann ends), its mean and Nyquist modes zero."""
    nz, ny, nx = rhs.shape
    r = torch.fft.rfft2(rhs) * (dz * dz)
    k2 = wave(ny, YL)[:, None] ** 2 + wave(nx, XL)[None, : nx // 2 + 1] ** 2
    k2[0, 0] = 1.0
    d = [1.0 / (-dz * dz * k2 - 1.0)]
    for z in range(1, nz):
        d.append(1.0 / (-dz * dz * k2 - (1.0 if z == nz - 1 else 2.0) - d[-1]))
        r[z] -= d[z - 1] * r[z - 1]
    r[nz - 1] *= d[nz - 1]
    for z in range(nz - 2, -1, -1):
        r[z] = d[z] * (r[z] - r[z + 1])
    r[:, 0, 0] = 0.0
    r[:, ny // 2] = 0.0
    r[:, :, nx // 2] = 0.0
    return torch.fft.irfft2(r, s=(ny, nx))


class Channel:
    """The RK3 channel, every level at once.  Padded fields are stored with
    their ghost levels: row L + 1 holds level L of u, v, w, e, L = -1..nz+1."""

    def __init__(self, case, fields, dt):
        self.nx, self.ny, self.nz, self.dt = case["nx"], case["ny"], case["nz"], dt
        self.smag, self.production = case.get("imodel") == 4, case.get("production", False)
        self.u, self.v, self.w, self.e = (resize(a.double(), self.ny, self.nx) for a in fields)
        self.w[-1] = 0.0
        self.ru, self.rv, self.rw, self.re = (torch.zeros_like(self.u) for _ in range(4))
        self.dz = ZL / self.nz
        self.dsl = (XL / self.nx * YL / self.ny * self.dz) ** (1.0 / 3.0)
        self.zody = math.log(self.dz / 2.0 / z0_of(case))
        self.prof = torch.zeros((19, self.nz), device=DEV, dtype=torch.float64)

    def wall(self, U, V, sg):
        u1, v1 = float(U.mean()), float(V.mean())
        vsfc = max(math.hypot(u1, v1), 0.01)
        ut = vsfc * 0.4 / self.zody
        a, b = -ZL / 2 * (FORCING - self.dudt), ZL / 2 * self.dvdt
        c = ut * self.utau_s / vsfc
        return sg * (c * (U - u1) - a), sg * (c * (V - v1) - b), ut

    def stage(self, s, mnout):
        nz, dz, n = self.nz, self.dz, self.nz
        gama, zeta = (8 / 15, 5 / 12, 3 / 4)[s], (0.0, 17 / 60, 5 / 12)[s]
        d1, d2, xkmax = self.dt * gama, self.dt * zeta, dz * dz / self.dt / 5.0
        pad = lambda a, lo, hi: torch.nn.functional.pad(a, (0, 0, 0, 0, lo, hi))
        big = lambda a: resize(a, 3 * self.ny // 2, 3 * self.nx // 2)
        self.e[nz - 1] = self.e[nz - 2]
        u, v, w = big(self.u), big(self.v), big(self.w[: nz - 1])
        e = torch.clamp(big(self.e[: nz - 1]), min=EMIN)
        U, V, W = pad(u, 2, 2), pad(v, 2, 2), pad(w, 2, 3)
        E = torch.cat([e[:1], e[:1], e, e[-1:], e[-1:], e[-1:]])
        lev = lambda A, a, b: A[a + 1: b + 2]  # levels a..b
        ux, vx, uy, vy = (pad(q, 1, 1) for q in (dx(u), dx(v), dy(u), dy(v)))  # levels 0..nz+1
        wx, wy = pad(dx(w), 1, 1), pad(dy(w), 1, 1)                           # levels 0..nz
        wz = (lev(W, 0, n + 1) - lev(W, -1, n)) / dz                          # levels 0..nz+1
        wz[0], wz[n + 1] = 0.0, 0.0
        ends = lambda q: torch.cat([q[:1], q, q[-1:]])
        uz, vz = ends((u[1:] - u[:-1]) / dz), ends((v[1:] - v[:-1]) / dz)      # levels 0..nz
        if self.smag or self.production:
            sh = (ux[:-1] ** 2 + ux[1:] ** 2 + vy[:-1] ** 2 + vy[1:] ** 2 + wz[:-1] ** 2 + wz[1:] ** 2
                  + 0.5 * (uy + vx)[:-1] ** 2 + 0.5 * (uy + vx)[1:] ** 2 + (uz + wx) ** 2 + (vz + wy) ** 2)
        if self.smag:
            xk = torch.clamp((0.1 * self.dsl) ** 2 * torch.sqrt(sh), max=xkmax)
        else:
            xk = torch.clamp(0.1 * self.dsl * torch.sqrt(lev(E, 0, n)), max=xkmax)  # levels 0..nz
        self.dudt, self.dvdt = float(self.ru.mean()), float(self.rv.mean())
        self.utau_s = math.sqrt(ZL / 2 * math.hypot(self.dvdt, FORCING - self.dudt))
        tuw, tvw = -xk * (uz + wx), -xk * (vz + wy)
        tuw[0], tvw[0], low = self.wall(u[0], v[0], -1.0)
        tuw[n], tvw[n], top = self.wall(u[-1], v[-1], 1.0)
        self.scalars = (top, self.utau_s, self.dudt, self.dvdt, low)
        xs = xk[:-1] + xk[1:]                                                 # levels 1..nz
        tuu, tvv, tuv = -xs * ux[1:-1], -xs * vy[1:-1], -0.5 * xs * (uy + vx)[1:-1]
        tww = torch.cat([-xs * wz[1:-1], torch.zeros_like(wz[:1])])           # levels 1..nz+1
        div = (ux + vy + wz)[1:-1].square_().mean(dim=(1, 2))
        if mnout and s == 0:
            for row, q in zip(range(13, 19), (tuu, tvv, tuv, tww[:-1], tuw[1:], tvw[1:])):
                self.prof[row] = q.mean(dim=(1, 2))
        self.prof[2] = div
        del uy, vx, vy, wx, wy, uz, vz
        Um, U0, U1, Vm, V0, V1 = (lev(A, 1 + o, n + o) for A in (U, V) for o in (-1, 0, 1))
        Wm, W0, W1 = (lev(W, 1 + o, n + o) for o in (-1, 0, 1))
        small = lambda a: resize(a, self.ny, self.nx)
        ru = small(FORCING - dx(U0 * U0 + tuu) - dy(U0 * V0 + tuv) - ((U1 + U0) * W0 - (Um + U0) * Wm) / (2 * dz)
                   - (tuw[1:] - tuw[:-1]) / dz)
        rv = small(-dx(U0 * V0 + tuv) - dy(V0 * V0 + tvv) - ((V1 + V0) * W0 - (Vm + V0) * Wm) / (2 * dz)
                   - (tvw[1:] - tvw[:-1]) / dz)
        del tuu, tvv, tuv
        rw = small(-dx(0.5 * (U0 + U1) * W0 + tuw[1:]) - dy(0.5 * (V0 + V1) * W0 + tvw[1:])
                   - ((0.5 * (W1 + W0)) ** 2 - (0.5 * (W0 + Wm)) ** 2) / dz - (tww[1:] - tww[:-1]) / dz)
        rw -= rw.mean(dim=(1, 2), keepdim=True)
        rw[-1] = 0.0
        del tuw, tvw, tww
        m = n - 1
        at = torch.tensor([min(i, n - 3) for i in range(m)], device=DEV)  # level min(iz, nz-2)
        E0, E1, Em, x0 = e, lev(E, 2, n), lev(E, 0, n - 2), xk[1:n]
        us, vs = 0.5 * (U0 + U1)[:m], 0.5 * (V0 + V1)[:m]
        re = (-dx(us * E0 - 2 * x0 * dx(e)[at]) - dy(vs * E0 - 2 * x0 * dy(e)[at])
              - (W1[:m] * E1 - Wm[:m] * Em) / (2 * dz)
              + ((xk[2: n + 1] + x0) * (E1 - E0) - (x0 + xk[: n - 1]) * (E0 - Em)) / dz ** 2
              - 0.93 / self.dsl * E0 * torch.sqrt(E0))
        if self.production:
            re += x0 * sh[1:n]
        re = small(re)
        if s:
            self.u -= d2 * self.ru
            self.v -= d2 * self.rv
            self.w -= d2 * self.rw
            self.e[:m] -= d2 * self.re[:m]
        q = self.w / d1 + rw
        q[-1] = 0.0
        p = poisson(dx(ru + self.u / d1) + dy(rv + self.v / d1) + (q - pad(q, 1, 0)[:-1]) / dz, dz)
        self.ru, self.rv = ru - dx(p), rv - dy(p)
        self.rw = rw
        self.rw[:m] -= (p[1:] - p[:-1]) / dz
        self.re[:m] = re
        self.u += d1 * self.ru
        self.v += d1 * self.rv
        self.w[:m] += d1 * self.rw[:m]
        self.w[:m] -= self.w[:m].mean(dim=(1, 2), keepdim=True)
        self.e[:m] = torch.clamp(self.e[:m] + d1 * re, min=EMIN)

    def profiles(self):
        mean = lambda a: a.mean(dim=(1, 2))
        um, vm = mean(self.u), mean(self.v)
        fu, fv = (torch.nn.functional.pad(a - b[:, None, None], (0, 0, 0, 0, 0, 1)) for a, b in
                  ((self.u, um), (self.v, vm)))
        ul, vl = 0.5 * (fu[:-1] + fu[1:]), 0.5 * (fv[:-1] + fv[1:])
        q = [mean(a * b) for a, b in ((ul, ul), (vl, vl), (self.w, self.w), (ul, self.w), (vl, self.w), (ul, vl))]
        p = self.prof
        p[0], p[1], p[3], p[4], p[5] = 0.5 * (q[0] + q[1] + q[2]), mean(self.e), um, vm, mean(self.w)
        for i in range(6):
            p[6 + i] = q[i]
        return p


def exact_train(case, seed):
    data, params = batches(case, seed)
    p = torch.tensor(params, device=DEV, dtype=torch.float64)
    m, v = torch.zeros_like(p), torch.zeros_like(p)

    def forward(q, x):
        x, o = x[:, :NIN].double(), 0
        for i, (rows, cols) in enumerate(((HID, NIN), (HID, HID), (HID, HID), (NOUT, HID))):
            x = x @ q[o: o + rows * cols].view(rows, cols).T + q[o + rows * cols: o + rows * cols + rows]
            o += rows * cols + rows
            x = torch.nn.functional.gelu(x, approximate="tanh") if i < 3 else x
        return x

    def grad_of(x, t):
        q = p.clone().requires_grad_(True)
        loss = (forward(q, x) - t[:, :NOUT].double()).square().mean()
        loss.backward()
        return float(loss.detach()), q.grad

    for i in range(case["steps"]):
        g = grad_of(*data[i % 2])[1]
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        p = p - 1e-3 * (m / (1 - 0.9 ** (i + 1))) / (torch.sqrt(v / (1 - 0.999 ** (i + 1))) + 1e-8)
    loss, g = grad_of(*data[2])
    y = torch.zeros((case["batch"], 8), device=DEV, dtype=torch.float64)
    y[:, :NOUT] = forward(p, data[2][0])
    return {"loss": loss, "grad": g, "out": y, "params": p.cpu().numpy()}


def exact(case, seed):
    if case["kind"] == "train":
        return exact_train(case, seed)
    if case["kind"] == "ops":
        g = torch.Generator(device=DEV).manual_seed(seed)
        real = torch.float64 if case["bits"] == 64 else torch.float32
        n, nx, ny = case["planes"], case["nx"], case["ny"]
        s, l = (torch.randn(q, generator=g, device=DEV, dtype=real).double() for q in
                ((n, ny, nx), (n, 3 * ny // 2, 3 * nx // 2)))
        return {"expand": resize(s, 3 * ny // 2, 3 * nx // 2), "compress": resize(l, ny, nx), "deal": resize(s, ny, nx),
                "xderiv": dx(l), "yderiv": dy(l)}
    if case.get("form") == "learned":
        return None  # the stresses are a 16-bit network's: no 64-bit value stands for them
    fields = initial(case, seed)
    c = Channel(case, fields, time_step(case, fields))
    for i in range(case["steps"]):
        for s in range(3):
            c.stage(s, i == case["steps"] - 1)
    out = dict(zip("uvwe", (c.u, c.v, c.w, c.e)), profiles=c.profiles().cpu().numpy())
    if case.get("form", "fp64") == "fp64":
        out["scalars"] = np.array(c.scalars)
    return out
