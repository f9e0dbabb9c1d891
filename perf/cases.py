"""Performance cases: the work a program has this library do, through the Python mirror of the C ABI.

Each case is one call (or the short sequence of calls) that such a program makes over and over: a time step of a jet
whose state lies on the device, the full 3D transforms, a step with the turbulence statistics, a run on host buffers,
a block of steps of an ensemble, a handful of served requests.  Sizes and parameters are those of the project's own
workloads (64^3 to 512^3 temporal jets, ensembles of 64^3 to 192^3, mixed grids of the tests).

``exact`` restates the same work with torch.fft in 64 bits.
"""
from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = str(Path(__file__).resolve().parents[1] / "gnss-1_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import gnss_b200 as G  # noqa: E402

_JET = dict(precision="fp64", scalars=1, alpha=0.0, scheme="cnab2", re=1000.0, sc=0.7, sc_c=1.0, dt=1e-3,
            alias=2.0 / 3.0)


def _jet(name, kind, nx, ny=None, nz=None, **kw):
    c = dict(kind=kind, nx=nx, ny=ny or nx, nz=nz or nx, **_JET)
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest jet of the configurations: a step is a handful of short launches, latency counts
        _jet("step_64_fp64", "step", 64),
        # a mixed grid with radix-3 axes, two scalars and the colloid drift term
        _jet("step_48x96x64_fp64_drift", "step", 48, 96, 64, scalars=2, alpha=0.05),
        # the 256^3 run with two scalars in plain FP64
        _jet("step_256_fp64_2s", "step", 256, scalars=2, re=3000.0, dt=5e-4),
        # the 512^3 mixed-precision run
        _jet("step_512_fp32", "step", 512, precision="fp32", re=5000.0, dt=2.5e-4),
        # the 512^3 run with the reference's whole field set u v w s c in FP64: the largest step
        _jet("step_512_fp64_2s", "step", 512, scalars=2, re=5000.0, sc_c=0.7, dt=2.5e-4),
        # a flat mixed-precision box, every axis of another length, two scalars
        _jet("step_256x384x192_fp32_2s", "step", 256, 384, 192, precision="fp32", scalars=2, re=2000.0, dt=5e-4),
        # the integrating-factor RK3 scheme (three substeps a step) in mixed precision
        _jet("rk3if_192_fp32", "step", 192, precision="fp32", scheme="rk3if"),
        # spectral -> physical for output and physical -> spectral for input, one field each
        _jet("transforms_192x256x128_fp64", "transforms", 192, 256, 128),
        # a step with the statistics and mean profiles of the state it starts from
        _jet("step_turb_256_fp32", "turb", 256, precision="fp32", dt=5e-4),
        # a whole run on host buffers: state up, steps with per-step statistics, state down
        _jet("run_host_128_fp32_2s", "run_host", 128, precision="fp32", scalars=2, steps=20),
        # the ensemble of 32 uneven jets, a block of steps as one graph launch
        dict(name="ensemble_32_fp32", kind="ensemble", m64=16, m96=8, m128=6, m192=2, precision="fp32", scalars=1,
             steps=10, branches=8),
        # requests of several sizes submitted together to the server and fetched
        dict(name="served_6_fp32", kind="served", m64=3, m96=2, m128=1, m192=0, precision="fp32", scalars=1, steps=40),
    ]


_SIZES = (16, 24, 32, 48, 64, 96, 128, 192, 256, 384, 512)


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["transforms", "transforms", "turb", "run_host", "ensemble", "served"])
    precision = rng.choice(["fp64", "fp32"])
    scalars = rng.choice([1, 2])
    if kind in ("ensemble", "served"):
        c = dict(kind=kind, m64=rng.randint(1, 8), m96=rng.randint(0, 4), m128=rng.randint(0, 2), m192=rng.randint(0, 1),
                 precision=precision, scalars=scalars, steps=rng.randint(4, 8))
        if kind == "ensemble":
            c["branches"] = rng.choice([1, 4, 8])
        return c
    base = rng.randrange(len(_SIZES))
    top = 512 ** 3 if kind == "step" else 256 ** 3
    while True:
        # the axes of one box lie within a factor of about two of each other
        n = [_SIZES[min(max(base + rng.randint(-1, 1), 0), len(_SIZES) - 1)] for _ in range(3)]
        if n[0] * n[1] * n[2] <= top:
            break
        base -= 1
    c = _jet(None, kind, *n, precision=precision, scalars=scalars, re=round(rng.uniform(500.0, 5000.0), 1),
             sc=rng.choice([0.7, 1.0, 2.0]), dt=rng.choice([2.5e-4, 5e-4, 1e-3]))
    if kind == "step":
        c["scheme"] = rng.choice(["cnab2", "cnab2", "cnab2", "rk3if"])
        if scalars == 2 and c["scheme"] == "cnab2" and rng.random() < 0.3:
            c["alpha"] = 0.05
        if c["scheme"] == "rk3if" and n[0] * n[1] * n[2] > 256 ** 3:
            c["scheme"] = "cnab2"
    if kind == "run_host":
        c["steps"] = rng.randint(5, 20)
    return c


# ------------------------------------------------------------------ inputs
def _config(c):
    return dict(nx=c["nx"], ny=c["ny"], nz=c["nz"], re=c["re"], sc=c["sc"], sc_c=c["sc_c"], alpha=c["alpha"],
                dt=c["dt"], alias_filter=c["alias"], n_scalars=c["scalars"],
                scheme=G.GNSS_SCHEME_RK3IF if c["scheme"] == "rk3if" else G.GNSS_SCHEME_CNAB2,
                precision=G.GNSS_FP64 if c["precision"] == "fp64" else G.GNSS_FP32)


def _dtype(c):
    return torch.complex128 if c["precision"] == "fp64" else torch.complex64


def _waves(c, device="cuda"):
    def k(n):
        i = torch.arange(n, dtype=torch.float64, device=device)
        return torch.where(i < n // 2, i, i - n)
    kz = torch.arange(c["nz"] // 2 + 1, dtype=torch.float64, device=device)
    kz = torch.where(kz < c["nz"] // 2, kz, kz - c["nz"])
    return k(c["nx"])[None, :, None], k(c["ny"])[:, None, None], kz[None, None, :]


def _kept(c):
    kx, ky, kz = _waves(c)
    return (kx * kx + ky * ky + kz * kz) <= (c["alias"] * c["nx"] / 2) ** 2


def _to_spectral(p):
    """Real [nx, ny, nz] -> complex [ny, nx, nz2], unnormalised."""
    return torch.fft.rfftn(p).transpose(0, 1).contiguous()


def _to_physical(f, nz):
    """Complex [ny, nx, nz2] -> real [nx, ny, nz] with the 1/N factor (the imaginary parts of the kz = 0 and kz = nz/2
    entries are ignored after the x and y transforms)."""
    t = torch.fft.ifftn(f, dim=(0, 1))
    t[..., 0].imag.zero_()
    if nz % 2 == 0:
        t[..., nz // 2].imag.zero_()
    return torch.fft.irfft(t, n=nz, dim=2).transpose(0, 1)


def _initial(c, seed):
    """Truncated spectral state [u, v, w, s(, c)] in the case's precision: the tanh jet along y plus solenoidal noise
    of 5% that falls off towards the small scales, as in a jet under way."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    shape = (c["nx"], c["ny"], c["nz"])
    kx, ky, kz = _waves(c)
    k2 = kx * kx + ky * ky + kz * kz
    keep = (k2 <= (c["alias"] * c["nx"] / 2) ** 2) & (kx.abs() < c["nx"] / 2) & (ky.abs() < c["ny"] / 2) & \
        (kz.abs() < c["nz"] / 2)
    shape_k = torch.where(keep, (1.0 + k2 / 64.0) ** -1.4, torch.zeros((), dtype=torch.float64, device="cuda"))
    noise = [_to_spectral(torch.randn(shape, dtype=torch.float64, device="cuda", generator=g)).mul_(shape_k)
             for _ in range(3)]
    div = (noise[0] * kx + noise[1] * ky + noise[2] * kz) / k2.clamp(min=1.0)
    for f, k in zip(noise, (kx, ky, kz)):
        f.sub_(div * k)
    del div
    y = -math.pi + torch.arange(c["ny"], dtype=torch.float64) * (2 * math.pi / c["ny"])
    prof = torch.fft.fft(0.5 - 0.5 * torch.tanh(5.0 * (2.0 * y.abs() - 1.0))).cuda() * (c["nx"] * c["nz"])
    prof = torch.where(keep[:, 0, 0], prof, torch.zeros_like(prof))
    nn = float(c["nx"] * c["ny"] * c["nz"])
    scale = 0.05 * nn / math.sqrt(2.0 * sum(float(f.abs().square().sum()) for f in noise) / 3.0)
    out = []
    for q in range(3 + c["scalars"]):
        if q < 3:
            f = noise[q] * scale
        else:   # scalars: the jet profile and noise of their own
            f = noise[(q + 1) % 3] * (0.5 * scale)
        if q != 1 and q != 2:
            f[:, 0, 0] += prof
        out.append(f.to(_dtype(c)))
    return out


def _members(c):
    """Configurations of an ensemble's or a stream's jets: uneven sizes, Reynolds and Schmidt numbers."""
    out, i = [], 0
    for n in (64, 96, 128, 192):
        for _ in range(c["m%d" % n]):
            out.append(_jet(None, "step", n, precision=c["precision"], scalars=c["scalars"],
                            re=500.0 + (i * 977) % 3501, sc=(0.7, 1.0, 2.0)[i % 3]))
            i += 1
    return out


def _host_state(m, seed):
    t = torch.stack(_initial(m, seed))
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h


class _DeviceArray:
    """A library-owned device buffer as torch sees it; it keeps the buffer's owner alive."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=shape, typestr=typestr, data=(ptr, False), version=2)


def prepare(case, seed):
    c = case
    kind = c["kind"]
    if kind == "ensemble":
        ms = _members(c)
        ens = G.Ensemble([G.make_config(**_config(m)) for m in ms], n_branches=c["branches"])
        views = []
        for i, m in enumerate(ms):
            ens.upload(i, _host_state(m, seed * 100 + i))
            _, sf, _ = ens.member(i)
            t = torch.as_tensor(_DeviceArray(ens, sf.u, (3 + m["scalars"], m["ny"], m["nx"], m["nz"] // 2 + 1),
                                             "<c16" if m["precision"] == "fp64" else "<c8"), device="cuda")
            t.owner = ens   # the buffers live as long as the ensemble
            views.append(t)
        ens.step(1)
        return dict(kind=kind, ens=ens, views=views, steps=c["steps"])
    if kind == "served":
        ms = _members(c)
        srv = G.Server(150 << 30, max_active=16, steps_per_launch=20)
        reqs = [(G.make_config(**_config(m)), _host_state(m, seed * 100 + i).numpy()) for i, m in enumerate(ms)]
        return dict(kind=kind, srv=srv, reqs=reqs, steps=c["steps"])
    ctx = G.Context(**_config(c))
    if kind == "transforms":
        spec = _initial(c, seed)[0]
        phys = torch.zeros((c["nx"], c["ny"], 2 * (c["nz"] // 2 + 1)), device="cuda",
                           dtype=torch.float64 if c["precision"] == "fp64" else torch.float32)
        phys[..., :c["nz"]] = _to_physical(_initial(c, seed + 7)[1].to(torch.complex128), c["nz"])
        return dict(kind=kind, ctx=ctx, spec=spec, phys=phys, a=torch.empty_like(spec), b=torch.empty_like(phys))
    if kind == "run_host":
        h = _host_state(c, seed)
        return dict(kind=kind, ctx=ctx, host_in=h, host_out=torch.empty(h.shape, dtype=h.dtype, pin_memory=True),
                    stats=np.zeros((c["steps"], G.GNSS_NSTATS)), steps=c["steps"])
    state = _initial(c, seed)
    if c["scheme"] == "rk3if":
        return dict(kind=kind, ctx=ctx, state=state, hist=None)
    hist = [torch.zeros_like(f) for f in state]
    ctx.solver_ps(state, hist, True)   # a run under way: its first step has been made
    return dict(kind=kind, ctx=ctx, state=state, hist=hist)


def run(state):
    s = state
    kind = s["kind"]
    if kind == "step":
        s["ctx"].solver_ps(s["state"], s["hist"], False)
        return dict(state=s["state"], hist=s["hist"])
    if kind == "turb":
        stats, prof = s["ctx"].step_turb(s["state"], s["hist"], False)
        return dict(state=s["state"], hist=s["hist"], stats=stats, profiles=prof)
    if kind == "transforms":
        s["a"].copy_(s["spec"])
        s["ctx"].inverse_transform(s["a"])
        s["b"].copy_(s["phys"])
        s["ctx"].forward_transform(s["b"])
        return dict(physical=s["ctx"].physical_view(s["a"]), spectral=torch.view_as_complex(
            s["b"].view(-1, 2)).view(s["spec"].shape))
    if kind == "run_host":
        s["ctx"].run_host(s["host_in"], s["host_out"], s["steps"], True, s["stats"])
        return dict(state=s["host_out"], stats=s["stats"])
    if kind == "ensemble":
        s["ens"].step(s["steps"])
        return s["views"]
    ids = [s["srv"].submit(cfg, h, s["steps"]) for cfg, h in s["reqs"]]
    out = []
    for i in ids:
        s["srv"].wait(i)
        final, stats, _ = s["srv"].result(i)
        out.append(dict(state=final, stats=stats))
    return out


# ------------------------------------------------------------------ what a pass cannot do without
def _step_work(c):
    """A step reads the modes inside the dealiasing sphere of state and history once, writes them once, and takes the
    transforms of 9 (12, 14) fields to physical space and of 4 (5) products back."""
    two = c["scalars"] == 2
    elem = 16 if c["precision"] == "fp64" else 8
    points = c["nx"] * c["ny"] * c["nz"]
    r = c["alias"] * c["nx"] / 2
    modes = min(points / 2.0, 2.0 / 3.0 * math.pi * r ** 3)
    ffts = (14 if two and c["alpha"] else 12 if two else 9) + (5 if two else 4)
    subs = 3 if c["scheme"] == "rk3if" else 1
    rw = 2 if c["scheme"] == "rk3if" else 4
    return subs * (3 + c["scalars"]) * rw * modes * elem, subs * ffts * 2.5 * points * math.log2(points)


def work(case):
    c = case
    if c["kind"] in ("ensemble", "served"):
        b = f = 0.0
        for m in _members(c):
            wb, wf = _step_work(m)
            b, f = b + wb * c["steps"], f + wf * c["steps"]
        return dict(bytes=b, flops=f)
    if c["kind"] == "transforms":
        points = c["nx"] * c["ny"] * c["nz"]
        return dict(bytes=4.0 * points * (8 if c["precision"] == "fp64" else 4), flops=5.0 * points * math.log2(points))
    b, f = _step_work(c)
    n = c.get("steps", 1)
    return dict(bytes=b * n, flops=f * n)


# ------------------------------------------------------------------ the same in 64 bits
class _Exact:
    """The time step of the jet with torch.fft in 64 bits (rotational form, scalars in gradient form, projection,
    Crank-Nicolson with Euler / Adams-Bashforth, or the integrating-factor low-storage RK3)."""

    def __init__(self, c):
        self.c = c
        self.kx, self.ky, self.kz = _waves(c)
        self.k2 = self.kx * self.kx + self.ky * self.ky + self.kz * self.kz
        self.keep = _kept(c)
        self.num = [c["re"]] * 3 + [c["re"] * c["sc"], c["re"] * c["sc_c"]]

    def phys(self, f):
        return _to_physical(f, self.c["nz"])

    def rhs(self, st):
        c, kx, ky, kz = self.c, self.kx, self.ky, self.kz
        st = [torch.where(self.keep, f, torch.zeros_like(f)) for f in st]
        vel = [self.phys(f) for f in st[:3]]
        if c["scheme"] == "cnab2":   # the velocity makes a round trip through physical space
            st[:3] = [_to_spectral(p) for p in vel]
        u, v, w = st[:3]
        out = []
        o1, o2, o3 = (self.phys(1j * t) for t in (ky * w - kz * v, kz * u - kx * w, kx * v - ky * u))
        out.append(_to_spectral(o2 * vel[2] - o3 * vel[1]))
        out.append(_to_spectral(o3 * vel[0] - o1 * vel[2]))
        out.append(_to_spectral(o1 * vel[1] - o2 * vel[0]))
        del o1, o2, o3
        gs = [self.phys(1j * k * st[3]) for k in (kx, ky, kz)]
        out.append(_to_spectral(vel[0] * gs[0] + vel[1] * gs[1] + vel[2] * gs[2]))
        if c["scalars"] == 2:
            gc = [self.phys(1j * k * st[4]) for k in (kx, ky, kz)]
            n = vel[0] * gc[0] + vel[1] * gc[1] + vel[2] * gc[2]
            if c["alpha"]:
                n = n + c["alpha"] * (self.phys(-self.k2 * st[3]) * self.phys(st[4]) + gc[0] * gs[0] + gc[1] * gs[1] +
                                      gc[2] * gs[2])
            out.append(_to_spectral(n))
        k2 = self.k2.clone()
        k2[0, 0, 0] = 1.0
        pr = (kx * out[0] + ky * out[1] + kz * out[2]) / k2
        for q, k in enumerate((kx, ky, kz)):
            out[q] = k * pr - out[q]
        for q in range(3, len(out)):
            out[q] = -out[q]
        for q in range(len(out)):
            out[q][0, 0, 0] = 0
            out[q] = torch.where(self.keep, out[q], torch.zeros_like(out[q]))
        return out, st

    def step(self, st, hist, euler):
        c, dt = self.c, self.c["dt"]
        if c["scheme"] == "rk3if":
            gam, zet, q_ = (8 / 15, 5 / 12, 3 / 4), (0.0, -17 / 60, -5 / 12, 0.0), [0.0] * len(st)
            for s in range(3):
                n, _ = self.rhs(st)
                st = [torch.where(self.keep, f, torch.zeros_like(f)) for f in st]
                for q in range(len(st)):
                    e = torch.exp(-self.k2 * ((gam[s] + zet[s]) * dt / self.num[q]))
                    st[q] = e * (st[q] + gam[s] * dt * n[q] + q_[q])
                    q_[q] = zet[s + 1] * dt * e * n[q]
            return st, None
        n, st = self.rhs(st)
        new = []
        for q in range(len(st)):
            h = self.k2 * (dt / 2.0 / self.num[q])
            r = n[q] if euler else 1.5 * n[q] - 0.5 * hist[q]
            new.append(((1.0 - h) * st[q] + dt * r) / (1.0 + h))
        return new, n

    def _sum(self, f):
        w = torch.full((self.c["nz"] // 2 + 1,), 2.0, dtype=torch.float64, device="cuda")
        w[0] = w[-1] = 1.0
        return float((f * w).sum())

    def stats(self, st):
        c, nu = self.c, 1.0 / self.c["re"]
        nn2 = float(c["nx"] * c["ny"] * c["nz"]) ** 2
        e = sum(f.abs().square() for f in st[:3])
        su, se = self._sum(e) / nn2, self._sum(e * self.k2) / nn2
        sl = self._sum(torch.where(self.k2 > 0, e / (2 * self.k2.clamp(min=1e-30).sqrt()), torch.zeros_like(e))) / nn2
        chi, var = [0.0, 0.0], [0.0, 0.0]
        for q in range(3, len(st)):
            m = st[q].abs().square()
            chi[q - 3] = 2.0 * nu / (c["sc"], c["sc_c"])[q - 3] * self._sum(m * self.k2) / nn2
            m[0, 0, 0] = 0
            var[q - 3] = self._sum(m) / nn2
        return dict(ke=su / 2, vrms2=su / 3, eps=nu * se, sl=sl, chi=chi, var=var)

    def turb(self, st):
        c, nu, t = self.c, 1.0 / self.c["re"], self.stats(st)
        u, v, w = st[:3]
        om = [self.phys(1j * f) for f in (self.ky * w - self.kz * v, self.kz * u - self.kx * w,
                                          self.kx * v - self.ky * u)]
        d = dict(vrms=math.sqrt(t["vrms2"]), ke=t["ke"], epsilon=t["eps"], eta=(nu ** 3 / t["eps"]) ** 0.25,
                 l=3 * math.pi / 4 * t["sl"] / t["ke"], chi=t["chi"][0],
                 omega=float(sum(o.square() for o in om).sqrt().mean()))
        d["lambda"] = math.sqrt(15.0 * nu * t["vrms2"] / t["eps"])
        for k, o in zip("xyz", om):
            d["omega_" + k] = float(o.square().mean().sqrt())
        prof = torch.zeros((5, c["ny"]), dtype=torch.float64)
        for q, f in enumerate(st):
            prof[q] = self.phys(f).mean(dim=(0, 2)).cpu()
        return d, prof


def _run_exact(c, first, steps):
    x = _Exact(c)
    st, hist = [f.to(torch.complex128) for f in first], None
    for i in range(steps):
        st, hist = x.step(st, hist, i == 0)
    return x, st, hist


def exact(case, seed):
    c = case
    kind = c["kind"]
    if kind == "transforms":
        spec = _initial(c, seed)[0].to(torch.complex128)
        p = torch.zeros((c["nx"], c["ny"], 2 * (c["nz"] // 2 + 1)), dtype=torch.float64, device="cuda")
        p[..., :c["nz"]] = _to_physical(spec, c["nz"])
        f = _to_physical(_initial(c, seed + 7)[1].to(torch.complex128), c["nz"])
        f = f.to(torch.float64 if c["precision"] == "fp64" else torch.float32).to(torch.float64)
        return dict(physical=p, spectral=_to_spectral(f))
    if kind in ("ensemble", "served"):
        out = []
        for i, m in enumerate(_members(c)):
            n = c["steps"] + (1 if kind == "ensemble" else 0)
            x, st, _ = _run_exact(m, _initial(m, seed * 100 + i), n)
            st = torch.stack(st).cpu()
            if kind == "served":
                t = x.stats([f.cuda() for f in st])
                st = dict(state=st, stats=dict(ke=t["ke"], vrms2=t["vrms2"], eps=t["eps"], chi_s=t["chi"][0],
                                               chi_c=t["chi"][1], var_s=t["var"][0], var_c=t["var"][1]))
            out.append(st)
        return out
    first = _initial(c, seed)
    if kind == "run_host":
        x = _Exact(c)
        st, hist, rows = [f.to(torch.complex128) for f in first], None, []
        for i in range(c["steps"]):
            st, hist = x.step(st, hist, i == 0)
            t = x.stats(st)
            rows.append([t["ke"], t["vrms2"], t["eps"], *t["chi"], *t["var"]])
        return dict(state=torch.stack(st).cpu(), stats=np.array(rows))
    if c["scheme"] == "rk3if":
        _, st, _ = _run_exact(c, first, 1)
        return dict(state=st, hist=None)
    x, st, hist = _run_exact(c, first, 1)
    stats = x.turb(st) if kind == "turb" else None
    st, hist = x.step(st, hist, False)
    if kind == "turb":
        return dict(state=st, hist=hist, stats=stats[0], profiles=stats[1].numpy())
    return dict(state=st, hist=hist)
