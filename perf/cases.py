"""The work that users of this framework have it do, as cases to measure.

Every case goes through the public entry points (instaheat_gb300.gpu and the
C ABI under it): single right-hand sides on host and on device arrays, RK4 and
DOPRI853 steps with the state read back, saved slices, the start of a run and
ensembles, in the plain FP64 form and the mixed FP32/FP64 form, from 32^3 to
256^3 with non-cubic and radix-3 grids among them.

The physics of every case is the same: a homogeneous inflaton with seeded
vacuum-like fluctuations in a periodic box, psi from the constraints, small
tensor modes, GW sources and filter on.  Step sizes are given and small enough
that every DOPRI853 try is accepted, except in the ensemble, which runs on its
own controller.
"""
from __future__ import annotations

import json
import math
from pathlib import Path

import numpy as np
import torch

from instaheat_gb300 import gpu

DEV = "cuda"
F64 = torch.float64


def _case(name, kind, n, prec="f64", steps=1, output=False, tuned=False, proposer=False,
          box=20.0, phi0=1.0):
    return {"name": name, "kind": kind, "nx": n[0], "ny": n[1], "nz": n[2], "prec": prec,
            "steps": steps, "output": output, "tuned": tuned, "proposer": proposer,
            "box": box, "phi0": phi0}


def listed():
    return [
        # mk_rhs as a C host program calls it through the drop-in layer: host
        # arrays in and out, the smallest production grid (latency, launches)
        _case("rhs_host_32_f64", "rhs_host", (32, 32, 32)),
        # fixed-step RK4 at 32^3, the reference's plain configuration: ten
        # steps between two reads of the state
        _case("rk4_32_f64", "rk4", (32, 32, 32), steps=10),
        # DOPRI853 at 64^3 with a saved slice (spectra, constraints, summaries)
        # after three steps: the drop-in's run loop
        _case("dopri_64_f64", "dopri", (64, 64, 64), steps=3, output=True),
        # a filtered output RHS on device arrays on a non-cubic radix-3 grid
        _case("rhs_dev_96x64x48_f64", "rhs_dev", (96, 64, 48), output=True),
        # the diagnostics of a saved slice and the state, as run loops save them
        _case("slice_128_f64", "slice", (128, 128, 128)),
        # DOPRI853 step and state at 128^3, plain FP64
        _case("dopri_128_f64", "dopri", (128, 128, 128)),
        # one plain RHS on device arrays at 256^3: a host program's own stepper
        _case("rhs_dev_256_f64", "rhs_dev", (256, 256, 256)),
        # the largest plain FP64 work: one DOPRI853 step at 256^3
        _case("dopri_256_f64", "dopri", (256, 256, 256)),
        # realisations of mixed grid sizes stepped together, the ensemble
        # configuration's sizes and proportions at a quarter of its members
        _case("ensemble_32_64_96_mixed", "ensemble", (96, 96, 96), prec="mixed", tuned=True),
        # mixed form at 128^3, untuned as a plain Context is
        _case("dopri_128_mixed", "dopri", (128, 128, 128), prec="mixed", steps=4),
        # mixed form at 256^3 with tuned engines and the learned proposer: four
        # steps and a saved slice
        _case("dopri_256_mixed", "dopri", (256, 256, 256), prec="mixed", steps=4, output=True,
              tuned=True, proposer=True),
        # the start of a run: state from the host, psi solve, the opening RHS
        _case("start_128_mixed", "start", (128, 128, 128), prec="mixed"),
    ]


def _smooth(n):
    for p in (2, 3):
        while n % p == 0:
            n //= p
    return n == 1


_AXES = [n for n in range(16, 513, 2) if _smooth(n)]
_POW2 = [32, 64, 128, 256, 512]


def draw(rng):
    kind = rng.choice(["rhs_host", "rhs_dev", "rk4", "dopri", "dopri", "slice", "start"])
    prec = "f64" if kind == "rhs_dev" else rng.choice(["f64", "mixed"])
    radix3 = rng.random() < 0.4
    # odd sizes up to 128^3 points, powers of two up to 256^3 (every other
    # kind but a DOPRI853 step also there)
    top = 128 ** 3 if radix3 else 256 ** 3
    target = math.exp(rng.uniform(math.log(16 ** 3), math.log(top)))
    axes = _AXES if radix3 else _POW2
    best = None
    for _ in range(200):
        n = sorted((rng.choice(axes) for _ in range(3)), reverse=True)
        if n[0] > 8 * n[2] or n[0] * n[1] * n[2] > top:
            continue
        d = abs(math.log(n[0] * n[1] * n[2] / target))
        if best is None or d < best[0]:
            best = (d, n)
    c = _case("", kind, tuple(best[1]), prec=prec,
              steps=rng.choice([1, 2, 3]) if kind == "rk4" else 1,
              output=rng.random() < 0.5, tuned=False,
              box=round(rng.uniform(10.0, 40.0), 3), phi0=round(rng.uniform(0.8, 1.2), 4))
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# inputs


def _members(case):
    """(n, box, phi0) of every ensemble member: sizes 32, 64, 96 at 6:6:4, box
    and phi0 over the ensemble configuration's ranges."""
    out = []
    for n, count in ((32, 6), (64, 6), (96, 4)):
        for i in range(count):
            out.append(((n, n, n), 10.0 + 30.0 * (i + 0.5) / count, 0.8 + 0.4 * (i + 0.5) / count))
    return out


class _Grid:
    """k vectors and spectral operations of one grid in FP64 (torch)."""

    def __init__(self, n, box):
        self.n, self.box = n, box
        self.N = n[0] * n[1] * n[2]
        self.mz = n[2] // 2 + 1
        self.M = n[0] * n[1] * self.mz
        u = 2.0 * math.pi / box
        full, deriv = [], []
        for axis, N in enumerate(n):
            i = torch.arange(self.mz if axis == 2 else N, dtype=F64, device=DEV)
            f = torch.where(i > N // 2, i - N, i) * u
            shape = [1, 1, 1]
            shape[axis] = -1
            full.append(f.reshape(shape))
            deriv.append(torch.where(2 * i == N, torch.zeros_like(f), f).reshape(shape))
        self.k, self.kd = full, deriv
        self.k2 = full[0] ** 2 + full[1] ** 2 + full[2] ** 2
        # |k|^2 for the shells of the spectra, summed as the reference's C code
        # does (z, x, y), so that modes on a shell's edge fall to the same side
        u2 = (2.0 * math.pi) * (2.0 * math.pi) / (box * box)
        i = [torch.arange(self.mz if a == 2 else N, dtype=F64, device=DEV) for a, N in enumerate(n)]
        sq = [(u2 * j) * j for j in (torch.where(j > N // 2, N - j, j) for j, N in zip(i, n))]
        self.shell2 = (sq[2].reshape(1, 1, -1) + sq[0].reshape(-1, 1, 1)) + sq[1].reshape(1, -1, 1)
        self.shell_max = math.sqrt(u2 * (n[0] // 2) * (n[0] // 2) + u2 * (n[1] // 2) * (n[1] // 2) +
                                   u2 * (n[2] // 2) * (n[2] // 2))

    def fft(self, x):
        return torch.fft.rfftn(x.reshape(self.n))

    def ifft(self, c):
        """Inverse transform divided by N."""
        return torch.fft.irfftn(c, s=self.n)

    def mask(self):
        frac = torch.zeros((1, 1, 1), dtype=F64, device=DEV)
        for k, N in zip(self.k, self.n):
            frac = torch.maximum(frac, k.abs() / ((N // 2) * 2.0 * math.pi / self.box))
        return torch.exp(-36.0 * frac ** 36)

    def split(self, f):
        """Views of a state: phi, dphi, psi, dpsi, h1, h2, dh1, dh2, a."""
        real = [f[i * self.N:(i + 1) * self.N].reshape(self.n) for i in range(4)]
        spec = []
        for i in range(4):
            s = f[4 * self.N + 2 * self.M * i:4 * self.N + 2 * self.M * (i + 1)]
            spec.append(torch.view_as_complex(s.reshape(self.n[0], self.n[1], self.mz, 2)))
        return real, spec, f[-1]


MASS = 1.0
AMP = 1.0e-3


def _potential(phi):
    return 0.5 * MASS * MASS * phi * phi


def _input_state(n, box, phi0, seed, psi=True):
    """A seeded state: phi0 and its slow-roll velocity plus fluctuations with
    variance AMP^2 / (2 omega box^3) per mode, psi and dpsi from the
    constraints, tensor modes of relative size 1e-5, a = 1."""
    g = _Grid(n, box)
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed) * 7919 + 17)
    omega = torch.sqrt(g.k2 + MASS * MASS)
    scale = AMP * math.sqrt(g.N) / torch.sqrt(2.0 * omega * box ** 3)
    f = torch.zeros(4 * g.N + 8 * g.M + 1, dtype=F64, device=DEV)
    (phi, dphi, ps, dps), spec, _ = g.split(f)

    def noise(weight):
        c = g.fft(torch.randn(n, dtype=F64, device=DEV, generator=gen)) * weight
        c[0, 0, 0] = 0.0
        return c

    dphi0 = -MASS * MASS * phi0 / (3.0 * math.sqrt(_potential(phi0) / 3.0))
    phi.copy_(phi0 + g.ifft(noise(scale)))
    dphi.copy_(dphi0 + g.ifft(noise(scale * omega)))
    for i, s in enumerate(spec):
        s.copy_(noise(1e-5 * AMP * (omega if i >= 2 else torch.ones_like(omega)) /
                      torch.sqrt(omega)))
    f[-1] = 1.0
    if psi:
        r, aux = _rhs(g, f)
        H, dm = aux["H"], dphi.mean()
        ddm = r[g.N:2 * g.N].mean()
        cphi, cdphi = g.fft(phi - phi.mean()), g.fft(dphi - dm)
        c = (-dm * cdphi + ddm * cphi) / (-dm * dm + 2.0 * g.k2)
        c[0, 0, 0] = 0.0
        ps.copy_(g.ifft(c))
        dps.copy_(0.5 * dm * (phi - phi.mean()) - H * ps)
    return f


class _State:
    pass


def _context(case):
    return gpu.Context(n=(case["nx"], case["ny"], case["nz"]), L=(case["box"],) * 3, mass=MASS,
                       precision=gpu.PREC_MIXED if case["prec"] == "mixed" else gpu.PREC_F64)


def _dt(case):
    return min(0.01, 0.1 * case["box"] / case["nx"])


def _proposer():
    rec = json.loads((Path(gpu.__file__).parent / "data" / "dt_mlp.json").read_text())
    m = gpu.MLP()
    m.params = np.array(rec["params"], dtype=np.float32)
    m.set_norm(rec["in_mean"], rec["in_std"], rec["out_mean"], rec["out_std"])
    return m


def prepare(case, seed):
    s = _State()
    s.case = case
    s.host32 = {}
    s.dt = _dt(case)
    kind = case["kind"]
    n = (case["nx"], case["ny"], case["nz"])
    if kind == "ensemble":
        members = _members(case)
        s.ens = gpu.Ensemble([dict(n=m, L=(box,) * 3, precision=gpu.PREC_MIXED)
                              for m, box, _ in members])
        if case["tuned"]:
            s.ens.autotune()
        s.buf = []
        for i, (ctx, (m, box, phi0)) in enumerate(zip(s.ens.members, members)):
            f = _input_state(m, box, phi0, 100 * int(seed) + i)
            buf = torch.empty(f.numel(), dtype=F64, pin_memory=True)
            buf.copy_(f)
            ctx.set_state(buf.numpy())
            s.buf.append(buf)
        s.ens.dopri_init(gpu.dopri_cfg(1e-8, 1e-8), 0.0, 1e-3)
        s.t = 0.0
        return s
    f = _input_state(n, case["box"], case["phi0"], seed, psi=kind != "start")
    s.ctx = _context(case)
    if case["tuned"]:
        s.ctx.autotune()
    if kind == "rhs_dev":
        s.f, s.out = f, torch.zeros_like(f)
        return s
    s.buf = torch.empty(f.numel(), dtype=F64, pin_memory=True)
    s.buf.copy_(f)
    if kind == "rhs_host":
        s.f = s.buf.numpy()
        return s
    if kind == "start":
        s.f = s.buf.numpy()
        s.buf = torch.empty(f.numel(), dtype=F64, pin_memory=True)
        s.dbuf = torch.empty(f.numel(), dtype=F64, pin_memory=True)
        return s
    s.ctx.set_state(s.buf.numpy())
    if kind == "dopri":
        s.ctx.dopri_init(gpu.dopri_cfg(1e-8, 1e-8), 0.0, s.dt)
        if case["proposer"]:
            s.ctx.set_proposer(_proposer())
    return s


# ---------------------------------------------------------------------------
# one pass


def _typed(s, i, host):
    """Host array i of a pass in the type that the form computes in: FP64, or
    FP32 in a buffer that the program keeps."""
    if s.case["prec"] != "mixed":
        return host
    if i not in s.host32:
        s.host32[i] = torch.empty(host.numel(), dtype=torch.float32)
    return s.host32[i].copy_(host)


def _diagnostics(out):
    return {k: out[k] for k in ("phi_ps", "psi_ps", "rho_ps", "gw", "cstr", "smry")}


def run(s):
    case, kind = s.case, s.case["kind"]
    if kind == "ensemble":
        s.t += 0.05
        s.ens.run(s.t)
        for ctx, buf in zip(s.ens.members, s.buf):
            ctx.get_state_into(buf.numpy())
        return [_typed(s, i, buf) for i, buf in enumerate(s.buf)]
    ctx = s.ctx
    if kind == "rhs_host":
        res, f = ctx.mk_rhs(s.f, filter=int(case["output"]), output=int(case["output"]))
        r = {"result": _typed(s, 0, torch.from_numpy(res)),
             "field": _typed(s, 1, torch.from_numpy(f))}
        if case["output"]:
            r["diag"] = _diagnostics(ctx.output())
            if case["prec"] == "mixed":
                r["diag"] = {k: v.astype(np.float32) for k, v in r["diag"].items()}
        return r
    if kind == "rhs_dev":
        flag = int(case["output"])
        # f is filtered in place with the filter flag, as the reference does
        ctx._ck(ctx.L_.ih_mk_rhs_dev(ctx.h, 0.0, s.f.data_ptr(), s.out.data_ptr(), flag, flag),
                "ih_mk_rhs_dev")
        r = {"result": s.out, "field": s.f}
        if flag:
            r["diag"] = _diagnostics(ctx.output())
        return r
    if kind == "start":
        ctx.set_state(s.f)
        ctx.initial_psi()
        ctx.dopri_init(gpu.dopri_cfg(1e-8, 1e-8), 0.0, s.dt)
        ctx.get_state_into(s.buf.numpy())
        ctx.get_dstate(s.dbuf.numpy())
        return {"state": _typed(s, 0, s.buf), "dstate": _typed(s, 1, s.dbuf)}
    r = {}
    if kind == "rk4":
        for i in range(case["steps"]):
            ctx.rk4_step(s.dt)
    elif kind == "dopri":
        for i in range(case["steps"]):
            ctx.dopri_step(s.dt, output=case["output"] and i == case["steps"] - 1)
        if case["output"]:
            r["diag"] = _diagnostics(ctx.output())
    else:
        r["diag"] = _diagnostics(ctx.prepare_output())
    ctx.get_state_into(s.buf.numpy())
    if case["prec"] == "mixed" and "diag" in r:
        r["diag"] = {k: v.astype(np.float32) for k, v in r["diag"].items()}
    r["state"] = _typed(s, 0, s.buf)
    return r


# ---------------------------------------------------------------------------
# necessary work


def work(case):
    """Bytes: every input of the pass read once and every output written once
    (the state on the device, its host copy in FP64).  Flops: 7 forward and 4
    inverse real transforms and the pointwise work per right-hand side, the
    filter's and the diagnostics' transforms, the stage combinations."""
    kind, out = case["kind"], case["output"] or case["kind"] == "slice"
    sizes = [m for m, _, _ in _members(case)] if kind == "ensemble" else \
        [(case["nx"], case["ny"], case["nz"])]
    bytes_, flops = 0.0, 0.0
    for n in sizes:
        N, M = n[0] * n[1] * n[2], n[0] * n[1] * (n[2] // 2 + 1)
        ntot = 4 * N + 8 * M + 1
        dev = ntot * (4 if case["prec"] == "mixed" else 8)
        fft = 2.5 * N * math.log2(N)
        rhs = 11 * fft + 60.0 * N + 120.0 * M
        flt = 8 * fft
        diag = (3 * fft + 60.0 * N) if out else 0.0
        steps = 3 if kind == "ensemble" else case["steps"]
        if kind in ("rhs_host", "rhs_dev"):
            bytes_ += 8 * ntot * (3 if case["output"] else 2)
            flops += rhs + (flt + diag if case["output"] else 0.0)
        elif kind == "start":
            bytes_ += 3 * 8 * ntot
            flops += 2 * rhs + flt + 3 * fft
        else:
            bytes_ += dev + 8 * ntot
            per = {"slice": rhs + flt, "rk4": 4 * rhs + flt + 14 * ntot}
            flops += steps * per.get(kind, 12 * rhs + flt + 160 * ntot) + diag
    return {"bytes": bytes_, "flops": flops}


# ---------------------------------------------------------------------------
# the same in 64 bits, with torch's transforms


def _tt(g, d):
    s = {}
    for i in range(3):
        for j in range(i, 3):
            s[i, j] = s[j, i] = g.fft(d[i] * d[j])
    k2 = g.k2.clone()
    k2[0, 0, 0] = 1.0
    K = g.k
    F = [k / k2 for k in K]
    t1 = sum(K[i] * F[i] * s[i, i] for i in range(3))
    t1 = t1 + 2.0 * (K[0] * F[1] * s[0, 1] + K[0] * F[2] * s[0, 2] + K[1] * F[2] * s[1, 2])
    t2 = s[0, 0] + s[1, 1] + s[2, 2]
    S1, S2 = t1 + t2, t1 - t2

    def row(i):
        return K[0] * s[i, 0] + K[1] * s[i, 1] + K[2] * s[i, 2]

    def n_of(a, b, ra, rb):
        c = 0.5 * F[a] * K[b] * S1 + (0.5 * S2 if a == b else 0.0)
        return s[a, b] - F[a] * rb - F[b] * ra + c

    r = [row(i) for i in range(3)]
    n0, n1 = n_of(0, 0, r[0], r[0]), n_of(0, 1, r[0], r[1])
    # kz = 0: the second mode from xz; kz = ky = 0: the modes from yy and yz
    n1[:, 1:, 0] = n_of(0, 2, r[0], r[2])[:, 1:, 0]
    n0[:, 0, 0] = n_of(1, 1, r[1], r[1])[:, 0, 0]
    n1[:, 0, 0] = n_of(1, 2, r[1], r[2])[:, 0, 0]
    n0[0, 0, 0] = n1[0, 0, 0] = 0.0
    return n0, n1


def _rhs(g, f):
    """The right-hand side of state f and what the diagnostics need of it."""
    (phi, dphi, psi, dpsi), (h1, h2, d1, d2), a = g.split(f)
    c = g.fft(phi)
    grad = [g.ifft(1j * k * c) for k in g.kd]
    lap = g.ifft(-g.k2 * c)
    a2 = a * a
    kin = (0.5 - psi) * dphi ** 2
    gr = (0.5 + psi) * (grad[0] ** 2 + grad[1] ** 2 + grad[2] ** 2) / a2
    V = _potential(phi)
    rho, p = kin + gr + V, kin - gr / 3.0 - V
    rm, pm = rho.mean(), p.mean()
    H = torch.sqrt(rm / 3.0)
    out = torch.empty_like(f)
    (o0, o1, o2, o3), (q1, q2, q3, q4), _ = g.split(out)
    o0.copy_(dphi)
    o1.copy_((1 + 4 * psi) * lap / a2 - (3 * H - 4 * dpsi) * dphi -
             (1 + 2 * psi) * MASS * MASS * phi)
    o2.copy_(dpsi)
    o3.copy_(0.5 * p + (psi - 0.5) * pm - 4 * H * dpsi)
    n0, n1 = _tt(g, grad)
    tm = -(2 * pm + g.k2 / a2)
    q1.copy_(d1)
    q2.copy_(d2)
    q3.copy_(tm * h1 - 3 * H * d1 + 2 * n0 / a2)
    q4.copy_(tm * h2 - 3 * H * d2 + 2 * n1 / a2)
    out[-1] = a * H
    return out, {"H": H, "rho": rho, "p": p, "rm": rm}


def _filter(g, f):
    real, _, _ = g.split(f)
    m = g.mask()
    for x in real:
        x.copy_(g.ifft(g.fft(x) * m))


def _bins(g, values):
    nb = g.n[0] // 2
    idx = torch.trunc(nb * torch.sqrt(g.shell2) / g.shell_max - 1e-14).long().clamp(0, nb - 1)
    v = values.clone()
    v[0, 0, 0] = 0.0
    return torch.zeros(nb, dtype=F64, device=DEV).index_add_(0, idx.reshape(-1), v.reshape(-1))


def _exact_diag(g, f, summary_of=None):
    """The diagnostics of the filtered state f; the field summaries are those
    of `summary_of` (a step's start state) where it is given."""
    _, aux = _rhs(g, f)
    (phi, dphi, psi, dpsi), (_, _, d1, d2), a = g.split(f)
    H = aux["H"]
    twice = torch.where(g.kd[2] != 0.0, 2.0, 1.0).to(F64)

    def spectrum(x):
        return _bins(g, g.fft(x).abs() ** 2 * twice / g.N)

    t1 = H * psi + dpsi
    lap_psi = g.ifft(-g.k2 * g.fft(psi))
    ham = lap_psi / (a * a) - 3 * H * t1 - 0.5 * (aux["rho"] - aux["rm"])
    mom = t1 - 0.5 * dphi.mean() * (phi - phi.mean())
    cstr = torch.stack([(ham ** 2).mean(), ham.abs().max(), (mom ** 2).mean(), mom.abs().max()])
    src = g.split(f if summary_of is None else summary_of)[0]
    smry = torch.stack([torch.stack([x.mean(), x.var(), x.min(), x.max()])
                        for x in (*src, aux["rho"], aux["p"])])
    kx, ky, kz = (k.expand(g.k2.shape) for k in g.k)
    a1, a2 = d1.abs() ** 2, d2.abs() ** 2
    x12 = d1.real * d2.real + d1.imag * d2.imag
    one = torch.ones_like(g.k2)
    kzs, kys = torch.where(kz != 0, kz, one), torch.where(ky != 0, ky, one)
    pz = 2 * g.k2 / (kzs ** 2 * (ky ** 2 + kzs ** 2)) * (
        (kx ** 2 + kz ** 2) * a1 + 2 * kx * ky * x12 + (ky ** 2 + kz ** 2) * a2)
    py = 2 * (kx ** 2 + ky ** 2) / kys ** 4 * ((kx ** 2 + ky ** 2) * a1 + ky ** 2 * a2)
    pw = torch.where(kz != 0, pz, torch.where(ky != 0, py, 2 * (a1 + a2))) * twice
    fac = math.pi * 0.01 ** (1 / 3) / (3 * H * H * g.box ** 3)
    gw = _bins(g, fac * g.k2 ** 1.5 * pw / g.N)
    return {"phi_ps": spectrum(phi), "psi_ps": spectrum(psi), "rho_ps": spectrum(aux["rho"]),
            "gw": gw, "cstr": cstr, "smry": smry}


# Dormand-Prince 8(5,3), Hairer, Norsett and Wanner's coefficients: stage,
# weights of the stages before it (the weights of the result last)
_DP = [
    {1: 5.26001519587677318785587544488e-2},
    {1: 1.97250569845378994544595329183e-2, 2: 5.91751709536136983633785987549e-2},
    {1: 2.95875854768068491816892993775e-2, 3: 8.87627564304205475450678981324e-2},
    {1: 2.41365134159266685502369798665e-1, 3: -8.84549479328286085344864962717e-1,
     4: 9.24834003261792003115737966543e-1},
    {1: 3.7037037037037037037037037037e-2, 4: 1.70828608729473871279604482173e-1,
     5: 1.25467687566822425016691814123e-1},
    {1: 3.7109375e-2, 4: 1.70252211019544039314978060272e-1,
     5: 6.02165389804559606850219397283e-2, 6: -1.7578125e-2},
    {1: 3.70920001185047927108779319836e-2, 4: 1.70383925712239993810214054705e-1,
     5: 1.07262030446373284651809199168e-1, 6: -1.53194377486244017527936158236e-2,
     7: 8.27378916381402288758473766002e-3},
    {1: 6.24110958716075717114429577812e-1, 4: -3.36089262944694129406857109825e0,
     5: -8.68219346841726006818189891453e-1, 6: 2.75920996994467083049415600797e1,
     7: 2.01540675504778934086186788979e1, 8: -4.34898841810699588477366255144e1},
    {1: 4.77662536438264365890433908527e-1, 4: -2.48811461997166764192642586468e0,
     5: -5.90290826836842996371446475743e-1, 6: 2.12300514481811942347288949897e1,
     7: 1.52792336328824235832596922938e1, 8: -3.32882109689848629194453265587e1,
     9: -2.03312017085086261358222928593e-2},
    {1: -9.3714243008598732571704021658e-1, 4: 5.18637242884406370830023853209e0,
     5: 1.09143734899672957818500254654e0, 6: -8.14978701074692612513997267357e0,
     7: -1.85200656599969598641566180701e1, 8: 2.27394870993505042818970056734e1,
     9: 2.49360555267965238987089396762e0, 10: -3.0467644718982195003823669022e0},
    {1: 2.27331014751653820792359768449e0, 4: -1.05344954667372501984066689879e1,
     5: -2.00087205822486249909675718444e0, 6: -1.79589318631187989172765950534e1,
     7: 2.79488845294199600508499808837e1, 8: -2.85899827713502369474065508674e0,
     9: -8.87285693353062954433549289258e0, 10: 1.23605671757943030647266201528e1,
     11: 6.43392746015763530355970484046e-1},
    {1: 5.42937341165687622380535766363e-2, 6: 4.45031289275240888144113950566e0,
     7: 1.89151789931450038304281599044e0, 8: -5.8012039600105847814672114227e0,
     9: 3.1116436695781989440891606237e-1, 10: -1.52160949662516086556178806805e-1,
     11: 2.01365400804030348374776537501e-1, 12: 4.47106157277725905176885569043e-2},
]


def _axpy(f, dt, weights, k):
    acc = torch.zeros_like(f)
    for j, w in weights.items():
        acc.add_(k[j], alpha=w)
    return f + dt * acc


def exact(case, seed):
    kind = case["kind"]
    if kind == "ensemble":  # its step sizes are its own controller's
        return None
    n = (case["nx"], case["ny"], case["nz"])
    g = _Grid(n, case["box"])
    f = _input_state(n, case["box"], case["phi0"], seed, psi=True)
    dt, flag = _dt(case), case["output"]
    if kind in ("rhs_host", "rhs_dev"):
        if flag:
            _filter(g, f)
        r = {"result": _rhs(g, f)[0], "field": f}
        if flag:
            r["diag"] = _exact_diag(g, f)
        return r
    if kind == "start":
        _filter(g, f)
        return {"state": f, "dstate": _rhs(g, f)[0]}
    if kind == "slice":
        _filter(g, f)
        return {"diag": _exact_diag(g, f), "state": f}
    if kind == "rk4":
        for _ in range(case["steps"]):
            _filter(g, f)
            k1 = _rhs(g, f)[0]
            k2 = _rhs(g, f + 0.5 * dt * k1)[0]
            k3 = _rhs(g, f + 0.5 * dt * k2)[0]
            k4 = _rhs(g, f + dt * k3)[0]
            f = f + dt * (k1 + 2.0 * k2 + 2.0 * k3 + k4) / 6.0
        return {"state": f}
    _filter(g, f)
    for _ in range(case["steps"]):
        k = {1: _rhs(g, f)[0]}
        for s, w in enumerate(_DP[:-1]):
            k[s + 2] = _rhs(g, _axpy(f, dt, w, k))[0]
        start, f = f, _axpy(f, dt, _DP[-1], k)
        del k
        _filter(g, f)
    r = {"state": f}
    if flag:
        r["diag"] = _exact_diag(g, f, summary_of=start)
    return r
