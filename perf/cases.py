"""What the engine is timed on: forward modelling and gradients of seismic
shots through its public entry points (``engine.Plan`` and
``autograd.seismograms``), over the grids, orders, media and storage options
its users run.

A program that models shots has the acquisition and a plan with its model in
hand, and calls ``Plan.forward`` for each shot; an inversion calls
``forward(save_boundaries=True)``, forms the residual, scales it and calls
``adjoint`` and ``gradient`` for each batch of shots, or differentiates
``autograd.seismograms`` and hands over a new model in every iteration.

Sizes follow the repository's benchmark workloads (2D P-SV 300 x 400; 3D
viscoelastic 256^3; 2D FWI 300 x 1000, 4th order; 3D FWI 200 x 400 x 400) and
its service mix (2D 100-800 x 100-2000, 3D 64-256 cells a side, order 4 or
8, L 0-2, 1-8 shots), with fewer time steps where a whole run would take
seconds; grids are ragged as often as not (the engine wants nz even only).
"""
import math

import numpy as np
import torch

from seiscl_b200.autograd import seismograms
from seiscl_b200.engine import Config, Plan

DH, DT, F0, NAB = 10.0, 1e-3, 20.0, 16
FL = (8.0, 40.0)          # relaxation frequencies (Hz)
TAU = 0.03                # relaxation strength, Q about 50 with two mechanisms
DEV = "cuda"


def _case(name, op, nz, ny, nx, nt, order, L=0, freesurf=1, fields="fp32", shots=1, save="", store="fp32", src=100):
    c = dict(op=op, nz=nz, ny=ny, nx=nx, nt=nt, order=order, L=L, freesurf=freesurf, fields=fields, shots=shots,
             save=save, store=store, src=src)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # a small 2D section, as tutorials and quick tests model: launches and host calls count
        _case("psv2d_small", "model", 100, 0, 150, 500, 4),
        # the benchmark's 2D elastic shot in full
        _case("psv2d", "model", 300, 0, 400, 2000, 8),
        # a large ragged 2D viscoelastic section without a free surface
        _case("visco2d", "model", 602, 0, 1503, 500, 8, L=2, freesurf=0),
        # the benchmark's 3D viscoelastic grid
        _case("visco3d", "model", 256, 256, 256, 100, 8, L=2, src=2),
        # the same physics with wave fields stored in FP16, a smaller grid
        _case("visco3d_fp16", "model", 160, 176, 190, 150, 8, L=2, fields="fp16"),
        # a small 3D elastic box of the service mix
        _case("elastic3d_small", "model", 72, 64, 80, 300, 8),
        # a ragged 3D elastic grid, 4th order
        _case("elastic3d_o4", "model", 130, 121, 147, 200, 4, freesurf=0),
        # a ragged 3D viscoelastic grid, 8th order
        _case("visco3d_ragged", "model", 122, 131, 117, 200, 8, L=1),
        # the 2D FWI gradient grid: 8 shots advanced together, saved boundaries
        _case("fwi2d", "gradient", 300, 0, 1000, 400, 4, freesurf=0, shots=8, save="bnd"),
        # a 3D elastic FWI gradient, boundaries stored in BF16
        _case("fwi3d", "gradient", 100, 200, 200, 120, 8, save="bnd", store="bf16"),
        # a 3D viscoelastic gradient by snapshot checkpointing
        _case("fwi3d_ckpt", "gradient", 96, 92, 104, 120, 8, L=1, save="ckpt"),
        # one iteration of an inversion that differentiates the modelling: new model, forward, backward
        _case("autograd2d", "autograd", 240, 0, 480, 600, 8, freesurf=0, shots=4),
    ]


def draw(rng):
    """One more case of these ranges; its cost stays below the largest listed one's."""
    op = rng.choice(["model", "model", "model", "gradient", "gradient", "autograd"])
    three = op != "autograd" and rng.random() < 0.55

    def size(lo, hi, step=1):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) // step * step

    order, L, fs = rng.choice([4, 8]), rng.choice([0, 0, 1, 2]), rng.choice([0, 1])
    if three:
        nz, ny, nx = size(64, 240, 2), size(64, 240), size(64, 240)
    else:
        nz, ny, nx = size(100, 800, 2), 0, size(100, 2000)
    c = _case("", op, nz, ny, nx, 0, order, L=L, freesurf=fs, src=rng.choice([100, 2]))
    if op == "model":
        if three and rng.random() < 0.3:
            c["fields"] = "fp16"
    else:
        c["src"] = 100
        if op == "gradient" and three:
            c["save"] = rng.choice(["bnd", "ckpt"])
            if c["save"] == "bnd":
                c["store"], c["L"] = rng.choice(["fp32", "bf16"]), 0
            # snapshots of a larger grid are a matter of memory, not of speed
            c["nz"], c["ny"], c["nx"] = min(nz, 128), min(ny, 160), min(nx, 160)
        else:
            c["L"], c["shots"] = 0, rng.randint(1, 8)
            if op == "gradient":
                c["save"], c["nx"] = "bnd", min(nx, 1200)
            else:
                c["freesurf"], c["shots"] = 0, min(c["shots"], 4)
                c["nz"], c["nx"] = min(nz, 400), min(nx, 1000)
    # steps: as many as keep a pass near 0.1 s, and no fewer than let the waves reach the receivers
    cells = c["nz"] * max(c["ny"], 1) * c["nx"] * c["shots"]
    c["nt"] = int(min(rng.uniform(100, 400) if three else rng.uniform(300, 1500),
                      max(100, (1.0e9 if op == "model" else 3e8) / cells)))
    return c


# ------------------------------------------------------------------ inputs
def _nd(case):
    return 3 if case["ny"] else 2


def _shape(case):
    return (case["nx"], case["ny"], case["nz"]) if case["ny"] else (case["nx"], case["nz"])


def _model(case, seed, base=0):
    """A seeded layered model with smooth lateral variations, [nx][(ny)][nz]
    float32: vp 2000-4000 m/s, vs = vp / 1.8 (smoothly varied), density from
    Gardner's relation, constant relaxation strengths."""
    g = torch.Generator().manual_seed(1000 * seed + base)
    shape = _shape(case)
    nz = shape[-1]
    depth = torch.sort(torch.randint(8, nz - 8, (5,), generator=g)).values
    vals = torch.sort(torch.rand(6, generator=g) * 1900 + 2000).values
    layer = vals[torch.searchsorted(depth, torch.arange(nz), right=True)].to(DEV)

    def smooth():
        coarse = torch.randn((1, 1) + tuple(max(2, n // 12) for n in shape), generator=g).to(DEV)
        mode = "trilinear" if len(shape) == 3 else "bilinear"
        return torch.nn.functional.interpolate(coarse, size=shape, mode=mode, align_corners=True)[0, 0].clamp(-2, 2)

    vp = layer * (1 + 0.02 * smooth())
    vs = vp / 1.8 * (1 + 0.01 * smooth())
    m = {"vp": vp, "vs": vs, "rho": 310.0 * vp ** 0.25}
    if case["L"]:
        m["taup"] = TAU * (1 + 0.1 * smooth())
        m["taus"] = TAU * (1 + 0.1 * smooth())
    return {k: np.ascontiguousarray(v.float().cpu().numpy()) for k, v in m.items()}


def _ricker(nt):
    t = np.arange(nt) * DT - 1.2 / F0
    a = (math.pi * F0 * t) ** 2
    return ((1 - 2 * a) * np.exp(-a)).astype(np.float32)[None, :]


def _shots(case, seed):
    """[(src_pos, src, rec_pos)]: sources near the surface (below the
    absorbing layer without a free surface), receivers on a line in 2D and
    on a patch in 3D."""
    rng = np.random.default_rng(seed)
    top = 5 if case["freesurf"] else NAB + 5
    out = []
    for s in range(case["shots"]):
        at = [rng.integers(NAB + 8, n - NAB - 8) for n in (case["nx"], case["ny"] or 1000)]
        sp = np.array([[at[0] * DH, at[1] * DH if case["ny"] else 0.0, top * DH, s, case["src"]]], np.float32)
        if case["ny"]:
            gx, gy = np.meshgrid(np.arange(NAB + 2, case["nx"] - NAB - 2, 4), np.arange(NAB + 2, case["ny"] - NAB - 2, 4),
                                 indexing="ij")
            gx, gy = gx.ravel(), gy.ravel()
        else:
            gx = np.arange(NAB + 2, case["nx"] - NAB - 2, 2)
            gy = np.zeros_like(gx)
        rp = np.zeros((len(gx), 8), np.float32)
        rp[:, 0], rp[:, 1], rp[:, 2] = gx * DH, gy * DH, (top + 3) * DH
        rp[:, 3], rp[:, 4] = s, np.arange(1, len(gx) + 1)
        out.append((sp, _ricker(case["nt"]), rp))
    return out


def _outputs(case):
    return ["vx", "vy", "vz"] if case["ny"] else ["vx", "vz"]


def _observed(case, shots):
    """Observed traces: a direct arrival at 2500 m/s with geometric decay,
    of the size of a modelled one."""
    obs = []
    for sp, src, rp in shots:
        d = np.sqrt(((rp[:, :3] - sp[0, :3]) ** 2).sum(1)) + DH
        t = np.arange(case["nt"]) * DT
        a = (math.pi * F0 * (t[None, :] - 1.2 / F0 - d[:, None] / 2500.0)) ** 2
        w = ((1 - 2 * a) * np.exp(-a) * ((1e-11 if case["ny"] else 1e-10) * DH / d[:, None])).astype(np.float32)
        obs.append({n: w for n in _outputs(case)})
    return obs


def _config(case):
    N = [case["nz"], case["ny"], case["nx"]] if case["ny"] else [case["nz"], case["nx"]]
    return Config(N=N, ND=_nd(case), dh=DH, dt=DT, NT=case["nt"], L=case["L"], f0=F0, FL=FL[:max(1, case["L"])],
                  FDORDER=case["order"], freesurf=case["freesurf"], abs_type=1, nab=NAB, VPPML=3500.0, FPML=F0,
                  field_precision=case["fields"], precision=case["store"], batch=case["shots"] if case["op"] == "gradient" else 1,
                  checkpoint=50 if case["save"] == "ckpt" else 0)


def prepare(case, seed):
    torch.cuda.current_device()   # the plan takes the current device
    torch.zeros(1, device=DEV)
    st = {"case": case, "plan": Plan(_config(case)), "shots": _shots(case, seed)}
    m = _model(case, seed)
    if case["op"] == "autograd":
        # a torch program holds its model as tensors [nz][(ny)][nx]
        st["model"] = [torch.from_numpy(np.ascontiguousarray(m[k].T)).to(DEV) for k in ("vp", "vs", "rho")]
        st["observed"] = torch.from_numpy(np.stack([np.stack([o[n] for n in _outputs(case)]) for o in
                                                    _observed(case, st["shots"])])).to(DEV)
        return st
    st["plan"].set_model(m["vp"], m["vs"], m["rho"], m.get("taup"), m.get("taus"))
    if case["op"] == "gradient":
        st["observed"] = _observed(case, st["shots"])
    return st


def run(state):
    case, plan, shots = state["case"], state["plan"], state["shots"]
    outs = _outputs(case)
    if case["op"] == "model":
        sp, src, rp = shots[0]
        return plan.forward(sp, src, rp, outs)
    if case["op"] == "gradient":
        plan.zero_gradient()
        data = plan.forward_batch(shots, outs, save_boundaries=True)
        res = [plan.residual_scale(s[2], {n: d[n] - o[n] for n in outs})
               for s, d, o in zip(shots, data, state["observed"])]
        plan.adjoint_batch(shots, res)
        return {"data": data, "gradient": plan.gradient()}
    m = [t.clone().requires_grad_(True) for t in state["model"]]
    data = seismograms(plan, *m, shots, outs)
    loss = 0.5 * (data - state["observed"]).square().sum() * 1e20
    loss.backward()
    return {"data": data.detach(), "gradient": [t.grad for t in m]}


# -------------------------------------------------------------------- work
def work(case):
    """A time step reads and writes every wave field and memory variable once
    and reads every material parameter once, in their storage types; a
    gradient run steps the forward field twice (on, and back or again), the
    adjoint field once, and reads and writes three FP64 sums."""
    n = case["nz"] * max(1, case["ny"]) * case["nx"]
    three = bool(case["ny"])
    L, F = case["L"], case["order"] // 2
    nw, ns, nv = (9, 6, 3) if three else (5, 3, 2)
    npar = nv + (5 if three else 3) + (0 if L == 0 else (5 if three else 3))
    elem = 2 if case["fields"] == "fp16" else 4
    state, par = 2 * elem * (nw + ns * L), 4 * npar
    deriv = (18 if three else 8) * 3 * F
    flops = deriv + (4 * ns + 2 * nv) + 14 * ns * L
    if case["op"] == "model":
        b, f = state + par, flops
    else:
        b, f = 3 * state + 2 * par + 48, 3 * flops + 60
        if case["op"] == "autograd":   # the modelling before the backward pass
            b, f = b + state + par, f + flops
    steps = n * case["nt"] * case["shots"]
    return {"bytes": float(b) * steps, "flops": float(f) * steps}


def tolerance(case):
    if case["fields"] == "fp16":
        return {"rel": 2.5e-2}      # 11-bit fields rounded once a step
    if case["store"] == "bf16":
        return {"rel": 3e-2}        # 8-bit saved boundaries: 1e-2 measured, dominated by their rounding
    if case["op"] == "model":
        return {"rel": 5e-6}        # FP32 sums over some hundred steps
    return {"rel": 3e-5}            # gradients: up to 5e-6 measured, boundary shells amplify rounding a little


# ----------------------------------------------------------- 64-bit answers
_HOLBERG = {4: (1.1382, -0.046414), 8: (1.2257, -0.099537, 0.018063, -0.0026274)}


def _f(x):
    return float(np.float32(x))


class _Fd64:
    """The staggered-grid scheme in FP64 torch: CPML (Komatitsch and Martin
    2007), free surface by imaging, relaxation mechanisms, and its adjoint.
    Arrays are [shot][nx][(ny)][nz], wave fields padded by F on every axis."""

    def __init__(self, case, model):
        self.c, self.F, self.L = case, case["order"] // 2, case["L"]
        self.ax = "xyz" if case["ny"] else "xz"
        self.B = case["shots"]
        self.dt, self.dh, self.fs = _f(DT), _f(DH), case["freesurf"]
        self.hc = [_f(v) for v in _HOLBERG[case["order"]]]
        self.shape = _shape(case)
        self._params(model)
        self._cpml_profiles()
        self.pairs = [a + a for a in self.ax] + ([p for p in ("xy", "yz", "xz")] if case["ny"] else ["xz"])
        self.names = ["v" + a for a in self.ax] + ["s" + p for p in self.pairs]

    # parameters scaled by dt/dh, averaged onto the staggered positions
    def _params(self, m):
        t = {k: torch.from_numpy(v).to(DEV).double() for k, v in m.items()}
        s = self.dt / self.dh
        M, mu = t["vp"] ** 2 * t["rho"] * s, t["vs"] ** 2 * t["rho"] * s
        L = self.L
        self.eta = [2 * math.pi * _f(f) * self.dt for f in FL[:L]]
        if L:
            w = 2 * math.pi * _f(F0)
            u = sum((w * self.dt / e) ** 2 / (1 + (w * self.dt / e) ** 2) for e in self.eta)
            M, mu = M / (1 + u * t["taup"]), mu / (1 + u * t["taus"])
        b = self.dt / (self.dh * t["rho"])
        self.M, self.mu, self.b0 = M, mu, b
        taup, taus = (t["taup"], t["taus"]) if L else (0 * M, 0 * M)
        self.buoy = {a: self._ave1(b, i) for i, a in enumerate(self.ax)}
        self.gm, self.fm = M * (1 + L * taup), 2 * mu * (1 + L * taus)
        self.e, self.d = M * taup / self.dt, 2 * mu * taus / self.dt
        self.fs_, self.ds_ = {}, {}
        for i, a in enumerate(self.ax):
            for j, c in enumerate(self.ax):
                if j > i:
                    h, ts = self._ave2(mu, i, j, True), self._ave2(taus, i, j, False)
                    self.fs_[a + c], self.ds_[a + c] = h * (1 + L * ts), h * ts / self.dt

    @staticmethod
    def _ave1(p, d):
        out, n = p.clone(), p.shape[d]
        out.narrow(d, 0, n - 1).copy_(0.5 * (p.narrow(d, 0, n - 1) + p.narrow(d, 1, n - 1)))
        return out

    @staticmethod
    def _ave2(p, d, e, harmonic):
        out, n, m = torch.zeros_like(p), p.shape[d], p.shape[e]
        q = [p.narrow(d, i, n - 1).narrow(e, j, m - 1) for i in (0, 1) for j in (0, 1)]
        r = 4 / sum(1 / v for v in q) if harmonic else 0.25 * sum(q)
        out.narrow(d, 0, n - 1).narrow(e, 0, m - 1).copy_(r)
        out.narrow(d, n - 1, 1).copy_(p.narrow(d, n - 1, 1))   # the first direction's last slab is copied
        return out

    def _cpml_profiles(self):
        nab, dh, dt = NAB, self.dh, self.dt
        amax = 2 * math.pi * (_f(F0) / 2)
        d0 = -3.0 * 3500.0 * math.log(0.0008) / (2 * nab * dh)

        def at(x):
            p = (nab - x) / nab
            d, K, al = d0 * (0.25 * p + 0.75 * p * p), 1 + p * p, amax * (1 - p)
            b = math.exp(-(d / K + al) * dt)
            return K, (d * (b - 1) / (K * (d + K * al)) if abs(d) > 1e-6 else 0.0), b

        full, half = [at(i) for i in range(nab + 1)], [at(i + 0.5) for i in range(nab)]
        # near side k = 0..nab-1; far side: full nodes nab..1, half nodes nab-1..0
        self.prof = {(h, side): torch.tensor(v, dtype=torch.float64, device=DEV).T for h, side, v in (
            (0, 0, full[:nab]), (0, 1, full[:0:-1]), (1, 0, half), (1, 1, half[::-1]))}

    def zeros(self):
        pad = [self.B] + [n + 2 * self.F for n in self.shape]
        f = {n: torch.zeros(pad, dtype=torch.float64, device=DEV) for n in self.names}
        f["r"] = {p: [torch.zeros([self.B] + list(self.shape), dtype=torch.float64, device=DEV) for _ in range(self.L)]
                  for p in self.pairs}
        return f

    def inner(self, a):
        for d in range(1, a.dim()):
            a = a.narrow(d, self.F, a.shape[d] - 2 * self.F)
        return a

    def diff(self, a, axis, fwd):
        d, F = 1 + self.ax.index(axis), self.F
        for k in range(1, a.dim()):
            if k != d:
                a = a.narrow(k, F, a.shape[k] - 2 * F)
        n, out = a.shape[d] - 2 * F, None
        for m in range(1, F + 1):
            hi, lo = (m, 1 - m) if fwd else (m - 1, -m)
            t = self.hc[m - 1] * (a.narrow(d, F + hi, n) - a.narrow(d, F + lo, n))
            out = t if out is None else out.add_(t)
        return out

    def cpml(self, psi, key, q, axis, half):
        d = 1 + self.ax.index(axis)
        n = q.shape[d]
        for side in (0, 1):
            if axis == "z" and side == 0 and self.fs:
                continue
            s = q.narrow(d, 0 if side == 0 else n - NAB, NAB)
            K, a, b = (v.view([-1 if k == d else 1 for k in range(q.dim())]) for v in self.prof[half, side])
            old = psi.get((key, axis, side))
            p = a * s if old is None else b * old + a * s
            psi[key, axis, side] = p
            s.copy_(s / K + p)
        return q

    def vel_rates(self, f, psi):
        out = {}
        for c in self.ax:
            acc = 0
            for a in self.ax:
                q = self.diff(f["s" + "".join(sorted(a + c))], a, a == c)
                acc = acc + (self.cpml(psi, "s" + "".join(sorted(a + c)), q, a, int(a == c)) if psi is not None else q)
            out[c] = acc * self.buoy[c]
        return out

    def strains(self, f, psi):
        out = {}
        for c in self.ax:
            for a in self.ax:
                q = self.diff(f["v" + c], a, a != c)
                out[c + a] = self.cpml(psi, "v" + c, q, a, int(a != c)) if psi is not None else q
        return out

    def stress_rates(self, e):
        tr = sum(e[a + a] for a in self.ax)
        r = {}
        for p in self.pairs:
            if p[0] == p[1]:
                r[p] = (self.gm * tr - self.fm * (tr - e[p]), self.e * tr - self.d * (tr - e[p]))
            else:
                g = e[p] + e[p[::-1]]
                r[p] = (self.fs_[p] * g, self.ds_[p] * g)
        return r

    def step(self, f, psi):
        """velocities, stresses and memory variables, in place; the strains"""
        for c, r in self.vel_rates(f, psi).items():
            self.inner(f["v" + c]).add_(r)
        e = self.strains(f, psi)
        for p, (rate, mem) in self.stress_rates(e).items():
            s = self.inner(f["s" + p])
            s.add_(rate)
            for l, r in enumerate(f["r"][p]):
                h = self.eta[l] / 2
                s.add_(r, alpha=self.dt / 2)
                r.copy_((r * (1 - h) - self.eta[l] * mem) / (1 + h))
                s.add_(r, alpha=self.dt / 2)
        return e

    def surface(self, f, e):
        F, nl = self.F, self.ax[:-1]
        row = lambda a, k: a.narrow(a.dim() - 1, F + k, 1)   # noqa: E731
        row(f["szz"], 0).zero_()
        for r in f["r"]["zz"]:
            r[..., 0] = 0
        for m in range(1, F + 1):
            row(f["szz"], -m).copy_(-row(f["szz"], m))
            for a in nl:
                row(f["s" + a + "z"], -m).copy_(-row(f["s" + a + "z"], m - 1))
        hv, vz = sum(e[a + a][..., 0] for a in nl), e["zz"][..., 0]
        gm, fm, d, ee = (p[..., 0] for p in (self.gm, self.fm, self.d, self.e))
        h = -((gm - fm) ** 2 * hv / gm) - (gm - fm) * vz
        for a in nl:
            s = self.inner(f["s" + a + a])[..., 0]
            s += h
            for l, r in enumerate(f["r"][a + a]):
                s -= self.dt / 2 * r[..., 0]
                r[..., 0] += self.eta[l] / (1 + self.eta[l] / 2) * ((d - ee) * (fm / gm - 1) * hv - (d - ee) * vz)
                s += self.dt / 2 * r[..., 0]

    def points(self, shots):
        F = self.F
        idx = lambda p: [torch.from_numpy(np.rint(p[:, "xyz".index(a)] / DH).astype(np.int64) + F).to(DEV)   # noqa: E731
                         for a in self.ax]
        self.src = [(tuple([b] + [int(v[0]) for v in idx(sp)]), src[0].astype(np.float64)) for b, (sp, src, _) in enumerate(shots)]
        self.rec = [idx(rp) for _, _, rp in shots]
        self.rec_all = [torch.cat([torch.full_like(r[0], b) for b, r in enumerate(self.rec)])] + [
            torch.cat([r[k] for r in self.rec]) for k in range(len(self.ax))]
        self.cut = np.cumsum([0] + [len(r[0]) for r in self.rec])

    def add_sources(self, f, t, sign):
        for at, src in self.src:
            if sign < 0 and self.fs and at[-1] < 2 * self.F:
                continue
            amp = sign * self.dt * float(src[t])
            for n, q in ([("vz", amp)] if self.c["src"] == 2 else [("s" + a + a, amp / len(self.ax)) for a in self.ax]):
                f[n][at] += q

    def shell(self):
        """the saved boundary: the outermost F cells of the grid inside the absorbing layers"""
        box, core = [], []
        for k, n in enumerate(self.shape):
            z = torch.arange(n, device=DEV)
            lo = 0 if self.fs and k == len(self.shape) - 1 else NAB
            box.append((z >= lo) & (z < n - NAB))
            core.append((z >= lo + self.F) & (z < n - NAB - self.F))
        grid = lambda v: (v[0][:, None, None] & v[1][None, :, None] & v[2][None, None, :] if len(v) == 3   # noqa: E731
                          else v[0][:, None] & v[1][None, :])
        return grid(box) & ~grid(core)

    def forward(self, outs, keep=None):
        """traces {name: [all receivers][nt]}; keep = "bnd" or "all": what the adjoint needs of every step"""
        f, psi, nt = self.zeros(), {}, self.c["nt"]
        data = {n: torch.zeros((len(self.rec_all[0]), nt), dtype=torch.float64, device=DEV) for n in outs}
        mask, hist = self.shell() if keep == "bnd" else None, []
        for t in range(nt):
            self.add_sources(f, t, 1)
            if keep == "all":
                hist.append({n: self.inner(f[n]).clone() for n in self.names})
            e = self.step(f, psi)
            if keep == "bnd":
                hist.append({n: self.inner(f[n])[:, mask] for n in self.names})
            if self.fs:
                self.surface(f, e)
            for n in outs:
                data[n][:, t] = f[n][tuple(self.rec_all)]
        self.state = (f, psi, mask, hist)
        return data

    def scaled(self, res):
        """residuals as adjoint sources: times the buoyancy at (x, x, x) of each receiver and dt"""
        out = {}
        for n, r in res.items():
            x = self.rec_all[1] - self.F
            pos = (x * self.shape[1] + x) * self.shape[2] + x if len(self.ax) == 3 else x * self.shape[1] + x
            out[n] = r * (self.buoy[n[1]].reshape(-1)[pos] / self.dh * self.dt * self.dt)[:, None]
        return out

    def surface_adj(self, w):
        F, nl = self.F, self.ax[:-1]
        M, mu = self.M[..., 0], self.mu[..., 0]
        sxx, szz = self.inner(w["sxx"])[..., 0].clone(), self.inner(w["szz"])[..., 0].clone()
        if len(nl) == 1:
            lx = -(M * sxx + (2 * mu - M) * szz) / (4 * M * mu - 4 * mu * mu)
            ly, tot = 0, lx
        else:   # the y component is read from the x one
            a = 1 / (6 * M * mu - 8 * mu * mu)
            lx = ly = a * (-2 * (M - mu) * sxx + (2 * mu - M) * (-sxx - szz))
            tot = lx + ly
        q = -((M - 2 * mu) ** 2 / M) * tot
        vz = self.inner(w["vz"])
        for m in range(F):
            vz[..., m] += self.hc[m] * -(M - 2 * mu) * tot * self.buoy["z"][..., m]
        for k, a in enumerate(nl):
            acc, n = torch.zeros_like(q), q.shape[1 + k]
            for m in range(F):
                acc.narrow(1 + k, m, n - m).add_(q.narrow(1 + k, 0, n - m), alpha=self.hc[m])
                acc.narrow(1 + k, 0, n - m - 1).sub_(q.narrow(1 + k, m + 1, n - m - 1), alpha=self.hc[m])
            self.inner(w["v" + a])[..., 0] += acc * self.buoy[a][..., 0]
        self.inner(w["sxx"])[..., 0] = -(M * lx + (M - 2 * mu) * ly)
        if len(nl) == 2:
            self.inner(w["syy"])[..., 0] = -(M * ly + (M - 2 * mu) * lx)
        self.inner(w["szz"])[..., 0] = -((M - 2 * mu) * tot)

    def adjoint(self, res):
        """gradients of M, mu and the density sum; the forward field comes back from its boundary shells (elastic
        media) or, when every step was kept, from those"""
        f, psi, mask, hist = self.state
        w, nax, nt = self.zeros(), len(self.ax), self.c["nt"]
        gM, gmu, gr = (torch.zeros([self.B] + list(self.shape), dtype=torch.float64, device=DEV) for _ in range(3))
        c1 = 1 / (2 * self.M - 2 * self.mu) ** 2 if nax == 2 else 1 / (3 * self.M - 4 * self.mu) ** 2
        c3 = 1 / self.mu ** 2
        for t in range(nt - 1, 0, -1):
            if self.fs:
                self.surface_adj(w)
            for n, r in res.items():
                w[n].index_put_(tuple(self.rec_all), r[:, t], accumulate=True)
            if mask is not None:
                for p, (rate, _) in self.stress_rates(self.strains(f, None)).items():
                    s = self.inner(f["s" + p])
                    s.sub_(rate)
                    s[:, mask] = hist[t - 1]["s" + p]
                s = {p: self.inner(f["s" + p]) for p in self.pairs}
            else:
                s = {p: hist[t]["s" + p] for p in self.pairs}
            ls = {p: r for p, (r, _) in self.stress_rates(self.strains(w, psi)).items()}
            for p, r in ls.items():
                self.inner(w["s" + p]).add_(r)
            norm = [a + a for a in self.ax]
            tr, dM = sum(s[p] for p in norm), c1 * sum(s[p] for p in norm) * sum(ls[p] for p in norm)
            gM -= dM
            gmu -= c3 * sum(s[p] * ls[p] for p in self.pairs if p[0] != p[1])
            if nax == 2:
                gmu += dM - 0.25 * c3 * (s["xx"] - s["zz"]) * (ls["xx"] - ls["zz"])
            else:
                gmu += 4 / 3 * dM - c3 / 6 * sum(ls[p] * (3 * s[p] - tr) for p in norm)
            if mask is not None:
                for a, r in self.vel_rates(f, None).items():
                    v = self.inner(f["v" + a])
                    v.sub_(r)
                    v[:, mask] = hist[t - 1]["v" + a]
                v = {a: self.inner(f["v" + a]) for a in self.ax}
            else:
                v = {a: hist[t]["v" + a] for a in self.ax}
            for a, r in self.vel_rates(w, psi).items():
                self.inner(w["v" + a]).add_(r)
                gr -= v[a] * r
            if mask is not None:
                self.add_sources(f, t, -1)
        gM, gmu, gr = gM.sum(0) / self.dt, gmu.sum(0) / self.dt, gr.sum(0) / self.dt
        rho = self.dt / (self.dh * self.b0)
        M, mu = self.M * self.dh / self.dt, self.mu * self.dh / self.dt
        return {"vp": 2 * (rho * M).sqrt() * gM, "vs": 2 * (rho * mu).sqrt() * gmu, "rho": gr + M / rho * gM + mu / rho * gmu}


def exact(case, seed):
    steps = case["nz"] * max(1, case["ny"]) * case["nx"] * case["nt"] * case["shots"]
    # beyond this the kept history does not fit, or the answer takes too long
    if case["op"] != "model" and (steps * 72 > 70e9 if case["save"] == "ckpt" else steps > 1.2e9):
        return None
    shots, outs = _shots(case, seed), _outputs(case)
    fd = _Fd64(case, _model(case, seed))
    fd.points(shots)
    data = fd.forward(outs, keep={"model": None, "autograd": "bnd"}.get(case["op"], "all" if case["save"] == "ckpt" else "bnd"))
    if case["op"] == "model":
        return {n: d.cpu().numpy() for n, d in data.items()}
    obs = {n: torch.from_numpy(np.concatenate([o[n] for o in _observed(case, shots)])).to(DEV).double() for n in outs}
    unit = 1e20 if case["op"] == "autograd" else 1.0
    g = fd.adjoint(fd.scaled({n: unit * (data[n] - obs[n]) for n in outs}))
    per = [{n: data[n][a:b].cpu().numpy() for n in outs} for a, b in zip(fd.cut[:-1], fd.cut[1:])]
    if case["op"] == "gradient":
        return {"data": per, "gradient": {k: v.cpu().numpy() for k, v in g.items()}}
    for v in g.values():   # zero in the absorbing layers
        for k in range(v.dim()):
            v.narrow(k, 0, NAB).zero_()
            v.narrow(k, v.shape[k] - NAB, NAB).zero_()
    return {"data": np.stack([np.stack([p[n] for n in outs]) for p in per]),
            "gradient": [np.ascontiguousarray(g[k].cpu().numpy().T) for k in ("vp", "vs", "rho")]}
