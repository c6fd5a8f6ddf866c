"""What the engine is used for, as cases that can be timed and checked.

A case is one call of a user's program: a forward-modelling run, an FWI
gradient (forward, residual, time-reversed adjoint, preconditioning), several
surveys' gradients at once, or one shot through the drop-in ``kernel_PSV``.
Time axes are cropped to hundreds of steps so that a pass is short; the
wavelet's peak frequency follows the cropped length, so that the wave has left
the source and the record holds signal.

A plan's numbers cross the C ABI as FP64 arrays whatever its precision is; the
results of an FP32 plan carry 32 bits and are kept in 32 bits here.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from fwi_cuda_gb300 import engine
from fwi_cuda_gb300 import survey as S

BASE = dict(op="gradient", nz=301, nx=601, nt=400, nshot=8, nrec=120, order=4, npml=20,
            layout="surface", snap_dt=3, snap_step=1, precision=32, storage="full", interval=0)


def case(name, **kw):
    return dict(BASE, name=name, **kw)


def listed():
    return [
        # Modelling of one small survey: the smallest call, bound by launches and latency.
        case("model_101x201_1shot", op="forward", nz=101, nx=201, nshot=1, nrec=40, npml=10),
        # The one-shot gradient of the 301 x 601 configuration.
        case("grad_301x601_1shot", nshot=1),
        # The eight-shot gradient of that configuration: the benchmark's own workload.
        case("grad_301x601_8shots"),
        # The same shots' modelling: observed data, and each trial of the step-length search.
        case("model_301x601_8shots", op="forward"),
        # The reference's example layout (wells left and right, CPML on four sides, x-force velocity
        # sources) on an odd grid, order 6, with gradients on every second cell.
        case("grad_crosswell_187x133", nz=187, nx=133, nt=500, nshot=5, nrec=61, order=6, npml=12,
             layout="crosswell", snap_step=2),
        # One batch of the batched-survey configuration (1001 x 2001, order 8): wavefields larger than L2.
        case("grad_1001x2001_8shots", nz=1001, nx=2001, nt=320, nrec=400, order=8, npml=30),
        # Observed data of that survey for a few shots, as a modelling-only program makes them.
        case("model_1001x2001_3shots", op="forward", nz=1001, nx=2001, nt=240, nshot=3, nrec=400,
             order=8, npml=30),
        # A long-record survey on a mid-size ragged grid that keeps states instead of the history.
        case("grad_ckpt_601x1203_4shots", nz=601, nx=1203, nt=300, nshot=4, nrec=200, order=8, npml=30,
             storage="checkpoint", interval=25),
        # FP64 gradient: what a user checks the FP32 engine against.
        case("grad_f64_151x301_2shots", nz=151, nx=301, nt=300, nshot=2, nrec=80, npml=15,
             precision=64),
        # Four uneven surveys, one plan each, in one call.
        case("multi_4_surveys", op="multi", nz=201, nx=401, nshot=2, nrec=80, npml=15),
        # One shot through the reference's own call, wavefields and snapshot history returned to the host.
        case("dropin_101x201", op="dropin", nz=101, nx=201, nt=240, nshot=1, nrec=40, order=2, npml=10),
    ]


def updates(c):
    """Grid-point updates of a pass (a gradient steps twice)."""
    n = sum(z * x * t * s for z, x, t, s in sizes(c))
    return n * (2 if c["op"] in ("gradient", "multi") else 1)


def sizes(c):
    """(nz, nx, nt, shots) of each survey of the case."""
    if c["op"] != "multi":
        return [(c["nz"], c["nx"], c["nt"], c["nshot"])]
    return [(int(c["nz"] * f) | 1, int(c["nx"] * f) | 1, int(c["nt"] * (0.5 + 0.5 * f)), c["nshot"])
            for f in (0.5, 0.8, 1.0, 1.4)]


def draw(rng):
    """Another case of these ranges: 1 to 8 shots on grids from 61 x 91 to 1001 x 2001, orders 2 to 8."""
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    most = updates(BASE | dict(nz=1001, nx=2001, nt=120))
    while True:
        c = dict(BASE)
        c["op"] = rng.choice(["forward", "forward", "gradient", "gradient", "gradient", "multi"])
        c["order"] = rng.choice([2, 4, 4, 6, 8, 8])
        c["nz"], c["nx"] = log(81, 1001), log(121, 2001)
        c["nt"], c["nshot"] = rng.randrange(320, 560), rng.choice([1, 1, 2, 3, 4, 5, 8])
        c["npml"] = rng.randrange(8, 31)
        c["snap_dt"], c["snap_step"] = rng.choice([1, 2, 3, 3, 4]), rng.choice([1, 1, 1, 2])
        c["precision"] = rng.choice([32, 32, 32, 32, 32, 64])
        if c["op"] == "gradient" and rng.random() < 0.3:
            c["storage"], c["interval"] = "checkpoint", rng.randrange(10, 60)
        if c["op"] == "multi":
            c["nz"], c["nx"], c["nshot"] = log(121, 301), log(161, 601), rng.choice([1, 2, 3])
        elif rng.random() < 0.25:
            c["layout"], c["nz"], c["nx"] = "crosswell", log(121, 300), log(101, 160)
        c["nrec"] = rng.randrange(20, max(21, min(200, c["nx"] // 3)))
        cost = updates(c) * (8 if c["precision"] == 64 else 1)
        if 2 * (c["npml"] + c["order"]) + 40 < min(c["nz"], c["nx"]) and cost <= most:
            return c


# ------------------------------------------------------------------- inputs

def build(c, nz, nx, nt, seed):
    """(survey, true model, initial model): dipping layers with anomalies, and their smoothed version a few
    per cent slow, so that the direct waves have a residual too."""
    rng = np.random.default_rng(seed)
    fpad, npml, dx = c["order"] // 2, c["npml"], 0.5
    vp = S.layered_vp(nz, nx, 6, 1800.0, 3000.0, rng, dip_cells=0.05 * nz, top=2 * fpad)
    r = max(4, min(nz, nx) // 16)
    vp = S.add_anomalies(vp, rng, 3, amp=0.10, radius=(r, r), signs=(1, -1), margin=npml + fpad)
    true = S.model_from_vp(vp)
    init = S.smoothed(0.97 * vp, 5.0)
    dt = 5e-5
    fc = min(280.0, max(100.0, 1.5 / (0.3 * nt * dt)))
    if c["layout"] == "surface":
        nrec = c["nrec"]
        spacing = max(1, (nx - 2 * (npml + fpad) - 8) // max(nrec, 1))
        sv = S.surface_survey(nz, nx, dx, dx, nt, dt, fdorder=c["order"],
                              stencil="holberg", npml=npml, nshot=c["nshot"], nrec=nrec,
                              rec_spacing=spacing, fc=fc, vp_max=3300.0, snap_dt=c["snap_dt"],
                              surf_offset=0)
        # gradients below the source's near field, which the taper of an FWI run mutes
        sv.snap_z1 = int(sv.z_src[0]) + 24
    else:
        a, b = npml + fpad + 4, npml + fpad + 1
        n, m = c["nshot"], c["nrec"]
        w = S.ricker(nt, dt, fc)
        sv = S.Survey(nt=nt, nz=nz, nx=nx, dt=dt, dz=dx, dx=dx, fdorder=c["order"], stencil="holberg",
                      npml=(npml,) * 4, damp_v_pml=3300.0, freq_pml=fc, snap_z1=b, snap_z2=nz - b - 1,
                      snap_x1=a + 24, snap_x2=nx - a - 25, snap_dt=c["snap_dt"],
                      taper=(b, b + 4, nz - b, nz - b - 4, b, b + 4, nx - b, nx - b - 4), nshot=n,
                      stf_type=1, z_src=np.linspace(a, nz - a - 1, n).round(), x_src=np.full(n, a),
                      src_shot_to_fire=np.arange(n), stf_z=np.zeros((n, nt)), stf_x=np.stack([w] * n),
                      z_rec=np.linspace(a, nz - a - 1, m).round(), x_rec=np.full(m, nx - a - 1))
        sv.finalize()
    sv.snap_dz = sv.snap_dx = c["snap_step"]
    sv.imaging_sign = 1
    return sv, true, init


def inputs(c, seed):
    return [build(c, nz, nx, nt, seed * 16 + k) for k, (nz, nx, nt, _) in enumerate(sizes(c))]


# ---------------------------------------------------------------- the passes

class State:
    pass


def prepare(c, seed):
    """The plan of each survey with its observed data, and the model of the next call."""
    s = State()
    s.case, s.plans, s.models = c, [], []
    opts = dict(precision=c["precision"], storage=c["storage"], checkpoint_interval=c["interval"])
    for sv, true, init in inputs(c, seed):
        s.models.append(init)
        if c["op"] == "dropin":
            s.survey, s.averages = sv, [t.cpu().numpy() for t in averages(init)[:3]]
            continue
        p = engine.Plan(sv, **opts)
        if c["op"] != "forward":
            p.set_observed(*(t.cpu().numpy() for t in simulate(sv, true)[0]))
        s.plans.append(p)
    return s


def narrow(c, v):
    """A result in the precision of the plan that computed it."""
    if isinstance(v, dict):
        return {k: narrow(c, x) for k, x in v.items()}
    if isinstance(v, (list, tuple)):
        return [narrow(c, x) for x in v]
    return np.asarray(v, np.float32 if c["precision"] == 32 else np.float64)


def scaled(g):
    """Gradients with the moduli in GPa: in SI units their small values leave the range of 32 bits."""
    return [1e18 * g[0], 1e18 * g[1], g[2]]


def run(s):
    c = s.case
    if c["op"] == "forward":
        p = s.plans[0]
        p.set_model(*s.models[0])
        return narrow(c, p.forward())
    if c["op"] == "dropin":
        sv, (mu_zx, rho_zp, rho_xp) = s.survey, s.averages
        lam, mu, _ = s.models[0]
        names = ("a", "b", "K", "a_half", "b_half", "K_half")
        return narrow(c, engine.kernel_PSV(
            0, sv.nt, sv.nz, sv.nx, sv.dt, sv.dx, sv.dz, sv.surf, sv.isurf, sv.hc, sv.fdorder, lam, mu,
            mu_zx, rho_zp, rho_xp, False, sv.pml_z, [getattr(sv, n + "_z") for n in names], sv.pml_x,
            [getattr(sv, n + "_x") for n in names], sv.nsrc, sv.stf_type, sv.stf_z, sv.stf_x, sv.z_src,
            sv.x_src, sv.src_shot_to_fire, sv.nrec, sv.rtf_type, sv.z_rec, sv.x_rec, True,
            (sv.snap_z1, sv.snap_z2, sv.snap_x1, sv.snap_x2, sv.snap_dt, sv.snap_dz, sv.snap_dx),
            stencil=sv.stencil, precision=c["precision"]))
    for p, m in zip(s.plans, s.models):
        p.set_model(*m)
        p.reset_gradient()
    if c["op"] == "multi":
        L2 = engine.multi_gradient(s.plans)
        return narrow(c, [L2] + [scaled(p.get_gradient()) for p in s.plans])
    L2, g = s.plans[0].gradient()
    return narrow(c, [L2, scaled(g)])


def work(c):
    """Models, observed data and wavelets in, traces or gradients (and what else the call returns) out; the
    arithmetic of every grid-point update: eight staggered derivatives of 3 N - 1 operations, the
    updates, and in a gradient the energies, the displacement and the imaging sums."""
    N, wide = c["order"] // 2, c["precision"] // 8
    nbytes, flops = 0, 0.0
    for nz, nx, nt, ns in sizes(c):
        n, trace = nz * nx, 2 * ns * c["nrec"] * nt
        nbytes += 8 * 3 * n + 8 * 2 * nt
        step = 8 * (3 * N - 1) + 18
        if c["op"] == "forward":
            nbytes += 8 * trace
            flops += n * nt * ns * step
        elif c["op"] == "dropin":
            nbytes += 8 * (trace + 16 * n + 5 * n * (1 + (nt - 1) // c["snap_dt"]))
            flops += n * nt * ns * (step + 7)
        else:
            snaps = nt * ns * n // (c["snap_dt"] * c["snap_step"] ** 2)
            nbytes += 8 * trace + 8 * 3 * n
            if c["storage"] == "full":
                nbytes += 2 * 5 * wide * snaps
            flops += n * nt * ns * (2 * step + 10) + 25 * snaps
    return {"bytes": int(nbytes), "flops": float(flops)}


# ------------------------------------------------------ the same in 64 bits

def f64(a):
    return torch.as_tensor(np.asarray(a, np.float64), device="cuda" if torch.cuda.is_available() else "cpu")


def averages(model):
    """Harmonic mu and arithmetic buoyancies on the staggered points (zero in the last row and column), and
    the mean of each parameter over the other cells."""
    lam, mu, rho = (f64(a) for a in model)
    mu_zx, rho_zp, rho_xp = (torch.zeros_like(mu) for _ in range(3))
    mu_zx[:-1, :-1] = 4 / (1 / mu[:-1, :-1] + 1 / mu[:-1, 1:] + 1 / mu[1:, :-1] + 1 / mu[1:, 1:])
    rho_zp[:-1, :-1] = 1 / (0.5 * (rho[:-1, :-1] + rho[1:, :-1]))
    rho_xp[:-1, :-1] = 1 / (0.5 * (rho[:-1, :-1] + rho[:-1, 1:]))
    return mu_zx, rho_zp, rho_xp, [a[:-1, :-1].mean() for a in (lam, mu, rho)]


class Wave:
    """The velocity-stress time loop of every shot of a survey: fields [shot][nz][nx], one call a step."""

    def __init__(self, sv, model):
        self.sv, fp = sv, sv.fdorder // 2
        self.Z, self.X = (fp, sv.nz - fp), (fp, sv.nx - fp)
        self.I = (slice(None), slice(*self.Z), slice(*self.X))
        ns = fp if sv.stencil == "holberg" else 1
        self.hc = [float(h) for h in sv.hc[1:ns + 1]]
        self.lam, self.mu, self.rho = (f64(a) for a in model)
        self.mu_zx, self.rho_zp, self.rho_xp, self.mean = averages(model)
        self.vz, self.vx, self.szz, self.szx, self.sxx, self.uz, self.ux, self.We = (
            torch.zeros((sv.nshot, sv.nz, sv.nx), dtype=torch.float64, device=self.lam.device)
            for _ in range(8))
        self.strips, self.memory = {}, {}
        for half in ("", "_half"):
            for axis, (lo, hi) in (("z", self.Z), ("x", self.X)):
                a, b, K = (np.asarray(getattr(sv, n + half + "_" + axis))[lo:hi] for n in "abK")
                on = np.flatnonzero((a != 0) | (b != 1) | (K != 1))
                cut = np.split(on, np.flatnonzero(np.diff(on) > 1) + 1) if on.size else []
                shape = (-1, 1) if axis == "z" else (1, -1)
                self.strips[axis, half] = [
                    (slice(int(i[0]), int(i[-1]) + 1),
                     [f64(v[i[0]:i[-1] + 1]).reshape(shape) for v in (a, b, 1 / K)]) for i in cut]

    def d(self, f, axis, ahead, half, name):
        """Staggered derivative of f over the interior, forward (ahead = 1) or backward, with its CPML."""
        sv, (z1, z2), (x1, x2) = self.sv, self.Z, self.X
        h, out = (sv.dz if axis == "z" else sv.dx), None
        for k, c in enumerate(self.hc, 1):
            i, j = k - 1 + ahead, ahead - k
            if axis == "z":
                t = f[:, z1 + i:z2 + i, x1:x2] - f[:, z1 + j:z2 + j, x1:x2]
            else:
                t = f[:, z1:z2, x1 + i:x2 + i] - f[:, z1:z2, x1 + j:x2 + j]
            out = t.mul_(c / h) if out is None else out.add_(t, alpha=c / h)
        for n, (at, (a, b, ki)) in enumerate(self.strips[axis, half]):
            part = out[:, at] if axis == "z" else out[:, :, at]
            m = self.memory.get((name, axis, n))
            m = self.memory[name, axis, n] = a * part if m is None else m.mul_(b).add_(a * part)
            part.mul_(ki).add_(m)
        return out

    def step(self, displacement):
        """Stresses, then velocities, of one step (before injection); u and We with them."""
        sv, I = self.sv, self.I
        C = (slice(*self.Z), slice(*self.X))
        dt, lam, l2m = sv.dt, self.lam[C], (self.lam + 2 * self.mu)[C]
        vz_z, vx_x = self.d(self.vz, "z", 0, "", "vz"), self.d(self.vx, "x", 0, "", "vx")
        vx_z, vz_x = self.d(self.vx, "z", 1, "_half", "vx"), self.d(self.vz, "x", 1, "_half", "vz")
        old = self.sxx[:, sv.isurf[0]].clone() if sv.surf else None
        self.szz[I] += dt * (l2m * vz_z + lam * vx_x)
        self.sxx[I] += dt * (lam * vz_z + l2m * vx_x)
        self.szx[I] += dt * self.mu_zx[C] * (vx_z + vz_x)
        if sv.surf:  # traction-free row: sxx from the plane-stress modulus, nothing else
            st, x = sv.isurf[0], slice(*self.X)
            fs = 4 * dt * (lam * self.mu[C] + self.mu[C] ** 2) / l2m
            self.szz[:, st, x] = 0
            self.szx[:, st, x] = 0
            self.sxx[:, st] = old
            self.sxx[:, st, x] = fs[st - self.Z[0]] * vx_x[:, st - self.Z[0]]
            for k in range(1, st - self.Z[0] + 1):
                self.szz[:, st - k, x] = -self.szz[:, st + k, x]
                self.szx[:, st - k, x] = -self.szx[:, st + k, x]
        szz_z, sxx_x = self.d(self.szz, "z", 1, "", "szz"), self.d(self.sxx, "x", 1, "", "sxx")
        szx_z, szx_x = self.d(self.szx, "z", 0, "_half", "szx"), self.d(self.szx, "x", 0, "_half", "szx")
        if displacement:
            self.uz[I] += dt * self.vz[I]
            self.ux[I] += dt * self.vx[I]
        self.vz[I] += dt * self.rho_zp[C] * szz_z.add_(szx_x)
        self.vx[I] += dt * self.rho_xp[C] * sxx_x.add_(szx_z)
        self.We[I] += self.vx[I] ** 2 + self.vz[I] ** 2

    def inject(self, shot, pos, az, ax, kind):
        """Adds amplitudes az, ax at flat cells pos of shots `shot` (kind 0: forces, 1: velocities)."""
        n = self.sv.nz * self.sv.nx
        for v, a, r in ((self.vz, az, self.rho_zp), (self.vx, ax, self.rho_xp)):
            if kind == 0:
                a = self.sv.dt * r.reshape(-1)[pos] * a / (self.sv.dz * self.sv.dx)
            v.view(-1).index_add_(0, shot * n + pos, a)


def window(sv):
    return (slice(None), slice(sv.snap_z1, sv.snap_z2 + 1, sv.snap_dz),
            slice(sv.snap_x1, sv.snap_x2 + 1, sv.snap_dx))


def cells(z, x, nx, dev):
    return torch.as_tensor(np.asarray(z, np.int64) * nx + np.asarray(x, np.int64), device=dev)


def simulate(sv, model, keep=False, displacement=False):
    """((uz, ux) traces [shot][rec][nt], wave, snapshots): forward modelling of every shot."""
    w = Wave(sv, model)
    dev = w.vz.device
    rec = cells(sv.z_rec, sv.x_rec, sv.nx, dev)
    src = cells(sv.z_src, sv.x_src, sv.nx, dev)
    fire = torch.as_tensor(np.asarray(sv.src_shot_to_fire, np.int64), device=dev)
    fz, fx = f64(sv.stf_z), f64(sv.stf_x)
    traces = [torch.zeros((sv.nshot, sv.nrec, sv.nt), dtype=torch.float64, device=dev) for _ in range(2)]
    W, history = window(sv), []
    for it in range(sv.nt):
        w.step(displacement)
        w.inject(fire, src, fz[:, it], fx[:, it], sv.stf_type)
        for t, v in zip(traces, (w.vz, w.vx)):
            t[:, :, it] = v.view(sv.nshot, -1)[:, rec] * (sv.dt / (sv.dz * sv.dx))
        if keep and it % sv.snap_dt == 0:
            history.append([w.szz[W].clone(), w.szx[W].clone(), w.sxx[W].clone(), w.vz[W] / sv.dt,
                            w.vx[W] / sv.dt])
    return [t.cumsum_(2) for t in traces], w, history


def between(out, sv):
    """Fills the cells between the imaged ones by lines along x, then along z, inside the half-open window."""
    z1, z2, x1, x2, dz, dx = sv.snap_z1, sv.snap_z2, sv.snap_x1, sv.snap_x2, sv.snap_dz, sv.snap_dx
    if dx > 1:
        rows = torch.arange(z1, z2, dz, device=out.device)
        for x in range(x1, x2, dx):
            t = (out[rows, x + dx] - out[rows, x]) / dx
            for k in range(1, dx):
                out[rows, x + k] = out[rows, x] + t * k
    if dz > 1:
        for z in range(z1, z2, dz):
            t = (out[z + dz, x1:x2] - out[z, x1:x2]) / dz
            for k in range(1, dz):
                out[z + k, x1:x2] = out[z, x1:x2] + t * k
    return out


def gradient(sv, true, init):
    """[L2, [dlam, dmu, drho]] of one FWI gradient of every shot, as Plan.gradient returns it."""
    obs = simulate(sv, true)[0]
    mod, fwd, history = simulate(sv, init, keep=True)
    res = [m - o for m, o in zip(mod, obs)]
    L2 = float(sum((0.5 * sv.dt * r * r).sum() for r in res))
    w = Wave(sv, init)
    rec = cells(sv.z_rec, sv.x_rec, sv.nx, w.vz.device)
    pos, shot = rec.repeat(sv.nshot), torch.arange(sv.nshot, device=rec.device).repeat_interleave(sv.nrec)
    W = window(sv)
    kimg = sv.snap_dt * sv.dt
    g1 = (kimg * 0.25 / (w.lam + w.mu) ** 2)[W[1:]]
    g2 = (kimg / w.mu ** 2)[W[1:]]
    g = [torch.zeros_like(w.vz[W]) for _ in range(3)]
    for it in reversed(range(sv.nt)):
        w.step(True)
        if it % sv.snap_dt == 0:
            fzz, fzx, fxx, fvz, fvx = history.pop()
            s1 = g1 * ((fzz + fxx) * (w.szz[W] + w.sxx[W]))
            s23 = g2 * (fzx * w.szx[W] + 0.25 * (fzz - fxx) * (w.szz[W] - w.sxx[W]))
            g[0] -= s1
            g[1] -= s23 + s1
            g[2] -= kimg * (w.ux[W] * fvx + w.uz[W] * fvz)
        w.inject(shot, pos, res[0][:, :, it].reshape(-1), res[1][:, :, it].reshape(-1), sv.rtf_type)
    sign = -1.0 if sv.imaging_sign > 0 else 1.0
    H = (slice(sv.snap_z1, sv.snap_z2), slice(sv.snap_x1, sv.snap_x2))  # the preconditioner's half-open window
    total = [torch.zeros_like(w.lam) for _ in range(3)]
    for s in range(sv.nshot):
        e = (fwd.We[s] * w.We[s]).sqrt()[H]
        e = e + 0.005 * e.max()
        for k in range(3):
            out = w.We[s].clone()
            out[W[1:]] = sign * g[k][s]
            total[k][H] += between(out, sv)[H] / (e * w.mean[k] * w.mean[k])
    return [np.float64(L2), scaled([t.cpu().numpy() for t in total])]


def exact(c, seed):
    """The same results from torch in 64 bits."""
    S_ = inputs(c, seed)
    if c["op"] == "forward":
        return [t.cpu().numpy() for t in simulate(S_[0][0], S_[0][2])[0]]
    if c["op"] == "dropin":
        sv, _, init = S_[0]
        (uz, ux), w, history = simulate(sv, init, keep=True, displacement=True)
        fields = ("vz", "vx", "uz", "ux", "szz", "szx", "sxx", "We")
        out = {k: getattr(w, k)[0].cpu().numpy() for k in fields}
        out["rtf_uz"], out["rtf_ux"] = uz[0].cpu().numpy(), ux[0].cpu().numpy()
        out["history"] = {k: torch.stack([h[i][0] for h in history]).cpu().numpy()
                          for i, k in enumerate(("szz", "szx", "sxx", "vz", "vx"))}
        return out
    each = [gradient(*s) for s in S_]
    if c["op"] == "multi":
        return [np.array([e[0] for e in each])] + [e[1] for e in each]
    return each[0]
