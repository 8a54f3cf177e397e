"""The work this framework is used for, as cases that can be timed and compared.

Each case is one call (or the few calls that belong together) through the
package's public entry points:

* ``mirror``    the reference-named objects: RK3CN_Elin / RK3CN ``Step`` on a
                host-side ``solution``, a few steps (a driver written like the
                reference's main loop; the smallest calls);
* ``single``    one quasi-linear case resident on the device: state in, N steps
                with records, state out, all on device buffers (QLSolver);
* ``forced``    the same with the CFL time step and, where ``f_noise`` is not
                zero, driving noise after every step;
* ``ensemble``  many cases in one launch per call (QLBatch), state in from
                pinned host buffers, N steps with records, state out;
* ``adjoint``   gradient of the mean Maxwell stress for a set of seeds;
* ``dns``       the full 3-D DNS, state in, N steps with records, state out.

Sizes come from params.py (16x16 x NZ=32, 64x64 x NZ=128, 32x32 x NZ=64 adjoint,
64 x 128 x 64 DNS), from the ensemble law of batch.py and from the test suite's
ragged grids.  ``exact`` restates the equations in plain torch (complex128).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from ql_dns_b200.batch import QLBatch
from ql_dns_b200.dns import QLDns
from ql_dns_b200.initial import dns_initial_state, initial_state
from ql_dns_b200.params import DNSParams, QLParams
from ql_dns_b200.solver import RK3CN, MHD_BQlin, MHD_FullQlin, QLSolver, RK3CN_Elin, solution


def listed():
    return [
        # a driver with the reference's main loop on the small case: one Step per call
        dict(name="mirror 16x16 nz32", kind="mirror", model=0, integ=0, nx=16, ny=16, NZ=32, steps=4, every=0),
        # the small test case as a run: launches and latency count
        dict(name="single 16x16 nz32", kind="single", model=0, integ=0, nx=16, ny=16, NZ=32, steps=50, every=10),
        # the production case
        dict(name="single 64x64 nz128", kind="single", model=0, integ=0, nx=64, ny=64, NZ=128, steps=40, every=10),
        # the model with mean flow, Crank-Nicolson, fourth-order dissipation, ordinary size
        dict(name="single full 48x48 nz64 cn", kind="single", model=1, integ=1, nx=48, ny=48, NZ=64, steps=40,
             every=10, order=4),
        # the tallest box, ragged mode grid
        dict(name="single 22x18 nz256", kind="single", model=0, integ=0, nx=22, ny=18, NZ=256, steps=40, every=20),
        # driven run with the variable time step
        dict(name="forced 32x32 nz64", kind="forced", model=0, integ=0, nx=32, ny=32, NZ=64, steps=40, every=10,
             f_noise=0.02),
        # the 48-case parameter study
        dict(name="ensemble 48", kind="ensemble", model=0, integ=0, ncases=48, draw_seed=12345, steps=40, every=20),
        # a parameter study with the mean-flow model
        dict(name="ensemble full 12", kind="ensemble", model=1, integ=0, ncases=12, draw_seed=77, steps=20, every=10),
        # one gradient
        dict(name="adjoint 1 seed", kind="adjoint", integ=0, nx=32, ny=32, NZ=64, seeds=1, steps=100, ckpt=50),
        # the gradients of a set of seeds together
        dict(name="adjoint 16 seeds", kind="adjoint", integ=0, nx=32, ny=32, NZ=64, seeds=16, steps=100, ckpt=50),
        # the production DNS grid
        dict(name="dns 64x128x64", kind="dns", integ=0, Mx=64, My=128, NZ=64, steps=50, every=25, order=2),
        # a small DNS, Crank-Nicolson with fourth-order dissipation
        dict(name="dns 16x32x32 cn", kind="dns", integ=1, Mx=16, My=32, NZ=32, steps=50, every=25, order=4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mirror", "single", "single", "forced", "ensemble", "adjoint", "dns"])
    model, integ = rng.randrange(2), rng.randrange(2)
    every = rng.randrange(5, 15)
    if kind == "dns":
        c = dict(Mx=rng.choice([16, 32, 64]), My=rng.choice([16, 32, 64, 128]), NZ=rng.choice([16, 32, 64]),
                 steps=rng.randrange(10, 45), order=rng.choice([2, 2, 4]))
        return dict(kind=kind, integ=integ, every=every, **c)
    if kind == "ensemble":
        return dict(kind=kind, model=model, integ=integ, ncases=rng.randrange(2, 13), draw_seed=rng.randrange(1000),
                    steps=rng.randrange(8, 20), every=every)
    nx, ny = (2 * (_log_int(rng, 4, 64) // 2) for _ in range(2))
    if kind == "adjoint":
        return dict(kind=kind, integ=integ, nx=min(nx, 32), ny=min(ny, 32), NZ=rng.choice([16, 32, 64]),
                    seeds=rng.randrange(1, 9), steps=rng.randrange(10, 60), ckpt=rng.randrange(5, 30))
    NZ = rng.choice([16, 32, 64, 128, 256] if nx * ny <= 2048 else [16, 32, 64])
    c = dict(kind=kind, model=model, integ=integ, nx=nx, ny=ny, NZ=NZ)
    if kind == "mirror":
        return dict(c, steps=rng.randrange(1, 6), every=0)
    if kind == "forced":
        return dict(c, steps=rng.randrange(8, 40), every=every, f_noise=rng.choice([0.0, 0.02]))
    return dict(c, steps=rng.randrange(8, 40), every=every, order=rng.choice([2, 4]) if model else 2)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
CFL, DT_MAX, K_BAND = 0.1, 0.02, (0.5, 50.0)


def _ql_params(case):
    full = case["model"] == 1
    order = case.get("order", 2)
    re = 4000.0 if order == 2 else 4.0e7  # hyper-dissipation coefficients scale with k^2
    return QLParams(model=case["model"], integrator=case["integ"], nx=case["nx"], ny=case["ny"], NZ=case["NZ"],
                    nu=2.0 / re, eta=1.0 / re, B0z=0.02 if full else 0.0, omega=1.0, viscosity_order=order,
                    dt=0.005 if case["NZ"] >= 128 else 0.01)


def _ql_state(p, seed):
    # sigma well above the linear regime's round-off: the feedback on the mean fields counts
    return initial_state(p, seed, sigma=0.05, B0=0.05, mean_u=0.02 if p.nmf == 4 else 0.0)


def _ensemble(case, seed):
    """Cases of the ensemble law (mode grids, NZ, Rm, Pm) and their states."""
    rng = np.random.default_rng(case["draw_seed"])
    cases, states = [], []
    for c in range(case["ncases"]):
        n, NZ = int(rng.choice((16, 32, 48, 64))), int(rng.choice((32, 64, 128)))
        rm = math.exp(rng.uniform(math.log(500.0), math.log(16000.0)))
        pm, b0 = int(rng.choice((1, 2, 4))), rng.uniform(0.01, 0.1)
        p = QLParams(model=case["model"], integrator=case["integ"], nx=n, ny=n, NZ=NZ, nu=pm / rm, eta=1.0 / rm,
                     dt=0.01, B0z=0.02 if case["model"] else 0.0)
        cases.append(p)
        states.append(initial_state(p, seed * 1000 + c, sigma=1e-3, B0=b0, mean_u=0.02 if case["model"] else 0.0))
    return cases, states


def _dns_params(case):
    order = case["order"]
    re = 4000.0 if order == 2 else 4.0e7
    return DNSParams(integrator=case["integ"], Mx=case["Mx"], My=case["My"], NZ=case["NZ"], nu=1.0 / re, eta=1.0 / re,
                     viscosity_order=order, dt=0.005, B0z=0.01)


def _adjoint_params(case):
    return QLParams(nx=case["nx"], ny=case["ny"], NZ=case["NZ"], nu=1 / 4000, eta=1 / 4000, dt=0.01,
                    integrator=case["integ"])


def _pinned(a):
    return torch.from_numpy(a).pin_memory().numpy()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "mirror":
        p = _ql_params(case)
        model = (MHD_FullQlin if case["model"] else MHD_BQlin)(p)
        integ = (RK3CN if case["integ"] else RK3CN_Elin)(0.0, p, model)
        lin, mf, _ = _ql_state(p, seed)
        return dict(kind=kind, n=case["steps"], integ=integ, sol=solution(model), lin=lin, mf=mf)
    if kind in ("single", "forced"):
        p = _ql_params(case)
        s = QLSolver(p)
        if kind == "forced":
            s.set_cfl(CFL, DT_MAX)
            if case["f_noise"]:
                s.set_noise(case["f_noise"], *K_BAND, seed=7)
        ins = [torch.from_numpy(a).cuda() for a in _ql_state(p, seed)]
        outs = [torch.empty_like(a) for a in ins]
        torch.cuda.synchronize()
        return dict(kind="single", n=case["steps"], every=case["every"], s=s, ins=ins, outs=outs)
    if kind == "ensemble":
        cases, states = _ensemble(case, seed)
        b = QLBatch(cases)
        ins = [tuple(_pinned(a) for a in st) for st in states]
        # one pinned buffer per field over all cases, each case's part a view of it
        flat = [_pinned(np.empty(sum(st[k].size for st in states), dtype=states[0][k].dtype)) for k in range(3)]
        outs = []
        at = [0, 0, 0]
        for st in states:
            outs.append(tuple(flat[k][at[k]:at[k] + st[k].size].reshape(st[k].shape) for k in range(3)))
            at = [a + x.size for a, x in zip(at, st)]
        return dict(kind=kind, n=case["steps"], every=case["every"], b=b, ins=ins, outs=outs, flat=flat)
    if kind == "adjoint":
        p = _adjoint_params(case)
        states = [initial_state(p, seed * 1000 + i, sigma=1e-2, B0=0.05) for i in range(case["seeds"])]
        return dict(kind=kind, n=case["steps"], ckpt=case["ckpt"], solvers=[QLSolver(p) for _ in states],
                    lins=[s[0] for s in states], mfs=[s[1] for s in states], kxs=[s[2] for s in states])
    p = _dns_params(case)
    lin, kx0 = dns_initial_state(p, seed, sigma=1e-2, B0=0.05)
    return dict(kind=kind, n=case["steps"], every=case["every"], d=QLDns(p), lin=lin, kx0=kx0)


def run(st):
    kind = st["kind"]
    if kind == "mirror":
        sol, integ, t = st["sol"], st["integ"], 0.0
        sol.lin[...] = st["lin"]
        sol.mf[...] = st["mf"]
        for _ in range(st["n"]):
            t += integ.Step(t, sol)
        return [sol.lin, sol.mf]
    if kind == "single":
        s, (lin, mf, kx0), (lo, mo, ko) = st["s"], st["ins"], st["outs"]
        s.set_state_device(0.0, lin.data_ptr(), mf.data_ptr(), kx0.data_ptr())
        rec = s.step(st["n"], diag_every=st["every"])
        t = s.get_state_device(lo.data_ptr(), mo.data_ptr(), ko.data_ptr())
        return [lo, mo, ko, rec, t]
    if kind == "ensemble":
        b = st["b"]
        b.set_states(0.0, st["ins"])
        recs = b.step(st["n"], diag_every=st["every"])
        b.get_states(st["outs"])
        return st["flat"] + [np.stack(recs)]
    if kind == "adjoint":
        if len(st["solvers"]) == 1:
            J, gl, gm = st["solvers"][0].adjoint_maxwell(0.0, st["lins"][0], st["mfs"][0], st["kxs"][0], st["n"],
                                                         st["ckpt"])
        else:
            J, gl, gm = QLSolver.adjoint_maxwell_batch(st["solvers"], 0.0, st["lins"], st["mfs"], st["kxs"], st["n"],
                                                       st["ckpt"])
        return [J, gl, gm]
    d = st["d"]
    d.set_state(0.0, st["lin"], st["kx0"])
    rec = d.step(st["n"], diag_every=st["every"])
    t, lin, kx0 = d.get_state()
    return [lin, kx0, rec, t]


# ---------------------------------------------------------------------------
# work of one pass
# ---------------------------------------------------------------------------
def _ql_work(p, transforms):
    """Bytes and flops of one step: state and right-hand sides as ten passes over the four fields
    (two-register storage), `transforms` length-NZ complex transforms per mode and stage."""
    return 10.0 * 4 * p.nz * 16 * p.nxy, p.nxy * 3.0 * transforms * 5 * p.NZ * math.log2(p.NZ)


def work(case):
    kind, n = case["kind"], case["steps"]
    if kind == "dns":
        p = _dns_params(case)
        cols, kyn = p.nxy, p.ny // 2
        # 6 inverse and 9 forward fields per stage: z per column, x per (ky, z) row, y per real line
        per = cols * 5 * p.NZ * math.log2(p.NZ) + kyn * p.NZ * 5 * p.Mx * math.log2(p.Mx) \
            + p.Mx * p.NZ * 2.5 * p.My * math.log2(p.My)
        return {"bytes": n * 10.0 * 6 * p.nz * 16 * cols, "flops": n * 3.0 * 15 * per}
    if kind == "ensemble":
        ws = [_ql_work(p, 16 if case["model"] else 14) for p in _ensemble_params(case)]
        return {"bytes": n * sum(w[0] for w in ws), "flops": n * sum(w[1] for w in ws)}
    if kind == "adjoint":
        # forward run and the reverse sweep (23 transforms per mode and stage), state read and written
        b, f = _ql_work(_adjoint_params(case), 14 + 23)
        return {"bytes": 2.0 * b * n * case["seeds"], "flops": f * n * case["seeds"]}
    b, f = _ql_work(_ql_params(case), 16 if case["model"] else 14)
    return {"bytes": n * b, "flops": n * f}


def _ensemble_params(case):
    rng = np.random.default_rng(case["draw_seed"])
    ps = []
    for _ in range(case["ncases"]):
        n, NZ = int(rng.choice((16, 32, 48, 64))), int(rng.choice((32, 64, 128)))
        rng.uniform(), rng.choice((1, 2, 4)), rng.uniform()
        ps.append(QLParams(model=case["model"], nx=n, ny=n, NZ=NZ))
    return ps


# ---------------------------------------------------------------------------
# the same in plain torch, complex128
# ---------------------------------------------------------------------------
DEV = "cuda" if torch.cuda.is_available() else "cpu"
A_RK, B_RK = (8 / 15, 5 / 12, 3 / 4), (0.0, -17 / 60, -5 / 12)
P_RK = (0.0, 8 / 15, 2 / 3, 1.0)


def _f64(a):
    return torch.as_tensor(a, dtype=torch.float64, device=DEV)


class _QL:
    """One quasi-linear case (leading axes of the state may be a batch of seeds)."""

    def __init__(self, p):
        self.p = p
        ix = np.concatenate([np.arange(p.nx // 2), np.arange(1 - p.nx // 2, 0)])
        nyh, h = p.ny // 2, p.NZ // 3
        self.kxi, self.kyi = np.repeat(ix, nyh), np.tile(np.arange(nyh), ix.size)
        kzi = np.concatenate([np.arange(h + 1), np.arange(-h, 0)])
        self.kx_start = self.kxi * (2 * math.pi / p.L[0])
        self.ky_host = self.kyi * (2 * math.pi / p.L[1])
        self.idx = torch.as_tensor(kzi % p.NZ, device=DEV)
        self.ky = _f64(self.ky_host)[:, None]
        self.kz = _f64(kzi * (2 * math.pi / p.L[2]))
        self.kz2 = -self.kz * self.kz
        z0 = torch.as_tensor((self.kyi == 0)[:, None] & (np.arange(p.nz) == 0)[None, :], device=DEV)
        self.lap2 = torch.where(z0, 0.0, -self.ky * self.ky + self.kz2)
        self.il2 = torch.where(z0, 1.0, 1.0 / torch.where(z0, 1.0, self.lap2))
        self.mean0 = z0 & torch.as_tensor(self.kxi == 0, device=DEV)[:, None]
        self.mult = torch.where(self.ky == 0, 1.0, 2.0)
        self.rs = 1.0 / (p.ny // 2 * 2 * p.nx) ** 2
        self.om = 2.0 / 3.0 * p.q if p.model == 0 else p.omega

    def inv(self, a):  # a / NZ to the z grid
        full = torch.zeros(a.shape[:-1] + (self.p.NZ,), dtype=torch.complex128, device=DEV)
        return torch.fft.ifft(full.index_copy(-1, self.idx, a), dim=-1)

    def fwd(self, a):
        return torch.fft.fft(a, dim=-1).index_select(-1, self.idx)

    def kxt(self, kx0, t):  # rounded as the remap decision wants it
        return _f64(kx0 + (self.p.q * t) * self.ky_host)[:, None]

    def profiles(self, mf):
        """Real mean-field profiles and their z derivatives."""
        ik = 1j * self.kz
        if self.p.model == 0:
            return [self.inv(v).real[..., None, :] for v in (mf[..., 1, :], ik * mf[..., 1, :], self.kz2 * mf[..., 1, :])]
        return [self.inv(v).real for m in range(4) for v in (mf[m], ik * mf[m])]

    def rhs(self, t, lin, mf, kx0):
        p, ky, kz, il2, q, om = self.p, self.ky, self.kz, self.il2, self.p.q, self.om
        kx = self.kxt(kx0, t)
        Kx, Ky, Kz = 1j * kx, 1j * ky, 1j * kz
        ilapF = 1.0 / torch.where(self.mean0, 1.0, -kx * kx + self.lap2)
        u, ze, b, et = (lin[..., v, :] for v in range(4))
        uy, uz = (kx * ky * u + Kz * ze) * il2, (kx * kz * u - Ky * ze) * il2
        by, bz = (kx * ky * b + Kz * et) * il2, (kx * kz * b - Ky * et) * il2
        re = lambda x, y: x.real * y.real + x.imag * y.imag  # noqa: E731
        prof = self.profiles(mf)
        ms = lambda s: (self.mult * s).sum(-2).to(torch.complex128)  # noqa: E731
        if p.model == 0:
            By, dBy, ddBy = prof
            Ru, Rz, Rb, Re = self.inv(u), self.inv(ze), self.inv(b), self.inv(et)
            Ruz, Rbz, Rdz, Ruy, Rby = self.inv(uz), self.inv(bz), self.inv(Kz * uz), self.inv(uy), self.inv(by)
            F0 = self.fwd(Ky * Rb * By) + (2 * kx * ky * q * u + 2 * om * Kz * ze
                                           + self.fwd(2 * kx * ky * Rbz * dBy)) * ilapF
            F1 = self.fwd(Ky * Re * By - Kx * Rb * dBy + Rbz * ddBy) + (q - 2 * om) * Kz * u
            F2 = self.fwd(Ky * Ru * By)
            F3 = self.fwd(Ky * Rz * By - (2 * Rdz + Kx * Ru) * dBy - Ruz * ddBy) - q * Kz * b
            ex, ey = ms(re(Rbz, Ru) - re(Ruz, Rb)), ms(re(Rbz, Ruy) - re(Ruz, Rby))
            G0 = Kz * self.fwd(ex) * self.rs
            G1 = -q * mf[..., 0, :] + Kz * self.fwd(ey) * self.rs
            return torch.stack([F0, F1, F2, F3], dim=-2), torch.stack([G0, G1], dim=-2)
        MBx, dMBx, MBy, dMBy, MUx, dMUx, MUy, dMUy = prof
        Ux, Uy, Uz, Bx, By, Bz = (self.inv(v) for v in (u, uy, uz, b, by, bz))
        au, ab = Kx * MUx + Ky * MUy, Kx * MBx + Ky * MBy
        T1 = self.fwd(au * Ux + Uz * dMUx - ab * Bx - Bz * dMBx)
        T2 = self.fwd(au * Uy + Uz * dMUy - ab * By - Bz * dMBy)
        T3 = self.fwd(au * Uz - ab * Bz)
        S1 = self.fwd(au * Bx + Uz * dMBx - ab * Ux - Bz * dMUx)
        S2 = self.fwd(au * By + Uz * dMBy - ab * Uy - Bz * dMUy)
        S3 = self.fwd(au * Bz - ab * Uz)
        B0 = p.B0z
        F0 = (2 * kx * ky * q * u + 2 * om * Kz * ze - kx * kx * T1 - kx * ky * T2 - kx * kz * T3) * ilapF \
            + B0 * Kz * b - T1
        F1 = (q - 2 * om) * Kz * u + B0 * Kz * et - (Kz * T2 - Ky * T3)
        F2 = B0 * Kz * u - S1
        F3 = -q * Kz * b + B0 * Kz * ze - (Kz * S2 - Ky * S3)
        dUx, dBx, dUy, dBy = self.inv(Kz * u), self.inv(Kz * b), self.inv(Kz * uy), self.inv(Kz * by)
        sx, sy = ms(re(Bz, Ux) - re(Uz, Bx)), ms(re(Bz, Uy) - re(Uz, By))
        sux = ms(-(re(Ux, Kx * Ux) + re(Uy, Ky * Ux) + re(Uz, dUx)) + re(Bx, Kx * Bx) + re(By, Ky * Bx) + re(Bz, dBx))
        suy = ms(-(re(Ux, Kx * Uy) + re(Uy, Ky * Uy) + re(Uz, dUy)) + re(Bx, Kx * By) + re(By, Ky * By) + re(Bz, dBy))
        D = [Kz * self.fwd(sx) * self.rs, Kz * self.fwd(sy) * self.rs, self.fwd(sux) * self.rs, self.fwd(suy) * self.rs]
        G = torch.stack([B0 * Kz * mf[2] + D[0], -q * mf[0] + B0 * Kz * mf[3] + D[1],
                         2 * om * mf[3] + B0 * Kz * mf[0] + D[2], (q - 2 * om) * mf[2] + B0 * Kz * mf[1] + D[3]])
        return torch.stack([F0, F1, F2, F3], dim=-2), G

    def op(self, lap):
        """Dissipation of the four fields from the Laplacian."""
        p = self.p
        if p.model:
            lap = -torch.abs(lap) ** (p.viscosity_order // 2)
        return torch.stack([p.nu * lap, p.nu * lap, p.eta * lap, p.eta * lap], dim=-2)

    def step(self, t, dt, lin, mf, kx0, old=None, watch=None):
        """One step, remap included: (t, lin, mf, kx0, old operator)."""
        p, ky = self.p, self.ky
        Lm = torch.stack([c * self.kz2 for c in (p.eta, p.eta, p.nu, p.nu)[: p.nmf]])
        kx = self.kxt(kx0, t)
        old = self.op(-kx * kx + self.lap2) if old is None else old
        Fp = Gp = None
        for s in range(3):
            ts, dl = t + dt * P_RK[s], dt * (P_RK[s + 1] - P_RK[s])
            if s == 2 and watch is not None:
                watch(mf)
            F, G = self.rhs(ts, lin, mf, kx0)
            kxe = self.kxt(kx0, ts) + p.q * dl * ky
            L = self.op(-kxe * kxe - ky * ky + self.kz2)
            a, b = A_RK[s] * dt, B_RK[s] * dt
            acc, accm = a * F, a * G
            if s:
                acc, accm = acc + b * Fp, accm + b * Gp
            if p.integrator == 0:
                lin, mf = torch.exp((a + b) * L) * (acc + lin), torch.exp((a + b) * Lm) * (accm + mf)
            else:
                c = (a + b) / 2
                lin = (acc + (1 + c * old) * lin) / (1 - c * L)
                mf = (accm + (1 + c * Lm) * mf) / (1 - c * Lm)
                old = L
            Fp, Gp = F, G
        t = t + dt
        return t, lin, mf, kx0, old

    def remap(self, t, lin, kx0):
        p = self.p
        dk = 2 * math.pi / p.L[0]
        gone = kx0 + (p.q * t) * self.ky_host > (p.nx - 1) / 2.0 * dk
        if gone.any():
            lin = torch.where(torch.as_tensor(gone, device=DEV)[:, None, None], 0.0, lin)
            kx0 = np.where(gone, kx0 - (p.nx - 1) * dk, kx0)
        return lin, kx0

    def record(self, t, lin, mf, kx0):
        p, il2 = self.p, self.il2
        kx = self.kxt(kx0, t)
        lapF = -kx * kx + self.lap2
        u, ze, b, et = (lin[..., v, :] for v in range(4))
        n2 = lambda x: x.real ** 2 + x.imag ** 2  # noqa: E731
        div = p.L[2] / float(p.nx * (p.ny // 2 * 2) * p.NZ) ** 2
        out = []
        for f, g in ((u, ze), (b, et)):
            e = lapF * il2 * n2(f) - il2 * n2(g)
            y = (kx * self.ky * f + 1j * self.kz * g) * il2
            out.append([div * (self.mult * w).sum((-2, -1)) for w in (e, (f * y.conj()).real, -lapF * e)])
        (eu, au, du), (eb, ab, db) = out
        dm = p.L[2] / p.NZ ** 2
        ms = []
        for x, y, c in ((0, 1, p.eta), (2, 3, p.nu))[: p.nmf // 2]:
            x, y = mf[..., x, :], mf[..., y, :]
            e = n2(x) + n2(y)
            ms.append((dm * e.sum(-1), dm * (x * y.conj()).real.sum(-1), -c * dm * (self.kz2 * e).sum(-1)))
        eMB, aMB, dMB = ms[0]
        eMU, aMU, dMU = ms[1] if p.nmf == 4 else (0 * eMB, 0 * eMB, 0 * eMB)
        du, db = p.nu * du, p.eta * db
        kzm = 2 * math.pi / p.L[2] * (p.NZ // 3)
        return torch.stack([t + 0 * eu, eMU / 2, eMB / 2, eu / 2, eb / 2, aMU, aMB, au, ab, dMU, dMB, du, db,
                            (p.nu ** 3 / (dMU + du)) ** 0.25 * kzm, (p.eta ** 3 / (dMB + db)) ** 0.25 * kzm])

    # ---- driving noise: Philox4x32-10 per (step, mode, kz, field), Box-Muller ----
    def noise(self, t, dt, step, kx0, f_noise, klo, khi, seed):
        p, nxy, nz = self.p, self.p.nxy, self.p.nz
        src = np.arange(nxy)[:, None, None] + np.zeros((1, 4, nz), dtype=np.int64)
        kk = np.arange(nz)[None, None, :] + np.zeros((nxy, 4, 1), dtype=np.int64)
        fld = np.arange(4)[None, :, None] + 0 * src
        sign = np.ones(src.shape)
        on = np.broadcast_to((self.kyi > 0)[:, None, None], src.shape).copy()
        kxs = np.broadcast_to(kx0[:, None, None], src.shape).copy()
        if p.model:  # ky = 0 columns in conjugate pairs, kx < 0 drawn
            k0 = np.broadcast_to((self.kyi == 0)[:, None, None], src.shape)
            pos = k0 & (self.kxi > 0)[:, None, None]
            on |= k0 & (self.kxi != 0)[:, None, None] & (kk > 0)
            src = np.where(pos, ((2 * (p.nx // 2) - self.kxi - 1) * (p.ny // 2))[:, None, None], src)
            kxs, sign = np.where(pos, -kxs, kxs), np.where(pos, -1.0, 1.0)
            kk = np.where(pos & (kk > 0), nz - kk, kk)
        c = kk % nz * 0.0 + np.where(kk <= (nz - 1) // 2, kk, kk - nz) * (2 * math.pi / p.L[2])
        ky = self.ky_host[:, None, None]
        lap2 = -ky * ky + -(c * c)
        kx = kxs + (p.q * t) * ky
        lapF = -kx * kx + lap2
        on &= (lapF > -khi * khi) & (lapF < -klo * klo)
        mf = dt * float(p.nx * (p.ny // 2 * 2) * p.NZ) ** 2 / float(16 * 32 * 32) ** 2
        amp = np.sqrt(np.where(on, np.where(fld % 2 == 0, mf * lap2 / np.where(on, lapF, 1.0), -mf * lap2), 0.0))
        m32 = np.uint64(0xFFFFFFFF)
        w = [src.astype(np.uint64), (4 * kk + fld).astype(np.uint64), np.full(src.shape, step & 0xFFFFFFFF, np.uint64),
             np.full(src.shape, step >> 32, np.uint64)]
        k = [seed & 0xFFFFFFFF, seed >> 32]
        for _ in range(10):
            a, b = w[0] * np.uint64(0xD2511F53), w[2] * np.uint64(0xCD9E8D57)
            w = [(b >> np.uint64(32)) ^ w[1] ^ np.uint64(k[0]), b & m32, (a >> np.uint64(32)) ^ w[3] ^ np.uint64(k[1]),
                 a & m32]
            k = [(k[0] + 0x9E3779B9) & 0xFFFFFFFF, (k[1] + 0xBB67AE85) & 0xFFFFFFFF]
        u1 = ((((w[0] << np.uint64(32)) | w[1]) >> np.uint64(11)).astype(np.float64) + 0.5) / 2.0 ** 53
        u2 = (((w[2] << np.uint64(32)) | w[3]) >> np.uint64(11)).astype(np.float64) / 2.0 ** 53
        r, ang, sd = np.sqrt(-2 * np.log(u1)), 2 * math.pi * u2, f_noise / math.sqrt(2.0)
        return torch.as_tensor(amp * sd * r * (np.cos(ang) + 1j * sign * np.sin(ang)), device=DEV)

    def run(self, lin, mf, n, every, cfl=None, f_noise=0.0):
        p, t, kx0, old, recs = self.p, 0.0, self.kx_start.copy(), None, []
        lin, mf = (torch.as_tensor(a, device=DEV) for a in (lin, mf))
        seen = [None]
        kmax = max(2 * math.pi / l * (m / d) for l, m, d in zip(p.L, (p.nx, p.ny // 2 * 2, p.NZ), (2.0, 2.0, 3.0)))
        peak = lambda v: float(torch.abs(self.inv(v)).max())  # noqa: E731
        for i in range(n):
            dt = p.dt
            if cfl:
                if p.model == 0:
                    c = kmax * (0.0 if seen[0] is None else peak(seen[0][1])) + kmax * peak(mf[0]) + p.q
                else:
                    c = (0.0 if seen[0] is None else kmax * sum(peak(v) for v in seen[0])) + p.q
                dt = min(cfl[0] / c, cfl[1])
            t0 = t
            t, lin, mf, kx0, old = self.step(t, dt, lin, mf, kx0, old, lambda m: seen.__setitem__(0, m))
            if f_noise:
                lin = lin + self.noise(t0, dt, i, kx0, f_noise, *K_BAND, 7)
            if p.remap:
                lin, kx0 = self.remap(t, lin, kx0)
            if every and (i + 1) % every == 0:
                recs.append(self.record(t, lin, mf, kx0))
        return t, lin, mf, kx0, torch.stack(recs) if recs else torch.zeros((0, 15), dtype=torch.float64)


def _exact_adjoint(case, seed):
    p = _adjoint_params(case)
    st = [initial_state(p, seed * 1000 + i, sigma=1e-2, B0=0.05) for i in range(case["seeds"])]
    m, n = _QL(p), case["steps"]
    lin0, mf0 = (torch.as_tensor(np.stack([s[k] for s in st]), device=DEV) for k in (0, 1))
    # forward, one state kept per step; then each step again with its graph, last first
    kept, t, lin, mf, kx0, old = [], 0.0, lin0, mf0, m.kx_start.copy(), None
    with torch.no_grad():
        for _ in range(n):
            kept.append((t, lin, mf, kx0, old))
            t, lin, mf, kx0, old = m.step(t, p.dt, lin, mf, kx0, old)
            lin, kx0 = m.remap(t, lin, kx0)
    J = torch.zeros(len(st), dtype=torch.float64, device=DEV)
    gl, gm = torch.zeros_like(lin0), torch.zeros_like(mf0)
    for t, lin, mf, kx0, old in reversed(kept):
        lin, mf = lin.detach().requires_grad_(True), mf.detach().requires_grad_(True)
        t1, l1, m1, k1, _ = m.step(t, p.dt, lin, mf, kx0, old)
        l1, k1 = m.remap(t1, l1, k1)
        am = m.record(t1, l1, m1, k1)[8] / n
        J += am.detach()
        gl, gm = torch.autograd.grad((am.sum(), l1, m1), (lin, mf), (torch.ones((), dtype=torch.float64, device=DEV),
                                                                   gl, gm))
    if len(st) == 1:
        return [float(J[0]), gl[0].resolve_conj(), gm[0].resolve_conj()]
    return [J, gl.resolve_conj(), gm.resolve_conj()]


def _exact_dns(case, seed):
    p = _dns_params(case)
    q = _QL(p.ql())
    lin, kx0 = dns_initial_state(p, seed, sigma=1e-2, B0=0.05)
    lin = torch.as_tensor(lin, device=DEV)
    kz, dk = q.kz, 2 * math.pi / p.L[0]
    ky = q.ky + 0 * kz
    yb, zb = torch.as_tensor(q.kyi, device=DEV)[:, None], q.idx[None, :]
    kp2 = ky * ky + kz * kz
    ikp = torch.where(kp2 > 0, 1.0 / torch.where(kp2 > 0, kp2, 1.0), 0.0)

    def wave(t):
        return q.kxt(kx0, t) + 0 * kz

    def keep(t):
        return torch.as_tensor(np.abs(kx0 + (p.q * t) * q.ky_host) <= p.Mx / 3.0 * dk, device=DEV)[:, None, None]

    def rhs(t, lin):
        xb = torch.as_tensor(np.rint(kx0 / dk).astype(np.int64) % p.Mx, device=DEV)[:, None]
        S = torch.zeros((6, p.Mx, p.My // 2 + 1, p.NZ), dtype=torch.complex128, device=DEV)
        S[:, xb, yb, zb] = lin.transpose(0, 1)
        ux, uy, uz, bx, by, bz = torch.fft.irfft(torch.fft.ifft(torch.fft.ifft(S, dim=1), dim=3), n=p.My, dim=2)
        pr = torch.stack([ux * ux - bx * bx, uy * uy - by * by, uz * uz - bz * bz, ux * uy - bx * by,
                          ux * uz - bx * bz, uy * uz - by * bz, uy * bz - uz * by, uz * bx - ux * bz,
                          ux * by - uy * bx])
        S = torch.fft.fft(torch.fft.fft(torch.fft.rfft(pr, dim=2), dim=1), dim=3)
        xx, yy, zz, xy, xz, yz, ex, ey, ez = S[:, xb, yb, zb]
        Kx, om, B0 = wave(t), p.omega, p.B0z
        ux, uy, uz, bx, by, bz = (lin[:, c] for c in range(6))
        Ax = -1j * (Kx * xx + ky * xy + kz * xz) + 2 * om * uy + 1j * kz * B0 * bx
        Ay = -1j * (Kx * xy + ky * yy + kz * yz) + (p.q - 2 * om) * ux + 1j * kz * B0 * by
        Az = -1j * (Kx * xz + ky * yz + kz * zz) + 1j * kz * B0 * bz
        K2 = Kx * Kx + kp2
        s = (Kx * Ax + ky * Ay + kz * Az + p.q * ky * ux) * torch.where(K2 > 0, 1.0 / torch.where(K2 > 0, K2, 1.0), 0.0)
        F = torch.stack([Ax - Kx * s, Ay - ky * s, Az - kz * s, 1j * (ky * ez - kz * ey) + 1j * kz * B0 * ux,
                         1j * (kz * ex - Kx * ez) - p.q * bx + 1j * kz * B0 * uy,
                         1j * (Kx * ey - ky * ex) + 1j * kz * B0 * uz], dim=1)
        return torch.where(keep(t), F, 0.0)

    def op(t, dl):
        kx = q.kxt(kx0, t) + p.q * dl * q.ky
        lap = -torch.abs(-kx * kx - q.ky * q.ky + q.kz2) ** (p.viscosity_order // 2)
        lap[0] = q.kz2
        return torch.stack([p.nu * lap] * 3 + [p.eta * lap] * 3, dim=1)

    def constrain(t, lin):
        lin = torch.where(keep(t), lin, 0.0)
        Kx = wave(t)
        zonal, zero = (kp2 == 0) & (Kx != 0), (kp2 == 0) & (Kx == 0)
        out = []
        for b in (0, 3):
            x, y, z = lin[:, b], lin[:, b + 1], lin[:, b + 2]
            D = Kx * x + ky * y + kz * z
            out += [torch.where(zonal, 0.0, x), y - ky * D * ikp, torch.where(zero, 0.0, z - kz * D * ikp)]
        return torch.stack(out, dim=1)

    def record(t, lin):
        div, w = p.L[2] / float(p.Mx * p.My * p.NZ) ** 2, q.mult.clone()
        n2 = lin.real ** 2 + lin.imag ** 2
        K2 = wave(t) ** 2 + kp2
        w[0] = 0.0
        eu, eb = n2[:, :3].sum(1), n2[:, 3:].sum(1)
        xy = lambda a, b: (a * b.conj()).real  # noqa: E731
        Eu, Eb, Du, Db = ((w * v).sum() * div for v in (eu, eb, p.nu * K2 * eu, p.eta * K2 * eb))
        Au, Ab = ((w * xy(lin[:, b], lin[:, b + 1])).sum() * div for b in (0, 3))
        m, k2 = lin[0], -q.kz2
        eMU, eMB = ((n2[0, b] + n2[0, b + 1]) for b in (0, 3))
        aMU, aMB = (xy(m[b], m[b + 1]).sum() * div for b in (0, 3))
        dMU, dMB = p.nu * (k2 * eMU).sum() * div, p.eta * (k2 * eMB).sum() * div
        eMU, eMB = eMU.sum() * div, eMB.sum() * div
        kzm = 2 * math.pi / p.L[2] * (p.NZ // 3)
        return torch.stack([t + 0 * Eu, eMU / 2, eMB / 2, Eu / 2, Eb / 2, aMU, aMB, Au, Ab, dMU, dMB, Du, Db,
                            (p.nu ** 3 / (dMU + Du)) ** 0.25 * kzm, (p.eta ** 3 / (dMB + Db)) ** 0.25 * kzm])

    t, recs, dt, old = 0.0, [], p.dt, op(0.0, 0.0)
    for i in range(case["steps"]):
        Fp = None
        for s in range(3):
            ts = t + dt * P_RK[s]
            a, b = A_RK[s] * dt, B_RK[s] * dt
            F, L = rhs(ts, lin), op(ts, dt * (P_RK[s + 1] - P_RK[s]))
            acc = a * F + (b * Fp if s else 0.0)
            if p.integrator == 0:
                lin = torch.exp((a + b) * L) * (acc + lin)
            else:
                lin = (acc + (1 + (a + b) / 2 * old) * lin) / (1 - (a + b) / 2 * L)
                old = L
            lin, Fp = constrain(t + dt * P_RK[s + 1], lin), F
        t = t + dt
        if p.remap:
            lin, kx0 = q.remap(t, lin, kx0)
        if (i + 1) % case["every"] == 0:
            recs.append(record(t, lin))
    return [lin, kx0, torch.stack(recs) if recs else torch.zeros((0, 15), dtype=torch.float64), t]


def exact(case, seed):
    kind, n = case["kind"], case["steps"]
    with torch.no_grad():
        if kind == "dns":
            return _exact_dns(case, seed)
        if kind in ("mirror", "single", "forced"):
            p = _ql_params(case)
            lin, mf, _ = _ql_state(p, seed)
            cfl = (CFL, DT_MAX) if kind == "forced" else None
            t, lin, mf, kx0, rec = _QL(p).run(lin, mf, n, case["every"], cfl, case.get("f_noise", 0.0))
            return [lin, mf] if kind == "mirror" else [lin, mf, kx0, rec, t]
        if kind == "ensemble":
            cases, states = _ensemble(case, seed)
            outs = [_QL(p).run(lin, mf, n, case["every"]) for p, (lin, mf, _) in zip(cases, states)]
            return [torch.cat([o[k].reshape(-1) for o in outs]) for k in (1, 2)] + \
                [np.concatenate([o[3] for o in outs]), torch.stack([o[4] for o in outs])]
    return _exact_adjoint(case, seed)
