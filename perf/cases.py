"""Performance cases: the calls that a program using this framework makes, over the
sizes and options it is used with.

Steps (set_state, step, state: a program that owns the positions and advances them):
  dumbbells   one trapped colloid and a few dumbbells: the smallest system, all latency
  probe       two probes in a solution of short chains (shell path, block-Cholesky noise)
  replica     one polymer system with 0 to 2 probes, full hydrodynamics
  brush       one colloid with grafted FENE chains
  suspension  equal colloids at volume fraction 0.2, lubricated near contacts
  ensemble    a batch of ragged replicas advanced together
Single operations:
  mobility    one product with the grand mobility (the operator callback of a host solver)
  matmult     one product with the saddle matrix of a colloid suspension
  sqrt        Brownian displacements M^(1/2) z by Lanczos
  ksp         the saddle system by Jacobi MINRES (the KSPSolve stand-in)

The mixed form computes the monomer far field in FP32, so its results are FP32
numbers in FP64 storage: a program that runs it keeps what it records (frames,
velocities, products) as float32, as trajectory formats do, and the mixed cases
return that.  FP64 contexts return FP64.
"""
import math

import numpy as np
import torch

from polystokes_brownian_b200 import _capi, configs
from polystokes_brownian_b200.engine import Batch

STEPS = ("dumbbells", "probe", "replica", "brush", "suspension", "ensemble")


def _case(kind, name=None, *, n=0, reps=1, nper=0, mixed=False, lub=False, thermal=True, minres=False, refine=0):
    c = dict(kind=kind, n=n, reps=reps, nper=nper, mixed=mixed, lub=lub, thermal=thermal, minres=minres, refine=refine)
    return c if name is None else dict(c, name=name)


def listed():
    return [
        # the reference's thermal test: one colloid, four dumbbells; every launch is latency
        _case("dumbbells", "step_dumbbells", n=4),
        # polymer solution with two probes, 222 beads, shell path; the structured solve and
        # Jacobi MINRES (the step's default, the reference's own solver)
        _case("probe", "step_probe", n=220),
        _case("probe", "step_probe_minres", n=220, minres=True),
        # one replica of an ensemble on its own, odd size, lubricated: a serving loop with one request
        _case("replica", "step_replica_lub", n=985, mixed=True, lub=True),
        # 128 grafted chains of 32 beads, with the refinement sweep that keeps it within 1e-6
        _case("brush", "step_brush", n=128, nper=32, mixed=True, refine=1),
        # 1024 lubricated colloids
        _case("suspension", "step_suspension_lub", n=1024, lub=True),
        # the batched ensemble, 64 replicas of 64 to 4096 beads, lubricated, mixed precision
        _case("ensemble", "step_ensemble_lub", n=4096, reps=64, mixed=True, lub=True),
        # a smaller ensemble in FP64 without lubrication
        _case("ensemble", "step_ensemble_fp64", n=2048, reps=24),
        # one far-field product at the largest system served
        _case("mobility", "mobility_16k", n=16384, mixed=True),
        # one FP64 saddle product of a suspension
        _case("matmult", "matmult_suspension", n=512),
        # Brownian displacements of one odd-sized system in FP64
        _case("sqrt", "sqrt_1k", n=1023),
        # the saddle system of a medium system by MINRES to near machine accuracy
        _case("ksp", "ksp_minres", n=500, minres=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(STEPS + ("ensemble", "replica", "mobility", "matmult", "sqrt", "ksp"))
    if kind == "dumbbells":
        return _case(kind, n=rng.randint(1, 24), thermal=rng.random() < 0.8)
    if kind == "probe":
        return _case(kind, n=220, minres=rng.random() < 0.5, thermal=rng.random() < 0.7,
                     reps=rng.randint(1, 8))
    if kind == "replica":
        mixed = rng.random() < 0.6
        return _case(kind, n=_log(rng, 64, 4096), mixed=mixed, lub=rng.random() < 0.6, thermal=rng.random() < 0.8)
    if kind == "brush":
        mixed = rng.random() < 0.6
        return _case(kind, n=_log(rng, 8, 128), nper=rng.randint(5, 32), mixed=mixed, refine=int(mixed))
    if kind == "suspension":
        return _case(kind, n=_log(rng, 13, 900), lub=rng.random() < 0.7)
    if kind == "ensemble":
        return _case(kind, n=_log(rng, 128, 2048), reps=rng.randint(2, 48), mixed=rng.random() < 0.6,
                     lub=rng.random() < 0.6, thermal=rng.random() < 0.8)
    if kind == "mobility":
        return _case(kind, n=_log(rng, 64, 16000), mixed=rng.random() < 0.6)
    if kind == "matmult":
        return _case(kind, n=_log(rng, 13, 700))
    if kind == "sqrt":
        return _case(kind, n=_log(rng, 64, 1200), mixed=rng.random() < 0.4)
    return _case(kind, n=_log(rng, 64, 1000), minres=True)


def _sizes(case):
    """Bead counts of an ensemble: spread evenly over the logarithm of [64, n], whatever the seed."""
    if case["kind"] != "ensemble":
        return [case["n"]]
    R, hi = case["reps"], case["n"]
    return [int(round(64 * (hi / 64) ** ((i + 0.5) / R))) for i in range(R)]


class _Sized:
    """The generator of one replica: its whole numbers (probes, chain length) by its place in
    the batch, so that all seeds have the same sizes, and all else from the seed."""

    def __init__(self, seed, i):
        self.integers = np.random.default_rng(i).integers
        g = np.random.default_rng([seed, i])
        self.uniform, self.normal = g.uniform, g.normal


def _chains(seed, n):
    """A solution of chains without probes: the monomers of an ensemble replica."""
    s = configs.ensemble_member(_Sized(seed, n), n)
    Nm = s.params["Nm"]
    return configs.System(s.name, dict(s.params, Nc=0, ktrap=0.0), s.x[:Nm])


def _systems(case, seed):
    k, n = case["kind"], case["n"]
    if k == "dumbbells":
        out = [configs.dumbbells(seed=seed, n_db=n)]
    elif k == "probe":
        out = [configs.polymer_probe(seed=seed + 1000 * i) for i in range(case["reps"])]
    elif k in ("replica", "ensemble", "mobility"):
        out = [configs.ensemble_member(_Sized(seed, i + N), N, lub=case["lub"])
               for i, N in enumerate(_sizes(case))]
    elif k == "brush":
        out = [configs.brush(nchain=n, nper=case["nper"], seed=seed)]
    elif k in ("suspension", "matmult"):
        s = configs.suspension(n=n, seed=seed)
        out = [configs.System(s.name, dict(s.params, lub_on=int(case["lub"])), s.x)]
    else:
        out = [_chains(seed, n)]
    if not case["thermal"]:
        out = [configs.System(s.name, dict(s.params, kT=0.0), s.x) for s in out]
    return out


def _normal(n, seed, i=0):
    g = torch.Generator(device="cuda").manual_seed(2 * (seed % (1 << 40)) + i)
    return torch.randn(n, dtype=torch.float64, device="cuda", generator=g)


def prepare(case, seed):
    b = Batch(_systems(case, seed), precision=_capi.PS_PREC_MIXED if case["mixed"] else _capi.PS_PREC_FP64)
    b.set_seed(seed)
    st = {"case": case, "b": b}
    if case["kind"] in STEPS:
        st["x"], st["q"] = b.state()
        return st
    b.stage()   # pair lists and the operator at these positions
    st["u"] = _normal(b.ntop if case["kind"] in ("mobility", "sqrt") else b.nvec, seed)
    return st


def run(state):
    case, b = state["case"], state["b"]
    kind = case["kind"]
    if kind in STEPS:
        b.set_state(state["x"], state["q"] if b.ncoll else None)
        b.step(rtol=1e-8, maxit=50000, refine=case["refine"],
               solver=_capi.PS_SOLVE_MINRES if case["minres"] else _capi.PS_SOLVE_STRUCTURED)
        x, q = b.state()
        if case["mixed"]:
            return {"x": x.float(), "q": q.float(), "up": b.step_outputs()["up"].float()}
        return {"x": x, "q": q}
    if kind == "mobility":
        y = b.mobility_apply(state["u"])
    elif kind == "matmult":
        y = b.matmult(state["u"])
    elif kind == "sqrt":
        y, _ = b.sqrtm(state["u"], kmax=40, tol=1e-6)
    else:
        y, _ = b.solve(state["u"], rtol=1e-12, maxit=50000)
    return y.float() if case["mixed"] else y


def work(case):
    """One pass.  A far-field product takes 40 flops per ordered pair of monomers, 120 per
    monomer and colloid, 250 per ordered pair of colloids; a step cannot do with less than one
    product in each of its five solves and one for its noise (Krylov methods take more)."""
    kind = case["kind"]
    if kind in ("suspension", "matmult"):
        mono, coll = [0], [case["n"]]
    elif kind == "brush":
        mono, coll = [case["n"] * case["nper"]], [1]
    elif kind == "probe":
        mono, coll = [220] * case["reps"], [2] * case["reps"]
    elif kind == "dumbbells":
        mono, coll = [2 * case["n"]], [1]
    else:
        mono, coll = _sizes(case), [0] * case["reps"]
    far = sum((0.0 if kind == "probe" else 40.0 * m * m) + 120.0 * m * c + 250.0 * c * c for m, c in zip(mono, coll))
    beads = sum(mono) + sum(coll)
    products = (6 if case["thermal"] else 5) if kind in STEPS else 1
    vec = 6 * sum(mono) + 17 * sum(coll) if kind in ("matmult", "ksp") else 3 * sum(mono) + 11 * sum(coll)
    if kind in STEPS:
        return {"bytes": 8.0 * (2 * 3 * beads + 2 * 4 * sum(coll)), "flops": products * far}
    return {"bytes": 8.0 * (3 * beads + 2 * vec), "flops": products * far}


# ---------------------------------------------------------------------------
# 64-bit values in plain torch: the far-field pair tensors, row block by row block.

def _aa_rows(x, b, i0, i1):
    """RPY blocks of equal spheres of radius b (units 6 pi eta = 1), rows [i0, i1): (rows, 3, n, 3)."""
    n = x.shape[0]
    d = x[i0:i1, None, :] - x[None, :, :]
    r = d.norm(dim=2)
    own = torch.arange(i0, i1, device=x.device)
    r[own - i0, own] = 1.0
    far = r > 2 * b
    fx = torch.where(far, 1.5 / r - b * b / r ** 3, (1 - 0.1875 * r / b) / b)
    fy = torch.where(far, 0.75 / r + 0.5 * b * b / r ** 3, (1 - 0.28125 * r / b) / b)
    e = d / r[..., None]
    M = (fx - fy)[..., None, None] * e[..., :, None] * e[..., None, :]
    M = M + fy[..., None, None] * torch.eye(3, dtype=x.dtype, device=x.device)
    M[own - i0, own] = torch.eye(3, dtype=x.dtype, device=x.device) / b
    return M.permute(0, 2, 1, 3).reshape(3 * (i1 - i0), 3 * n)


def _sym(S):
    """(n, 5) stresslets as symmetric traceless matrices."""
    z = torch.zeros(S.shape[0], 3, 3, dtype=S.dtype, device=S.device)
    z[:, 0, 0], z[:, 1, 1], z[:, 2, 2] = S[:, 0], S[:, 4], -S[:, 0] - S[:, 4]
    z[:, 0, 1] = z[:, 1, 0] = S[:, 1]
    z[:, 0, 2] = z[:, 2, 0] = S[:, 2]
    z[:, 1, 2] = z[:, 2, 1] = S[:, 3]
    return z


def _flat(Z):
    """The five rates of strain of symmetric matrices (..., 3, 3)."""
    return torch.stack([Z[..., 0, 0] - Z[..., 2, 2], 2 * Z[..., 0, 1], 2 * Z[..., 0, 2], 2 * Z[..., 1, 2],
                        Z[..., 1, 1] - Z[..., 2, 2]], dim=-1)


def _outer(a, b):
    return a[..., :, None] * b[..., None, :] + b[..., :, None] * a[..., None, :]


def _mobility(s, u):
    """M u of one system (physical pair scalars), u = [F_m | F_c | T_c | S_c]."""
    x = torch.tensor(s.x, dtype=torch.float64, device=u.device)
    Nm, Nc, b = s.params["Nm"], s.params["Nc"], s.params["beta"]
    xm, xc = x[:Nm], x[Nm:]
    Fm = u[:3 * Nm].view(Nm, 3)
    F, T = u[3 * Nm:3 * (Nm + Nc)].view(Nc, 3), u[3 * (Nm + Nc):3 * Nm + 6 * Nc].view(Nc, 3)
    Sv = u[3 * Nm + 6 * Nc:].view(Nc, 5)
    Um = torch.empty(3 * Nm, dtype=u.dtype, device=u.device)
    for i0 in range(0, Nm, 512):
        i1 = min(Nm, i0 + 512)
        Um[3 * i0:3 * i1] = _aa_rows(xm, b, i0, i1) @ Fm.reshape(-1)
    Um = Um.view(Nm, 3)
    if not Nc:
        return Um.reshape(-1)
    S = _sym(Sv)
    dot = lambda p, q: (p * q).sum(-1, keepdim=True)  # noqa: E731
    U, W = F.clone(), 0.75 * T
    E = 0.9 * _flat(S)
    E[:, 1:4] = 1.8 * Sv[:, 1:4]
    if Nm:
        d = xm[:, None] - xc[None]
        r = d.norm(dim=2, keepdim=True)
        e = (d / r)
        fx, fy = 1.5 / r - 0.5 * (1 + b * b) / r ** 3, 0.75 / r + 0.25 * (1 + b * b) / r ** 3
        yb, xg = -0.75 / r ** 2, 2.25 / r ** 2 - 0.45 * (3 + 5 * b * b) / r ** 4
        yg = 0.9 * (0.5 + 5 * b * b / 6) / r ** 4
        v = torch.einsum("cij,mcj->mci", S, e)
        f = Fm[:, None].expand_as(e)
        Um = Um + (fy * F + (fx - fy) * dot(e, F[None]) * e + yb * torch.cross(e, T[None].expand_as(e), dim=2)
                   + 2 * yg * v - (xg + 2 * yg) * dot(e, v) * e).sum(1)
        U = U + (fy * f + (fx - fy) * dot(e, f) * e).sum(0)
        W = W + (yb * torch.cross(f, e, dim=2)).sum(0)
        Z = yg[..., None] * _outer(e, f) - ((xg + 2 * yg) * dot(e, f))[..., None] * e[..., :, None] * e[..., None, :]
        E = E + _flat(Z).sum(0)
    if Nc > 1:
        # rows against columns; e points from the higher to the lower index of the pair
        row = torch.arange(Nc, device=u.device)
        sg = torch.where(row[:, None] < row[None], 1.0, -1.0).to(u.dtype)[..., None]
        d = sg * (xc[:, None] - xc[None])
        r = d.norm(dim=2, keepdim=True) + torch.eye(Nc, dtype=u.dtype, device=u.device)[..., None]
        on = (1 - torch.eye(Nc, dtype=u.dtype, device=u.device))[..., None]
        e = d / r
        xa, ya, yb = 1.5 / r - 1 / r ** 3, 0.75 / r + 0.5 / r ** 3, -0.75 / r ** 2
        xg, yg, yh = 2.25 / r ** 2 - 3.6 / r ** 4, 1.2 / r ** 4, -1.125 / r ** 3
        xc_, yc = 0.75 / r ** 3, -0.375 / r ** 3
        xm_, ym, zm = -4.5 / r ** 3 + 10.8 / r ** 5, 2.25 / r ** 3 - 7.2 / r ** 5, 1.8 / r ** 5
        f, t = F[None].expand_as(e), T[None].expand_as(e)
        v = torch.einsum("cij,rcj->rci", S, e)
        s_ = dot(e, v)
        te = torch.cross(t, e, dim=2)
        ev = torch.cross(e, v, dim=2)
        U = U + (on * (ya * f + (xa - ya) * dot(e, f) * e - yb * te
                       + sg * (2 * yg * v - (xg + 2 * yg) * s_ * e))).sum(1)
        W = W + (on * (yb * torch.cross(f, e, dim=2) + (xc_ + yc) * dot(e, t) * e + yc * t - 2 * yc * e * e * t
                       + 2 * yh * ev)).sum(1)
        ee = e[..., :, None] * e[..., None, :]
        Z = ((1.5 * xm_ - 2 * ym + 0.5 * zm) * s_ + sg * (xg + 2 * yg) * dot(e, f))[..., None] * ee
        Z = Z + _outer(e, yh * te + (ym - zm) * v - sg * yg * f) + zm[..., None] * S[None]
        E = E + (on * _flat(Z)).sum(1)
    return torch.cat([Um.reshape(-1), U.reshape(-1), W.reshape(-1), E.reshape(-1)])


def exact(case, seed):
    kind = case["kind"]
    if kind in STEPS:
        return None
    s = _systems(case, seed)[0]
    Nm, Nc = s.params["Nm"], s.params["Nc"]
    top, vel = 3 * Nm + 11 * Nc, 3 * Nm + 6 * Nc
    u = _normal(top if kind in ("mobility", "sqrt") else top + vel, seed)
    if kind == "mobility":
        return _mobility(s, u)
    if kind == "matmult":
        y = torch.zeros_like(u)
        y[:top] = _mobility(s, u[:top])
        y[:vel] -= u[top:]
        y[top:] = -u[:vel]
        return y
    if kind == "ksp":
        # no colloids: the constraint rows give F, the velocity rows U
        F = -u[top:]
        return torch.cat([F, _mobility(s, F) - u[:top]])
    x = torch.tensor(s.x, dtype=torch.float64, device=u.device)
    lam, Q = torch.linalg.eigh(_aa_rows(x, s.params["beta"], 0, Nm))
    return Q @ (lam.clamp(min=0).sqrt() * (Q.T @ u))
