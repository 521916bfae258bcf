"""The work that users of this library have it do, as measurable cases.

Four kinds of call, through the public Python bindings (and, where those read
a state only to the host, through the C ABI they bind):

``ops``      the reference's operators one by one, as a drop-in user's time loop
             calls them: prim_to_cons, time_step, godunov, cons_to_prim.
``sim``      a device-resident simulation: load a state, advance it, read it back.
``batch``    many uneven grids advanced together.
``adjoint``  a differentiable evolution: the forward pass and its gradient.

Extents are those of the arrays, ghost layers included.  States are seeded:
``random`` is the operator benchmark's distribution (rho and p log-uniform on
[0.1, 10], u ~ N(0, 1)); ``implode`` is the implosion's two states with a
seeded density perturbation, so most of the gas starts at rest.
"""
from __future__ import annotations

import math
import os
import random
import sys

import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "benchmark-euler-kernels_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import euler_gb300 as E  # noqa: E402
from euler_gb300.autograd import evolve  # noqa: E402

GAMMA = 1.4
CFL = 0.4
BATCH_GAMMAS = (1.4, 5.0 / 3.0, 1.3)
BATCH_EXTENTS = (24, 32, 48, 64, 96, 128)  # interior extents of the batched workload


def listed():
    return [
        # a drop-in user's loop on the smallest grid the tests step: four launches, latency only
        dict(name="ops_f64_16", kind="ops", dtype="f64", bitwise=False, n0=18, n1=18, n2=18),
        # the reference's per-operator benchmark at the size its results are quoted on most
        dict(name="ops_f64_256", kind="ops", dtype="f64", bitwise=False, n0=258, n1=258, n2=258),
        # the bit-identical godunov on a ragged grid: someone reproducing reference results
        dict(name="ops_bitwise_ragged", kind="ops", dtype="f64", bitwise=True, n0=131, n1=98, n2=75),
        # the reference built with real_t = float
        dict(name="ops_f32_256", kind="ops", dtype="f32", bitwise=False, n0=258, n1=258, n2=258),
        # the reference's own program: the 64^3 implosion, 100 steps
        dict(name="sim_f64_implode_64", kind="sim", precision="f64", state="implode", n0=66, n1=66, n2=66, steps=100),
        # uneven extents with an odd row pitch: no 16-byte row alignment
        dict(name="sim_f64_ragged", kind="sim", precision="f64", state="random", n0=101, n1=130, n2=77, steps=20),
        # the headline size: 512^3, FP64
        dict(name="sim_f64_512", kind="sim", precision="f64", state="random", n0=514, n1=514, n2=514, steps=4),
        # the mixed-precision state on a production-sized grid
        dict(name="sim_f32c_256", kind="sim", precision="f32c", state="implode", n0=258, n1=258, n2=258, steps=100),
        # the double-float state, uneven extents
        dict(name="sim_hilo_ragged", kind="sim", precision="f32c_hilo", state="random", n0=202, n1=149, n2=133,
             steps=50),
        # a parameter sweep of small FP64 runs, tiling tuned first
        dict(name="batch_f64_24", kind="batch", precision="f64", grids=24, mix=1, ragged=False, tune=True, steps=20),
        # the same in mixed precision: more grids, default tiling
        dict(name="batch_f32c_48", kind="batch", precision="f32c", grids=48, mix=2, ragged=False, tune=False,
             steps=100),
        # an inverse problem's gradient evaluation
        dict(name="adjoint_64", kind="adjoint", n0=66, n1=66, n2=66, steps=20, every=10),
    ]


def draw(rng):
    """One more case of the same ranges; costs no more than sim_f64_512."""

    def extent(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("ops", "ops", "sim", "sim", "sim", "batch", "adjoint"))
    if kind == "ops":
        n = [extent(10, 300) for _ in range(3)]
        dtype = rng.choice(("f64", "f64", "f32"))
        return dict(kind="ops", dtype=dtype, bitwise=rng.random() < 0.3, n0=n[0], n1=n[1], n2=n[2])
    if kind == "sim":
        precision = rng.choice(("f64", "f64", "f32c", "f32c_hilo", "f32"))
        n = [extent(14, 300) for _ in range(3)]
        most = max(2, min(100, int(4e8 / (n[0] * n[1] * n[2]))))
        steps = extent(2, most) if most > 2 else 2
        return dict(kind="sim", precision=precision, state=rng.choice(("random", "implode")), n0=n[0], n1=n[1],
                    n2=n[2], steps=steps)
    if kind == "batch":
        grids = extent(4, 48)
        return dict(kind="batch", precision=rng.choice(("f64", "f32c", "f32", "f32c_hilo")), grids=grids,
                    mix=rng.randrange(1 << 20), ragged=rng.random() < 0.6, tune=False,
                    steps=2 * extent(2, 10))
    n = [extent(14, 98) for _ in range(3)]
    steps = extent(4, 24)
    return dict(kind="adjoint", n0=n[0], n1=n[1], n2=n[2], steps=steps, every=rng.randint(2, 12))


# ------------------------------------------------------------------ inputs
def _spacing(n):
    return tuple(1.0 / (v - 2) for v in n)


def _random_prim(n, gen, dtype=torch.float64):
    p = torch.randn((5, n[2], n[1], n[0]), dtype=dtype, device="cuda", generator=gen)
    p[:2].uniform_(math.log(0.1), math.log(10.0), generator=gen).exp_()
    return p


def _implode_prim(n, gen):
    """The implosion's two states (a sphere of radius 1/4 around the cube's centre), density perturbed by 1 %."""
    dx = _spacing(n)
    x = [((torch.arange(v, device="cuda", dtype=torch.float64) - 0.5) * h - 0.5) ** 2 for v, h in zip(n, dx)]
    inside = x[2][:, None, None] + x[1][None, :, None] + x[0][None, None, :] < 0.25 ** 2
    p = torch.zeros((5, n[2], n[1], n[0]), dtype=torch.float64, device="cuda")
    p[0] = torch.where(inside, 1.0, 0.125)
    p[1] = torch.where(inside, 1.0, 0.14)
    p[0] *= 1.0 + 0.01 * torch.randn(p[0].shape, dtype=torch.float64, device="cuda", generator=gen)
    return p


def _step_prim(n, c, gen):
    """A plane discontinuity, as the batched workload starts from, density perturbed by 1 %."""
    x = [(torch.arange(v, device="cuda", dtype=torch.float64) - 0.5) / (v - 2) for v in n]
    inside = x[2][:, None, None] + x[1][None, :, None] + x[0][None, None, :] < c
    p = torch.zeros((5, n[2], n[1], n[0]), dtype=torch.float64, device="cuda")
    p[0] = torch.where(inside, 1.0, 0.125)
    p[1] = torch.where(inside, 1.0, 0.1)
    p[0] *= 1.0 + 0.01 * torch.randn(p[0].shape, dtype=torch.float64, device="cuda", generator=gen)
    return p


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _extents(case):
    return (case["n0"], case["n1"], case["n2"])


def _batch_grids(case):
    """(n0, n1, n2, gamma, dx0, dx1, dx2) of every grid: the case's own, whatever the seed."""
    r = random.Random(case["mix"])
    grids = []
    for g in range(case["grids"]):
        if case["ragged"]:
            n = [int(round(math.exp(r.uniform(math.log(12), math.log(110))))) + 2 for _ in range(3)]
        else:
            n = [r.choice(BATCH_EXTENTS) + 2 for _ in range(3)]
        grids.append((*n, BATCH_GAMMAS[g % 3], *_spacing(n)))
    return grids


def _batch_inputs(case, seed):
    gen = _generator(seed)
    r = random.Random(seed)
    return [_step_prim(g[:3], r.uniform(0.6, 1.8), gen) for g in _batch_grids(case)]


def _input(case, seed):
    n, gen = _extents(case), _generator(seed)
    if case["kind"] == "ops":
        return _random_prim(n, gen, torch.float64 if case["dtype"] == "f64" else torch.float32)
    if case["kind"] == "sim" and case["state"] == "implode":
        return _implode_prim(n, gen)
    return _random_prim(n, gen)


def _cotangent(case, seed):
    n = _extents(case)
    return torch.randn((5, n[2], n[1], n[0]), dtype=torch.float64, device="cuda", generator=_generator(seed + 1000003))


# ------------------------------------------------------------------- passes
def prepare(case, seed):
    s = dict(case)
    if case["kind"] == "ops":
        s["prim"] = _input(case, seed)
        s["cons"] = torch.empty_like(s["prim"])
        s["out"] = torch.empty_like(s["prim"])
        s["dt"] = torch.empty((), dtype=s["prim"].dtype, device="cuda")
        s["dx"] = _spacing(_extents(case))
    elif case["kind"] == "sim":
        n = _extents(case)
        s["prim"] = _input(case, seed)
        s["sim"] = E.Simulation(*n, gamma=GAMMA, dx=_spacing(n), cfl=CFL, precision=case["precision"])
        s["out"] = torch.empty_like(s["prim"])
        s["cons"] = torch.empty_like(s["prim"]) if case["precision"] == "f64" else None
    elif case["kind"] == "batch":
        grids = _batch_grids(case)
        s["prims"] = _batch_inputs(case, seed)
        torch.cuda.synchronize()  # the batch runs on a stream of its own
        s["batch"] = E.Batch(grids, cfl=CFL, precision=case["precision"])
        if case["tune"]:
            for g, p in enumerate(s["prims"]):
                s["batch"].set_prim(g, p)
            s["batch"].autotune()
        flat = torch.empty(sum(p.numel() for p in s["prims"]), dtype=torch.float64, device="cuda")
        s["flat"], s["outs"], at = flat, [], 0
        for p in s["prims"]:  # one buffer, a bundle of it for each grid
            s["outs"].append(flat[at:at + p.numel()].view(p.shape))
            at += p.numel()
    else:
        s["prim"] = _input(case, seed).requires_grad_(True)
        s["bar"] = _cotangent(case, seed)
        s["dx"] = _spacing(_extents(case))
    return s


def run(s):
    if s["kind"] == "ops":
        prim, cons, dt = s["prim"], s["cons"], s["dt"]
        E.prim_to_cons(prim, GAMMA, out=cons)
        E.time_step(prim, GAMMA, s["dx"], out=dt)
        if s["bitwise"] or s["dtype"] == "f32":  # these take dt as a number, as the reference does
            E.godunov(prim, cons, GAMMA, s["dx"], CFL * float(dt), exact=s["bitwise"])
        else:
            E.godunov(prim, cons, GAMMA, s["dx"], (dt, CFL))
        E.cons_to_prim(cons, GAMMA, out=s["out"])
        return {"cons": cons, "dt": dt, "prim": s["out"]}
    if s["kind"] == "sim":
        sim = s["sim"]
        sim.set_prim(s["prim"])
        sim.advance(s["steps"])
        if s["precision"] == "f64":
            sim.get_state(s["out"], s["cons"])
            return {"prim": s["out"], "cons": s["cons"], "t": sim.time()[0]}
        sim.get_state(s["out"])
        return {"prim": s["out"].float(), "t": sim.time()[0]}  # the state's own precision
    if s["kind"] == "batch":
        batch = s["batch"]
        for g, p in enumerate(s["prims"]):
            batch.set_prim(g, p)
        batch.advance(s["steps"])
        for g, o in enumerate(s["outs"]):
            E.check(E.load().eulr_batch_get_state_f64(batch._h, g, E.bundle(o), E.null_bundle()))
        return {"prim": s["flat"] if s["precision"] == "f64" else s["flat"].float()}
    out = evolve(s["prim"], s["steps"], GAMMA, s["dx"], CFL, checkpoint_every=s["every"])
    (grad,) = torch.autograd.grad(out, s["prim"], s["bar"])
    return {"prim": out.detach(), "grad": grad}


# --------------------------------------------------------------------- work
def work(case):
    """Words in and out once per operator, step or reverse step; FLOPs of the reference's templates with each
    face solved once: 250 godunov, 13 prim_to_cons, 14 cons_to_prim, 12 wavespeed, 276 a whole step."""
    if case["kind"] == "batch":
        word = 8 if case["precision"] == "f64" else 8 if case["precision"] == "f32c_hilo" else 4
        cells = sum(g[0] * g[1] * g[2] for g in _batch_grids(case))
        inner = sum((g[0] - 2) * (g[1] - 2) * (g[2] - 2) for g in _batch_grids(case))
        return {"bytes": 80 * cells + 10 * word * inner * case["steps"], "flops": 276 * inner * case["steps"]}
    n = _extents(case)
    cells = n[0] * n[1] * n[2]
    inner = (n[0] - 2) * (n[1] - 2) * (n[2] - 2)
    if case["kind"] == "ops":
        word = 8 if case["dtype"] == "f64" else 4
        return {"bytes": word * (10 + 5 + 15 + 10) * cells, "flops": 39 * cells + 250 * inner}
    if case["kind"] == "sim":
        word = 4 if case["precision"] in ("f32", "f32c") else 8
        return {"bytes": (120 if case["precision"] == "f64" else 80) * cells + 10 * word * inner * case["steps"],
                "flops": 276 * inner * case["steps"]}
    # a forward step, and a reverse step: the state and the cotangent in, the cotangent out; its FLOPs are
    # those of the forward step and twice as many again
    return {"bytes": 80 * cells + (80 + 120) * inner * case["steps"], "flops": 4 * 276 * inner * case["steps"]}


# -------------------------------------------------- the same in plain torch
def _p2c(p, gamma):
    ke = 0.5 * p[0] * (p[2] ** 2 + p[3] ** 2 + p[4] ** 2)
    return [p[0], ke + p[1] / (gamma - 1.0), p[0] * p[2], p[0] * p[3], p[0] * p[4]]


def _c2p(c, gamma):
    ke = 0.5 * (c[2] ** 2 + c[3] ** 2 + c[4] ** 2) / c[0]
    return [c[0], (gamma - 1.0) * (c[1] - ke), c[2] / c[0], c[3] / c[0], c[4] / c[0]]


def _time_step(p, gamma, dx):
    cs = torch.sqrt(gamma * p[1] / p[0])
    return 1.0 / sum((cs + p[2 + a].abs()) / dx[a] for a in range(3)).max()


def _hllc(L, R, a, gamma):
    """Flux of the faces between states L and R along axis a, in the global components."""
    t1, t2 = (2 + b for b in range(3) if b != a)
    un = 2 + a
    cmax = torch.maximum(torch.sqrt(gamma * L[1] / L[0]), torch.sqrt(gamma * R[1] / R[0]))
    SL = torch.minimum(L[un], R[un]) - cmax
    SR = torch.maximum(L[un], R[un]) + cmax
    del cmax
    rL, rR = L[0] * (SL - L[un]), R[0] * (SR - R[un])
    us = (R[1] - L[1] + rL * L[un] - rR * R[un]) / (rL - rR)
    ps = 0.5 * (L[1] + R[1] + rL * (us - L[un]) + rR * (us - R[un]))
    del rL, rR
    left = us > 0
    S = torch.where(left, SL, SR)
    over = SL * SR > 0
    del SL, SR
    d, p, u = (torch.where(left, L[f], R[f]) for f in (0, 1, un))
    v1, v2 = (torch.where(left, L[f], R[f]) for f in (t1, t2))
    e = p / (gamma - 1.0) + 0.5 * d * (u * u + v1 * v1 + v2 * v2)
    del left
    ratio = torch.where(over, torch.ones_like(u), (S - u) / (S - us))
    extra = torch.where(over, torch.zeros_like(u), (ps * us - p * u) / (S - us))
    un_o, p_o = torch.where(over, u, us), torch.where(over, p, ps)
    m = ratio * d * un_o
    f = [None] * 5
    f[0], f[1], f[un], f[t1], f[t2] = m, (ratio * e + extra + p_o) * un_o, m * un_o + p_o, m * v1, m * v2
    return f


def _inner(v, axes=(0, 1, 2)):
    for a in axes:
        v = v.narrow(2 - a, 1, v.shape[2 - a] - 2)
    return v


def _update(p, c, gamma, dx, dt):
    """cons after one godunov step: interior cells updated, ghosts kept."""
    total = None
    for a in range(3):
        q = [_inner(v, [b for b in range(3) if b != a]) for v in p]
        n = q[0].shape[2 - a]
        f = _hllc([v.narrow(2 - a, 0, n - 1) for v in q], [v.narrow(2 - a, 1, n - 1) for v in q], a, gamma)
        diff = [(v.narrow(2 - a, 1, n - 2) - v.narrow(2 - a, 0, n - 2)) * (dt / dx[a]) for v in f]
        del f
        total = diff if total is None else [t + v for t, v in zip(total, diff)]
    return [torch.nn.functional.pad(-t, (1,) * 6) + v for t, v in zip(total, c)]


def _evolve(p, gamma, dx, steps):
    p = list(p.unbind(0))
    c = _p2c(p, gamma)
    t = 0.0
    for _ in range(steps):
        with torch.no_grad():
            dt = CFL * _time_step(p, gamma, dx)
        t = t + dt
        c = _update(p, c, gamma, dx, dt)
        p = _c2p(c, gamma)
    return p, c, t


def exact(case, seed):
    if case["kind"] == "batch":
        outs = [torch.stack(_evolve(p, g[3], g[4:], case["steps"])[0]).reshape(-1)
                for g, p in zip(_batch_grids(case), _batch_inputs(case, seed))]
        return {"prim": torch.cat(outs)}
    n = _extents(case)
    dx = _spacing(n)
    prim = _input(case, seed).double()
    if case["kind"] == "ops":
        p = list(prim.unbind(0))
        dt = _time_step(p, GAMMA, dx)
        c = _update(p, _p2c(p, GAMMA), GAMMA, dx, CFL * dt)
        return {"cons": torch.stack(c), "dt": dt, "prim": torch.stack(_c2p(c, GAMMA))}
    if case["kind"] == "sim":
        p, c, t = _evolve(prim, GAMMA, dx, case["steps"])
        if case["precision"] == "f64":
            return {"prim": torch.stack(p), "cons": torch.stack(c), "t": float(t)}
        return {"prim": torch.stack(p), "t": float(t)}
    prim.requires_grad_(True)
    out = torch.stack(_evolve(prim, GAMMA, dx, case["steps"])[0])
    (grad,) = torch.autograd.grad(out, prim, _cotangent(case, seed))
    return {"prim": out.detach(), "grad": grad}
