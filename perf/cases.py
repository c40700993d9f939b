"""The work that programs built on hprqp have it do, as cases that can be timed.

A program either holds a built model and solves it (`optimize`), holds a
device-resident batch and solves it again and again (`Batch`), hands a whole
batch over in one call (`solve_batch`), trains through the layer (`QPLayer`),
or differentiates one large solve (`solve_for_backward`).  The sizes are those
of the repository's own recipes (hprqp.instances): the plain QP of n = 1000,
the large sparse QP, the factor portfolio, the batch of n = 50..2000, the
n = 500 differentiation batch and the cone models.  Every solve has an
iteration limit, as a program with a time budget sets one.

Outputs are the solution vectors, objectives, statuses and iteration counts
(and gradients); residual norms and times are not among them: the former are
differences of nearly equal numbers, the latter change from run to run.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "hpr-qp-c_b200", "python"))

import hprqp  # noqa: E402
from hprqp import instances  # noqa: E402
from hprqp.batch import Batch, pack, solve_batch  # noqa: E402
from hprqp.torch_layer import QPLayer  # noqa: E402


def listed():
    return [
        # a controller or a subproblem solver: one small QP per call, where the
        # call's fixed costs and the latency of an iteration count
        {"name": "single n=120", "kind": "single", "n": 120, "m": 60, "a_density": 0.05, "q_row_nnz": 6.0,
         "stoptol": 1e-6, "max_iter": 20000},
        # the plain recipe at its own size
        {"name": "single n=1000", "kind": "single", "n": 1000, "m": 500, "a_density": 0.01, "q_row_nnz": 6.0,
         "stoptol": 1e-6, "max_iter": 20000},
        # a mid-size QP, beyond what one thread block takes on
        {"name": "single n=3001", "kind": "single", "n": 3001, "m": 1700, "a_density": 0.015, "q_row_nnz": 40.0,
         "stoptol": 1e-6, "max_iter": 10000},
        # the large sparse QP (nnz(Q) 6.4e6, nnz(A) 2e6 at n = 200,000)
        {"name": "large n=200000", "kind": "large", "n": 200000, "max_iter": 800, "stoptol": 1e-6},
        # the factor portfolio: a diagonal Q and few, very long rows in A
        {"name": "portfolio n=60000", "kind": "portfolio", "assets": 60000, "factors": 120, "sectors": 300,
         "stoptol": 1e-6, "max_iter": 3000},
        # a second-order cone model (every cone on the host-driven path)
        {"name": "cone n=340", "kind": "cone", "n_lin": 300, "cone": 40, "m_lin": 90, "row_cone": 31,
         "stoptol": 1e-6, "max_iter": 3000},
        # scenarios of one decision, or the nodes of one branching step: a
        # few QPs of uneven size, solved together
        {"name": "batch 24", "kind": "batch", "count": 24, "n_low": 50, "n_high": 2000, "stoptol": 1e-6,
         "max_iter": 20000},
        # the batch recipe, held on the device
        {"name": "batch 400", "kind": "batch", "count": 400, "n_low": 50, "n_high": 2000, "stoptol": 1e-6,
         "max_iter": 20000},
        # a service that gets many small QPs at once, in one call from host arrays
        {"name": "one call 1500", "kind": "one_call", "count": 1500, "n_low": 50, "n_high": 500, "stoptol": 1e-6,
         "max_iter": 20000},
        # rolling horizon: the data moved by 1 %, started at the last solution
        {"name": "warm 96", "kind": "warm", "count": 96, "n_low": 100, "n_high": 800, "stoptol": 1e-6,
         "max_iter": 20000},
        # a training step through the layer (forward, backward to every input)
        {"name": "layer 256", "kind": "layer", "count": 256, "n": 500, "m": 300, "stoptol": 1e-8,
         "max_iter": 20000},
        # a training step through one larger QP
        {"name": "backward n=8000", "kind": "backward", "n": 8000, "m": 4000, "stoptol": 1e-8, "max_iter": 10000},
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["single", "single", "large", "portfolio", "cone", "batch", "batch", "one_call", "warm",
                       "layer", "backward"])
    if kind == "single":
        n = _log(rng, 60, 3001)
        return {"kind": kind, "n": n, "m": max(8, int(n * rng.uniform(0.25, 0.7))),
                "a_density": min(0.2, rng.uniform(6.0, 40.0) / n), "q_row_nnz": rng.uniform(3.0, 40.0),
                "stoptol": 1e-6, "max_iter": 10000}
    if kind == "large":
        return {"kind": kind, "n": _log(rng, 20000, 200000), "max_iter": 800, "stoptol": rng.choice([1e-4, 1e-6])}
    if kind == "portfolio":
        return {"kind": kind, "assets": _log(rng, 2000, 60000), "factors": _log(rng, 10, 120),
                "sectors": _log(rng, 10, 300), "stoptol": 1e-6, "max_iter": 2000}
    if kind == "cone":
        return {"kind": kind, "n_lin": _log(rng, 30, 300), "cone": _log(rng, 4, 40), "m_lin": _log(rng, 10, 90),
                "row_cone": _log(rng, 3, 31), "stoptol": 1e-6, "max_iter": 3000}
    if kind == "batch":
        return {"kind": kind, "count": _log(rng, 8, 400), "n_low": 50, "n_high": _log(rng, 200, 2000),
                "stoptol": 1e-6, "max_iter": 10000}
    if kind == "one_call":
        return {"kind": kind, "count": _log(rng, 64, 1500), "n_low": 50, "n_high": _log(rng, 100, 500),
                "stoptol": 1e-6, "max_iter": 10000}
    if kind == "warm":
        return {"kind": kind, "count": _log(rng, 16, 256), "n_low": 50, "n_high": _log(rng, 100, 1000),
                "stoptol": 1e-6, "max_iter": 10000}
    if kind == "layer":
        n = _log(rng, 60, 700)
        return {"kind": kind, "count": _log(rng, 8, 256), "n": n, "m": max(8, int(n * rng.uniform(0.3, 0.7))),
                "stoptol": 1e-8, "max_iter": 10000}
    n = _log(rng, 2000, 8000)
    return {"kind": kind, "n": n, "m": n // 2, "stoptol": 1e-8, "max_iter": 10000}


# ---- inputs -----------------------------------------------------------------

def _revalued(inst, seed, n_eq):
    """An instance of the same sizes and sparsity with values of its own, as
    a program has whose structure stays and whose data change: A ~ N(0, 1),
    Q scaled symmetrically by U(0.7, 1.4), new c and rows feasible again."""
    rng = np.random.default_rng(instances.SEED_BASE + seed)
    Q, A = inst.Q, inst.A
    d = rng.uniform(0.7, 1.4, inst.n)
    Q.data = Q.data * d[np.repeat(np.arange(inst.n), np.diff(Q.indptr))] * d[Q.indices]
    A.data = rng.standard_normal(A.nnz)
    inst.c = rng.standard_normal(inst.n)
    inst.AL, inst.AU = instances._feasible_rows(rng, A, inst.n, n_eq)
    return inst


def _plain(case, seed, structure=0):
    """The plain recipe: 60 % of the rows are equalities."""
    n, m = case["n"], case["m"]
    per = case.get("q_row_nnz", 6.0)  # about this many entries in a row of Q = M'M + 0.01 I, M of n/5 rows
    inst = instances.plain_qp(instances.SEED_BASE + structure, n=n, m=m,
                              a_density=case.get("a_density", min(1.0, max(0.01, 5.0 / n))), m_rows=max(1, n // 5),
                              m_density=min(1.0, math.sqrt(5.0 * per) / n), n_eq=int(0.6 * m))
    return _revalued(inst, seed, int(0.6 * m))


def _mixed(case, seed):
    """The batch recipe with n in the case's range."""
    rng = np.random.default_rng(instances.SEED_BASE + case["count"])
    out = []
    for i in range(case["count"]):
        n = int(rng.integers(case["n_low"], case["n_high"] + 1))
        m = int(rng.integers(-(-n // 4), n + 1))
        d_a, d_q = rng.uniform(0.005, 0.05), rng.uniform(0.001, 0.02)
        inst = instances.plain_qp(int(rng.integers(2**62)), n=n, m=m, a_density=d_a, m_rows=max(1, n // 5),
                                  m_density=min(1.0, math.sqrt(5.0 * d_q / n)), n_eq=int(0.6 * m))
        out.append(_revalued(inst, 100003 * seed + i, int(0.6 * m)))
    return out


def _model(case, seed):
    kind = case["kind"]
    if kind == "cone":
        s = instances.soc_case(seed, n_lin=case["n_lin"], cone=case["cone"], m_lin=case["m_lin"],
                               row_cone=case["row_cone"])
        q = s.qp
        return hprqp.build_from_qabc_soc(q.Q, q.c, q.A, q.AL, q.AU, q.l, q.u, s.var_offsets, s.row_offsets, s.rhs)
    if kind == "large":
        inst = instances.config1_sized_plain(scale=case["n"] / 1e6)
        inst = _revalued(inst, seed, int(0.4 * inst.m))
    elif kind == "portfolio":
        assets, factors = case["assets"], case["factors"]
        inst = instances.config2(n_assets=assets, k=factors, sectors=case["sectors"])
        rng = np.random.default_rng(instances.SEED_BASE + seed)  # the same sectors, new exposures, risks and returns
        inst.A.data[:factors * (assets + 1)].reshape(factors, -1)[:, :assets] = rng.normal(0.0, 0.1, (factors, assets))
        inst.Q.data[:assets] = 2.0 * rng.uniform(0.01, 0.1, assets)
        inst.c[:assets] = rng.normal(0.0005, 0.01, assets)
    else:
        inst = _plain(case, seed)
    return hprqp.build_from_instance(inst)


def prepare(case, seed):
    kind = case["kind"]
    opts = {"stoptol": case["stoptol"], "max_iter": case["max_iter"]}
    state = {"kind": kind, "opts": opts}
    if kind in ("single", "large", "portfolio", "cone", "backward"):
        state["model"] = _model(case, seed)
        state["params"] = hprqp.Parameters(verbose=False, **opts)
        if kind == "backward":
            state["g"] = np.random.default_rng(seed).standard_normal(case["n"])
    elif kind == "batch":
        state["batch"] = Batch(pack(_mixed(case, seed)))
    elif kind == "one_call":
        state["packed"] = pack(_mixed(case, seed))
    elif kind == "warm":
        packed = pack(_mixed(case, seed))
        first = solve_batch(packed, **opts)
        rng = np.random.default_rng(seed)
        packed.c *= 1.0 + 0.01 * rng.standard_normal(len(packed.c))
        state["batch"] = Batch(packed)
        state["point"] = (first.x, first.y, first.w, first.sigma)
    elif kind == "layer":
        packed = pack([_plain(case, 100003 * seed + i, i) for i in range(case["count"])])
        state["layer"] = QPLayer(packed, stoptol=case["stoptol"], max_iter=case["max_iter"])
        state["inputs"] = [torch.from_numpy(a.copy()).cuda().requires_grad_(True)
                           for a in (packed.q_data, packed.a_data, packed.c, packed.AL, packed.AU, packed.l, packed.u)]
        g = torch.Generator().manual_seed(seed)
        state["g"] = torch.randn(len(packed.c), generator=g, dtype=torch.float64).cuda()
    return state


# ---- one pass ---------------------------------------------------------------

def _result(r):
    return {"x": r.x, "y": r.y, "z": r.z, "w": r.w, "objective": r.objective, "iter": r.iter,
            "status": r.status if isinstance(r.status, np.ndarray) else r.status_code}


def run(state):
    kind, opts = state["kind"], state["opts"]
    if kind in ("single", "large", "portfolio", "cone"):
        return _result(hprqp.optimize(state["model"], state["params"], as_numpy=True))
    if kind == "batch":
        state["batch"].solve(**opts)
        return _result(state["batch"].results())
    if kind == "one_call":
        return _result(solve_batch(state["packed"], **opts))
    if kind == "warm":
        state["batch"].set_warm_start(*state["point"])
        state["batch"].solve(**opts)
        return _result(state["batch"].results())
    if kind == "layer":
        for t in state["inputs"]:
            t.grad = None
        x, y = state["layer"](*state["inputs"])
        (state["g"] @ x).backward()
        return {"x": x.detach(), "y": y.detach(), "grad": [t.grad for t in state["inputs"]]}
    r, solved = hprqp.solve_for_backward(state["model"], state["params"])
    try:
        g = solved.backward(state["g"])
    finally:
        solved.close()
    return {**_result(r), "grad": [g[k] for k in ("dc", "dl", "du", "dAL", "dAU", "dQ_values", "dA_values")]}


# ---- what a pass cannot do without ------------------------------------------

def work(case):
    """One reading of the data and one writing of the results, and the
    operations of the iterations that such a solve takes (2 flops an entry,
    four products an iteration; 1000 iterations, or the limit if that is less)."""
    kind = case["kind"]
    if kind == "large":
        n, m = case["n"], case["n"] / 2
        q, a, k = 32.25 * n, 10.0 * n, 1
    elif kind == "portfolio":
        n, m = case["assets"] + case["factors"], case["factors"] + case["sectors"] + 1
        q, a, k = n, case["assets"] * (case["factors"] + 2.0), 1
    elif kind == "cone":
        n, m = case["n_lin"] + case["cone"], case["cone"] + case["m_lin"] + case["row_cone"]
        q, a, k = n, 0.45 * m * case["n_lin"], 1
    elif kind in ("batch", "one_call", "warm"):
        lo, hi, k = case["n_low"], case["n_high"], case["count"]
        n = (lo + hi) / 2.0
        n2 = (lo * lo + lo * hi + hi * hi) / 3.0  # mean of n^2
        m, q, a = 0.625 * n, 0.0105 * n2 + n, 0.0275 * 0.625 * n2
    else:
        n, m, k = case["n"], case["m"], case.get("count", 1)
        q = (case.get("q_row_nnz", 6.0) + 1.0) * n
        a = case.get("a_density", min(1.0, max(0.01, 5.0 / n))) * m * n
    iters = min(1000, case["max_iter"])
    passes = 2 if kind in ("layer", "backward") else 1
    data = 12.0 * (q + a) + 8.0 * (3 * n + 2 * m)
    out = 8.0 * (3 * n + m) + (8.0 * (q + a + 3 * n + 2 * m) if passes == 2 else 0.0)
    return {"bytes": k * (data + out), "flops": k * passes * iters * (4.0 * q + 4.0 * a)}


# ---- the exact solution -----------------------------------------------------

def _optimum(inst):
    """The optimum of one strictly convex QP to 1e-10 or better: a primal-dual
    interior-point method (Mehrotra's steps) on dense matrices in 64 bits.
    Returns x, y, z in the solver's signs: Q x + c - A'y - z = 0."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=dev)  # noqa: E731
    Q, A = t(inst.Q.dense()), t(inst.A.dense())
    Q = 0.5 * (Q + Q.T)
    eq = np.asarray(inst.AL == inst.AU)
    E, b, G = A[t(eq).bool()], t(inst.AL[eq]), A[t(~eq).bool()]
    c, n, p = t(inst.c), inst.n, int(eq.sum())
    # inequalities H x <= h: both sides of the ranged rows and of the box
    eye = torch.eye(n, dtype=torch.float64, device=dev)
    H = torch.cat([G, -G, eye, -eye])
    h = torch.cat([t(inst.AU[~eq]), -t(inst.AL[~eq]), t(inst.u), -t(inst.l)])
    x, y = torch.zeros(n, dtype=torch.float64, device=dev), torch.zeros(p, dtype=torch.float64, device=dev)
    s, v = torch.ones_like(h), torch.ones_like(h)
    best = (math.inf, x, y, v)
    for _ in range(60):
        rd, rp, rh, mu = Q @ x + c + E.T @ y + H.T @ v, E @ x - b, H @ x + s - h, (s @ v).item() / len(h)
        off = max(rd.abs().max().item(), rp.abs().max().item() if p else 0.0, rh.abs().max().item(), mu)
        if off < best[0]:
            best = (off, x, y, v)
        if off < 1e-12 or mu < 1e-15 or not math.isfinite(off):
            break
        M = Q + H.T @ ((v / s)[:, None] * H)
        K = torch.cat([torch.cat([M, E.T], 1), torch.cat([E, torch.zeros(p, p, dtype=torch.float64, device=dev)], 1)])
        lu, piv = torch.linalg.lu_factor(K)

        def step(rc):
            rhs = torch.cat([-rd + H.T @ ((rc - v * rh) / s), -rp])
            d = torch.linalg.lu_solve(lu, piv, rhs[:, None])[:, 0]
            r = rhs - K @ d
            d = d + torch.linalg.lu_solve(lu, piv, r[:, None])[:, 0]
            dx, dy = d[:n], d[n:]
            ds = -rh - H @ dx
            return dx, dy, ds, (-rc - v * ds) / s

        def longest(a, da):
            neg = da < 0
            return min(1.0, (-a[neg] / da[neg]).min().item()) if bool(neg.any()) else 1.0

        _, _, ds, dv = step(s * v)
        ap, ad = longest(s, ds), longest(v, dv)
        sig = (((s + ap * ds) @ (v + ad * dv)).item() / len(h) / mu) ** 3
        dx, dy, ds, dv = step(s * v + ds * dv - sig * mu)
        a = 0.995 * min(longest(s, ds), longest(v, dv))
        x, y, s, v = x + a * dx, y + a * dy, s + a * ds, v + a * dv
    _, x, y, v = best
    g, yy = G.shape[0], np.zeros(inst.m)
    yy[eq] = -y.cpu().numpy()
    yy[~eq] = (v[g:2 * g] - v[:g]).cpu().numpy()
    return x.cpu().numpy(), yy, (v[2 * g + n:] - v[2 * g:2 * g + n]).cpu().numpy()


def exact(case, seed):
    """The exact optimum of the single QPs; the others are too large for a
    dense method, or end at their iteration limit."""
    if case["kind"] != "single" or case["n"] > 1500:
        return None
    inst = _plain(case, seed)
    x, y, z = _optimum(inst)
    obj = 0.5 * x @ (inst.Q.dense() @ x) + inst.c @ x
    return {"x": x, "y": y, "z": z, "w": x, "objective": float(obj), "iter": None, "status": None}
