"""Performance cases: the solves and network calls that programs make through the C ABI.

Every case is one call of the public C interface (include/sov_ipm.h) on host arrays, as a C or C++
program makes it: models, options and result arrays are in hand before the call, the call itself
builds the standard form, solves on the GPU and fills the caller's arrays. Instances are seeded and
synthetic, with the shapes of the generators in sovereign_b200/problems.py.

Outputs are what determines the answer: status, objective and primal values of a solve, and its row
multipliers or dual slacks where the optimum determines them. Transportation problems with integer
supplies and multicommodity flows are primal degenerate and have redundant rows: their multipliers
are not unique (a permutation of the columns moves them by 1e-2), so they are not returned here.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from sovereign_b200 import abi, problems as P
from sovereign_b200._lib import check, load
from sovereign_b200.model import Model
from sovereign_b200.warmstart import Mlp


def listed() -> list[dict]:
    return [
        # one small LP on its own, the latency of a single solve: the 2500-variable transportation LP
        dict(name="lp_transport_50x50", kind="transport", ns=50, nt=50),
        # one medium LP whose dense normal matrix dominates: m = 2000, n = 10000, 8 nonzeros a column
        dict(name="lp_random_2000", kind="random", m=2000, n=10000, k=8, precision=abi.PRECISION_FP64),
        # the mixed-precision option of the single-problem engine (FP32 factor, FP64 PCG)
        dict(name="lp_random_700_mixed", kind="random", m=700, n=3500, k=8, precision=abi.PRECISION_MIXED),
        # a handful of uneven LPs at once: too few to fill the GPU
        dict(name="batch_24", kind="batch", count=24, lo=10, hi=60),
        # a round of branch-and-bound nodes: one LP with bounds moved by branching, ragged bound rows
        dict(name="batch_nodes_200", kind="nodes", count=200, m=37, n=91),
        # the throughput workload: 4096 uneven transportation LPs
        dict(name="batch_4096", kind="batch", count=4096, lo=10, hi=60),
        # a parametric family that shares its constraint matrix: multicommodity flows, m = 1800
        dict(name="family_64", kind="family", count=64, nodes=200, arcs=1000),
        # convex-sequence QP (separable, banded rows): the double-double path
        dict(name="qp_sequence_20002", kind="sequence", n=20002),
        # portfolio QP with a coupled Hessian and sector rows: the dense H path
        dict(name="qp_portfolio_400", kind="portfolio", assets=400, sectors=24),
        # QP with a sparse coupled Hessian: the quasi-definite KKT path
        dict(name="qp_chain_5000", kind="chain", n=5000),
        # training: loss and gradient of the warm-start network on one mini-batch (multicommodity sizes)
        dict(name="warm_grad_256", kind="grad", n_in=4040, n_out=11800, hidden=512, layers=3, batch=256),
        # inference: interior starts for a batch of LPs (40 x 40 transportation family)
        dict(name="warm_predict_4096", kind="predict", ns=40, nt=40, hidden=512, layers=3, batch=4096),
    ]


def _log(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["transport", "random", "mixed", "batch", "nodes", "family", "sequence", "portfolio", "chain",
                       "grad", "predict"])
    if kind == "transport":
        return dict(kind=kind, ns=_log(rng, 5, 90), nt=_log(rng, 5, 90))
    if kind in ("random", "mixed"):
        m = _log(rng, 150, 1700 if kind == "random" else 900)
        return dict(kind="random", m=m, n=m * rng.randint(3, 5) + rng.randint(0, 99), k=rng.randint(5, 10),
                    precision=abi.PRECISION_FP64 if kind == "random" else abi.PRECISION_MIXED)
    if kind == "batch":
        return dict(kind=kind, count=_log(rng, 4, 3500), lo=rng.randint(6, 20), hi=rng.randint(30, 60))
    if kind == "nodes":
        m = rng.randint(10, 45)
        return dict(kind=kind, count=_log(rng, 8, 1024), m=m, n=int(m * rng.uniform(2.0, 3.0)))
    if kind == "family":
        nodes = rng.randint(60, 180)
        return dict(kind=kind, count=_log(rng, 8, 64), nodes=nodes, arcs=5 * nodes)
    if kind == "sequence":
        return dict(kind=kind, n=_log(rng, 400, 18000))
    if kind == "portfolio":
        return dict(kind=kind, assets=_log(rng, 60, 900), sectors=rng.randint(4, 60))
    if kind == "chain":
        return dict(kind=kind, n=_log(rng, 1200, 8000))
    if kind == "grad":
        nodes = rng.randint(60, 200)
        return dict(kind=kind, n_in=40 + 20 * nodes, n_out=59 * nodes, hidden=rng.choice([256, 512]),
                    layers=rng.randint(2, 3), batch=_log(rng, 32, 512))
    return dict(kind=kind, ns=rng.randint(15, 40), nt=rng.randint(15, 40), hidden=rng.choice([256, 512]),
                layers=rng.randint(2, 3), batch=_log(rng, 32, 4000))


# --------------------------------------------------------------------------------------- instances

def _nodes(count: int, m: int, n: int, seed: int) -> list[Model]:
    """Nodes of one branch-and-bound tree: an LP over m rows and n columns, about a third of them with
    a finite upper bound, and per node a few columns whose bounds branching has moved. A point x0
    stays feasible in every node, and the costs have a dual feasible point, so every node has an optimum."""
    rng = np.random.default_rng(seed)
    base = P.random_sparse_lp(m, n, 4, seed)
    ub = np.full(n, P.INF)
    has = rng.permutation(n)[: min(n // 3, 120 - m)]
    ub[has] = rng.uniform(1.0, 4.0, has.size)
    x0 = rng.uniform(0.2, 0.8, n) * np.minimum(ub, 1.5)
    cols = np.repeat(np.arange(n), 4)
    sense = rng.choice(np.array([abi.LE, abi.GE, abi.EQ], dtype=np.int8), m, p=[0.5, 0.25, 0.25])
    slack = rng.uniform(0.0, 1.0, m) * (rng.random(m) < 0.5)
    rhs = np.bincount(base.row_idx, weights=base.values * x0[cols], minlength=m)
    rhs += np.where(sense == abi.LE, slack, np.where(sense == abi.GE, -slack, 0.0))
    y0 = np.abs(rng.standard_normal(m))
    y0 = np.where(sense == abi.LE, -y0, np.where(sense == abi.GE, y0, rng.standard_normal(m)))
    obj = (base.values * y0[base.row_idx]).reshape(n, 4).sum(axis=1)
    obj += np.where(ub < P.INF, rng.standard_normal(n), rng.uniform(0.1, 1.0, n))
    out = []
    for _ in range(count):
        lo, hi = np.zeros(n), ub.copy()
        for j in rng.choice(has, size=int(rng.integers(0, 7)), replace=False):
            if rng.random() < 0.5:
                hi[j] = x0[j] + rng.uniform(0.05, 1.0) * (ub[j] - x0[j])
            else:
                lo[j] = x0[j] * rng.uniform(0.0, 0.9)
        out.append(Model(n=n, m=m, col_ptr=base.col_ptr, row_idx=base.row_idx, values=base.values, obj=obj, rhs=rhs,
                         sense=sense, lb=lo, ub=hi))
    return out


def _portfolio(assets: int, sectors: int, seed: int) -> Model:
    mdl = P.reference_portfolio(assets, sectors)
    rng = np.random.default_rng(seed)
    mdl.obj = mdl.obj * rng.uniform(0.5, 1.5, assets)
    cols = np.repeat(np.arange(assets), np.diff(mdl.q_col_ptr))
    diag = mdl.q_row_idx == cols
    mdl.q_values = np.where(diag, mdl.q_values * rng.uniform(0.8, 1.3, mdl.q_values.size), mdl.q_values)
    return mdl


def _models(case: dict, seed: int) -> list[Model]:
    kind = case["kind"]
    if kind == "transport":
        return [P.transport(case["ns"], case["nt"], seed)]
    if kind == "random":
        return [P.random_sparse_lp(case["m"], case["n"], case["k"], seed)]
    if kind == "batch":  # the case's own uneven sizes, every LP's data from the seed
        sizes = np.random.default_rng(case["count"]).integers(case["lo"], case["hi"] + 1, (case["count"], 2))
        return [P.transport(int(a), int(b), 1000003 * seed + q) for q, (a, b) in enumerate(sizes)]
    if kind == "nodes":
        return _nodes(case["count"], case["m"], case["n"], seed)
    if kind == "family":  # one network, demands and costs of each instance from the seed
        fam = P.MulticommodityFamily(nodes=case["nodes"], arcs=case["arcs"])
        return [fam.instance_from_seed(1000003 * seed + q)[0] for q in range(case["count"])]
    if kind == "sequence":
        return [P.convex_sequence_qp(case["n"], seed)]
    if kind == "portfolio":
        return [_portfolio(case["assets"], case["sectors"], seed)]
    return [P.coupled_chain_qp(case["n"], seed)]


# which arrays of a result the optimum determines
_OUT = dict(transport=("primal",), random=("primal", "dual_row"), batch=("primal",), nodes=("primal", "dual_row"),
            family=("primal",), sequence=("primal", "dual_row"), portfolio=("primal", "dual_row", "dual_col"),
            chain=("primal", "dual_row", "dual_col"))


class _Solves:
    """Models, options and result arrays of one call, with every result's arrays in three flat ones."""

    def __init__(self, case: dict, models: list[Model]):
        self.models = models
        qp = models[0].is_qp
        self.opt = abi.default_options(qp=qp)
        self.opt.precision = case.get("precision", abi.PRECISION_FP64)
        k = len(models)
        self.arr = (abi.SovModel * k)(*[m.to_abi() for m in models])
        self.res = (abi.SovResult * k)()
        n = np.array([m.n for m in models])
        m = np.array([m.m for m in models])
        self.flat = dict(primal=np.zeros(n.sum()), dual_col=np.zeros(n.sum()), dual_row=np.zeros(m.sum()))
        for name, size in (("primal", n), ("dual_col", n), ("dual_row", m)):
            at = np.concatenate([[0], np.cumsum(size)])
            for q in range(k):
                setattr(self.res[q], name, abi.dptr(self.flat[name][at[q]:]) if size[q] else None)
        lib = load()
        if case["kind"] in ("batch", "nodes", "family"):
            entry = lib.sov_lp_solve_family if case["kind"] == "family" else lib.sov_lp_solve_batch
            self.call = lambda: entry(k, self.arr, C.byref(self.opt), 0, self.res)
        else:
            entry = lib.sov_qp_solve if qp else lib.sov_lp_solve
            self.call = lambda: entry(C.byref(self.arr[0]), C.byref(self.opt), C.byref(self.res[0]))
        step = C.sizeof(abi.SovResult)
        self.out = {name: self.flat[name] for name in _OUT[case["kind"]]}
        self.out["status"] = np.ndarray((k,), np.int32, self.res, abi.SovResult.status.offset, (step,))
        self.out["objective"] = np.ndarray((k,), np.float64, self.res, abi.SovResult.objective_value.offset, (step,))

    def run(self) -> dict:
        check(self.call())
        return self.out


def _weights(dims: list[int], seed: int) -> np.ndarray:
    """Network parameters, layer by layer W (out x in, row-major) then b."""
    rng = np.random.default_rng(seed + 77)
    parts = []
    for a, b in zip(dims[:-1], dims[1:]):
        parts += [rng.standard_normal(a * b, dtype=np.float32) * np.float32(math.sqrt(2.0 / a)),
                  0.05 * rng.standard_normal(b, dtype=np.float32)]
    return np.concatenate(parts)


def _grad_data(case: dict, seed: int):
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((case["batch"], case["n_in"]), dtype=np.float32)
    t = rng.standard_normal((case["batch"], case["n_out"]), dtype=np.float32)
    dims = [case["n_in"]] + [case["hidden"]] * case["layers"] + [case["n_out"]]
    return dims, _weights(dims, seed), x, t


_DELTA = 1e-6


def _predict_data(case: dict, seed: int):
    rng = np.random.default_rng(seed)
    ns, nt, b = case["ns"], case["nt"], case["batch"]
    n_in, n, m = ns + nt + ns * nt, ns * nt, ns + nt
    p = np.concatenate([1.0 + 0.2 * rng.standard_normal((b, ns + nt)), 1.0 + 0.1 * rng.standard_normal((b, n))], axis=1)
    dims = [n_in] + [case["hidden"]] * case["layers"] + [2 * n + m]
    norm = (np.ones(n_in), np.concatenate([np.full(ns + nt, 0.2), np.full(n, 0.1)]),
            rng.uniform(-3.0, 3.0, 2 * n + m), rng.uniform(0.2, 0.8, 2 * n + m))
    return dims, _weights(dims, seed), p, norm, n, m


class _Grad:
    def __init__(self, case: dict, seed: int):
        dims, w, self.x, self.t = _grad_data(case, seed)
        self.mlp = Mlp(dims[0], dims[-1], case["hidden"], case["layers"])
        self.mlp.params = w
        self.grad, self.loss = np.zeros(w.size, dtype=np.float32), C.c_double()

    def run(self) -> dict:
        check(load().sov_mlp_loss_grad(self.mlp.h, self.x.ctypes.data, self.t.ctypes.data, self.x.shape[0],
                                       C.byref(self.loss), self.grad.ctypes.data))
        return dict(loss=self.loss.value, grad=self.grad)


class _Predict:
    def __init__(self, case: dict, seed: int):
        dims, w, self.p, self.norm, self.n, self.m = _predict_data(case, seed)
        self.mlp = Mlp(dims[0], dims[-1], case["hidden"], case["layers"])
        self.mlp.params = w
        b = self.p.shape[0]
        self.out = dict(x=np.zeros((b, self.n)), y=np.zeros((b, self.m)), s=np.zeros((b, self.n)))

    def run(self) -> dict:
        o = self.out
        check(load().sov_mlp_predict_start(self.mlp.h, self.p.ctypes.data, self.p.shape[0],
                                           *(v.ctypes.data for v in self.norm), self.n, self.m, _DELTA,
                                           o["x"].ctypes.data, o["y"].ctypes.data, o["s"].ctypes.data))
        return o


def prepare(case: dict, seed: int):
    if case["kind"] == "grad":
        return _Grad(case, seed)
    if case["kind"] == "predict":
        return _Predict(case, seed)
    return _Solves(case, _models(case, seed))


def run(state):
    return state.run()


# ------------------------------------------------------------------------------------------- work

def work(case: dict) -> dict:
    """Caller's arrays in and out once; arithmetic of the Newton systems at a typical iteration count
    (14 for the LPs, 12 for the coupled QPs, 60 for the convex sequence, whose values are two doubles)."""
    kind = case["kind"]
    if kind in ("grad", "predict"):
        if kind == "grad":
            dims = [case["n_in"]] + [case["hidden"]] * case["layers"] + [case["n_out"]]
        else:
            n, m = case["ns"] * case["nt"], case["ns"] + case["nt"]
            dims = [n + m] + [case["hidden"]] * case["layers"] + [2 * n + m]
        b = case["batch"]
        macs = sum(p * q for p, q in zip(dims[:-1], dims[1:]))
        params = macs + sum(dims[1:])
        if kind == "grad":
            return dict(bytes=4.0 * (b * (dims[0] + dims[-1]) + 2 * params), flops=6.0 * b * macs)
        return dict(bytes=8.0 * b * (dims[0] + dims[-1]) + 4.0 * params, flops=2.0 * b * macs)
    if kind == "batch":  # mean sizes over the uniform range
        mean = 0.5 * (case["lo"] + case["hi"])
        m, n, count = 2.0 * mean, mean * mean, case["count"]
        nnz, iters = 2.0 * n, 14.0
    elif kind == "transport":
        m, n, count = case["ns"] + case["nt"], case["ns"] * case["nt"], 1
        nnz, iters = 2.0 * n, 14.0
    elif kind == "random":
        m, n, count = case["m"], case["n"], 1
        nnz, iters = case["k"] * n, 14.0
    elif kind == "nodes":
        m, n, count = case["m"] + case["n"] // 3, case["n"], case["count"]
        nnz, iters = 4.0 * n, 14.0
    elif kind == "family":
        m, n, count = case["arcs"] + 4 * case["nodes"], 4 * case["arcs"], case["count"]
        nnz, iters = 3.0 * n, 14.0
    elif kind == "sequence":
        n = case["n"]
        return dict(bytes=8.0 * 8 * n, flops=60.0 * n * 30.0 * 20.0)
    elif kind == "portfolio":
        n, m = case["assets"], 1 + case["sectors"]
        return dict(bytes=8.0 * (12 * n + 4 * m), flops=12.0 * (n ** 3 / 3.0 + 2.0 * m * n * n))
    else:
        n = case["n"]
        return dict(bytes=8.0 * 20 * n, flops=12.0 * n * 40.0)
    if kind in ("batch", "transport", "random", "nodes"):
        per = m ** 3 / 3.0 + 4.0 * m * m + 12.0 * nnz
    else:  # sparse factor: far fewer operations than a dense one; the matrix passes alone
        per = 40.0 * nnz
    per_bytes = 12.0 * nnz + 8.0 * (5 * n + 3 * m)
    return dict(bytes=count * per_bytes, flops=count * iters * per)


# ------------------------------------------------------------------------------ 64-bit references

def _dense_form(mdl: Model):
    """(A with a slack column per inequality row, c, b, upper bounds shifted by lb) in float64."""
    rows = mdl.row_idx.astype(np.int64)
    cols = np.repeat(np.arange(mdl.n), np.diff(mdl.col_ptr))
    ineq = np.flatnonzero(mdl.sense != abi.EQ)
    A = np.zeros((mdl.m, mdl.n + ineq.size))
    np.add.at(A, (rows, cols), mdl.values)
    A[ineq, mdl.n + np.arange(ineq.size)] = np.where(mdl.sense[ineq] == abi.LE, 1.0, -1.0)
    b = mdl.rhs - A[:, :mdl.n] @ mdl.lb
    u = np.concatenate([np.where(mdl.ub < 1e29, mdl.ub - mdl.lb, np.inf), np.full(ineq.size, np.inf)])
    return A, np.concatenate([mdl.obj, np.zeros(ineq.size)]), b, u


def _interior(A, c, b, u, Q=None, rows=None, iterations=80):
    """min c'x + x'Qx/2, A x = b, 0 <= x <= u by a plain predictor-corrector method in 64 bits, for a
    stack of problems (leading dimension; A may be shared). rows: mask of real rows where problems
    are padded. Returns the iterate of the smallest residual, x, y and the lower bounds' duals."""
    T = lambda v: v.transpose(-1, -2)  # noqa: E731
    mv = lambda M, v: (M @ v.unsqueeze(-1)).squeeze(-1)  # noqa: E731
    has = torch.isfinite(u)
    uf = torch.where(has, u, torch.ones_like(u))
    one = torch.ones_like(c)
    scale = 1.0 + c.abs().amax(-1, keepdim=True)
    x = torch.where(has, 0.5 * uf, one * (1.0 + b.abs().amax(-1, keepdim=True)))
    w = torch.where(has, uf - x, one)
    zl = scale * one
    zu = torch.where(has, zl, torch.zeros_like(zl))
    y = torch.zeros_like(b)
    count = one.sum(-1, keepdim=True) + has.sum(-1, keepdim=True)
    best, keep = None, None
    for _ in range(iterations):
        qx = mv(Q, x) if Q is not None else 0.0
        rp = b - mv(A, x)
        ru = torch.where(has, uf - x - w, torch.zeros_like(x))
        rd = c + qx - mv(T(A), y) - zl + zu
        mu = ((x * zl).sum(-1, keepdim=True) + (w * zu).sum(-1, keepdim=True)) / count
        obj = (c * x).sum(-1, keepdim=True)
        err = torch.stack([rp.abs().amax(-1) / (1 + b.abs().amax(-1)), rd.abs().amax(-1) / scale[..., 0],
                           (mu * count / (1 + obj.abs()))[..., 0]]).amax(0)
        err = torch.where(torch.isfinite(err), err, torch.full_like(err, math.inf))
        if best is None:
            best, keep = err.clone(), [v.clone() for v in (x, y, zl)]
        better = err < best
        best = torch.where(better, err, best)
        keep = [torch.where(better[..., None], v, k) for v, k in zip((x, y, zl), keep)]
        if bool((best < 1e-13).all()):
            break
        h = zl / x + torch.where(has, zu / w, torch.zeros_like(w))
        if Q is None:
            AD = A / h.unsqueeze(-2)
            M = AD @ T(A)
        else:
            F = torch.linalg.cholesky_ex(Q + torch.diag_embed(h))[0]
            Y = torch.cholesky_solve(T(A).expand(*h.shape[:-1], -1, -1), F)
            M = A @ Y
        d = torch.diagonal(M, dim1=-2, dim2=-1)
        if rows is not None:
            d += (~rows).to(d.dtype)
        L = torch.linalg.cholesky_ex(M + torch.diag_embed(1e-12 * d))[0]

        def hinv(v):
            return v / h if Q is None else torch.cholesky_solve(v.unsqueeze(-1), F).squeeze(-1)

        def solve(r):
            z = torch.cholesky_solve(r.unsqueeze(-1), L).squeeze(-1)
            for _ in range(2):
                z = z + torch.cholesky_solve((r - mv(M, z)).unsqueeze(-1), L).squeeze(-1)
            return z

        def step(cl, cu):
            r1 = -rd + cl / x - torch.where(has, (cu - zu * ru) / w, torch.zeros_like(w))
            dy = solve(rp - mv(A, hinv(r1)))
            dx = hinv(r1 + mv(T(A), dy))
            dw = torch.where(has, ru - dx, torch.zeros_like(w))
            dzl = (cl - zl * dx) / x
            dzu = torch.where(has, (cu - zu * dw) / w, torch.zeros_like(w))
            ap = torch.minimum(_ratio(x, dx), _ratio(w, dw))
            ad = torch.minimum(_ratio(zl, dzl), _ratio(zu, dzu))
            return dx, dy, dw, dzl, dzu, ap, ad

        dx, dy, dw, dzl, dzu, ap, ad = step(-x * zl, -w * zu)
        if Q is not None:
            ap = ad = torch.minimum(ap, ad)
        mua = (((x + ap * dx) * (zl + ad * dzl)).sum(-1, keepdim=True) +
               ((w + ap * dw) * (zu + ad * dzu)).sum(-1, keepdim=True)) / count
        sm = (mua / mu) ** 3 * mu
        dx, dy, dw, dzl, dzu, ap, ad = step(sm - x * zl - dx * dzl, sm - w * zu - dw * dzu)
        if Q is not None:
            ap = ad = torch.minimum(ap, ad)
        ap, ad = (torch.clamp(0.995 * a, max=1.0) for a in (ap, ad))
        x, w, y = x + ap * dx, torch.where(has, w + ap * dw, w), y + ad * dy
        zl, zu = zl + ad * dzl, torch.where(has, zu + ad * dzu, zu)
    return keep


def _ratio(v, dv):
    r = torch.where(dv < 0, -v / torch.where(dv < 0, dv, -torch.ones_like(dv)), torch.full_like(v, 2.0))
    return r.amin(-1, keepdim=True)


def _tensor(a):
    return torch.tensor(np.asarray(a), dtype=torch.float64, device="cuda" if torch.cuda.is_available() else "cpu")


def _exact_lps(models: list[Model], shared: bool):
    """Primal values and row multipliers of every LP, problems of similar size solved together."""
    prim, dual = [None] * len(models), [None] * len(models)
    order = sorted(range(len(models)), key=lambda q: (models[q].m, models[q].n))
    size = 1 if not models else max(1, int(4e8 // max(1, max(m.n * m.m for m in models))))
    for at in range(0, len(order), min(size, 256)):
        part = order[at:at + min(size, 256)]
        forms = [_dense_form(models[q]) for q in part]
        m, n = max(f[0].shape[0] for f in forms), max(f[0].shape[1] for f in forms)
        if shared:
            A = _tensor(forms[0][0]).unsqueeze(0)
        else:
            a = np.zeros((len(part), m, n))
            for q, f in enumerate(forms):
                a[q, :f[0].shape[0], :f[0].shape[1]] = f[0]
            A = _tensor(a)
        pad = lambda k, size, fill: _tensor(  # noqa: E731
            np.stack([np.concatenate([f[k], np.full(size - f[k].size, fill)]) for f in forms]))
        rows = torch.stack([torch.arange(m) < f[0].shape[0] for f in forms]).to(A.device)
        x, y, _ = _interior(A, pad(1, n, 1.0), pad(2, m, 0.0), pad(3, n, np.inf), rows=rows)
        x, y = x.cpu().numpy(), y.cpu().numpy()
        for k, q in enumerate(part):
            prim[q], dual[q] = models[q].lb + x[k, :models[q].n], y[k, :models[q].m]
    return prim, dual


def _exact_qp(mdl: Model):
    A, c, b, u = _dense_form(mdl)
    Q = torch.zeros((A.shape[1], A.shape[1]), dtype=torch.float64, device=_tensor(0.0).device)
    cols = np.repeat(np.arange(mdl.n), np.diff(mdl.q_col_ptr))
    at = (torch.from_numpy(mdl.q_row_idx.astype(np.int64)).to(Q.device), torch.from_numpy(cols).to(Q.device))
    Q.index_put_(at, _tensor(mdl.q_values), accumulate=True)
    Q = 0.5 * (Q + Q.T)
    x, y, z = _interior(_tensor(A)[None], _tensor(c)[None], _tensor(b)[None], _tensor(u)[None], Q=Q[None])
    x, y, z = (v[0].cpu().numpy() for v in (x, y, z))
    n = mdl.n
    return x[:n], y, z[:n], float(mdl.obj @ x[:n] + 0.5 * x[:n] @ (Q[:n, :n].cpu().numpy() @ x[:n]) + mdl.obj_constant)


def _exact_forward(dims, w, x):
    params, at = [], 0
    for a, b in zip(dims[:-1], dims[1:]):
        params.append((_tensor(w[at:at + a * b]).reshape(b, a), _tensor(w[at + a * b:at + a * b + b])))
        at += a * b + b
    acts = [_tensor(x)]
    for k, (W, bias) in enumerate(params):
        v = acts[-1] @ W.T + bias
        acts.append(torch.relu(v) if k + 1 < len(params) else v)
    return params, acts


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "sequence":  # 64 bits do not reach its optimum: the row weights span more than 25 decades
        return None
    if kind == "grad":
        dims, w, x, t = _grad_data(case, seed)
        params, acts = _exact_forward(dims, w, x)
        diff = acts[-1] - _tensor(t)
        g, parts = 2.0 * diff / diff.numel(), []
        for k in reversed(range(len(params))):
            parts = [(g.T @ acts[k]).reshape(-1), g.sum(0)] + parts
            g = (g @ params[k][0]) * (acts[k] > 0)
        return dict(loss=float((diff * diff).mean()), grad=torch.cat(parts))
    if kind == "predict":
        dims, w, p, norm, n, m = _predict_data(case, seed)
        _, acts = _exact_forward(dims, w, (p - norm[0]) / norm[1])
        v = acts[-1] * _tensor(norm[3]) + _tensor(norm[2])
        start = lambda a: torch.clamp(torch.exp(torch.clamp(a, -40.0, 40.0)), min=_DELTA)  # noqa: E731
        return dict(x=start(v[:, :n]), y=v[:, n:n + m], s=start(v[:, n + m:]))
    models = _models(case, seed)
    if kind in ("portfolio", "chain"):
        x, y, z, obj = _exact_qp(models[0])
        return dict(primal=x, dual_row=y, dual_col=z, objective=np.array([obj]), status=None)
    prim, dual = _exact_lps(models, shared=kind == "family")
    out = dict(primal=np.concatenate(prim), status=None,
               objective=np.array([m.obj_constant + m.obj @ x for m, x in zip(models, prim)]))
    if "dual_row" in _OUT[kind]:
        out["dual_row"] = np.concatenate(dual)
    return out
