"""GPU: the double-double band QP path's odd-even reduction against elimination in the natural order
(SOVEREIGN_XBAND_SEGMENTS=1) and against the optimality conditions, for every half-bandwidth and at
block counts around the edges of its levels."""
import numpy as np
import pytest

from sovereign_b200 import abi
from sovereign_b200.ipm import QpInteriorPointSolver
from sovereign_b200.model import Model
from sovereign_b200.problems import INF

pytestmark = pytest.mark.gpu


def band_qp(n, kd, seed):
    rng = np.random.default_rng(seed)
    m = n - kd
    a = rng.standard_normal((m, kd + 1))
    x0 = rng.standard_normal(n)
    sense = rng.choice(np.array([abi.GE, abi.LE], dtype=np.int8), m)
    idx = np.arange(m)[:, None] + np.arange(kd + 1)[None, :]
    act = (a * x0[idx]).sum(axis=1)
    rhs = act - np.where(sense == abi.GE, 1.0, -1.0) * rng.uniform(0.0, 0.5, m)
    cols, rows, vals = idx.reshape(-1), np.repeat(np.arange(m), kd + 1), a.reshape(-1)
    order = np.lexsort((rows, cols))
    ptr = np.concatenate([[0], np.cumsum(np.bincount(cols, minlength=n))]).astype(np.int32)
    q = rng.uniform(0.5, 2.0, n)
    mdl = Model(n=n, m=m, col_ptr=ptr, row_idx=rows[order].astype(np.int32), values=np.ascontiguousarray(vals[order]),
                obj=rng.standard_normal(n) * 3.0, rhs=rhs, sense=sense, lb=np.full(n, -INF), ub=np.full(n, INF))
    mdl.q_col_ptr, mdl.q_row_idx, mdl.q_values = np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32), q
    return mdl, a, idx, q


@pytest.mark.parametrize("kd", [1, 2, 3, 4])
@pytest.mark.parametrize("blocks,extra", [(1, 1), (2, 0), (2, 1), (5, 0), (512, 0), (513, 1), (1101, 0)])
def test_odd_even_reduction_matches_natural_order(kd, blocks, extra, monkeypatch):
    n = max(kd + 1, blocks * kd + min(extra, kd - 1))
    mdl, a, idx, q = band_qp(n, kd, 10 * kd + blocks)
    r = QpInteriorPointSolver().solve(mdl)
    assert r.status_name == "OPTIMAL" and "double-double" in r.message, r.message
    # the path stops at 1e-10 on its residuals and relative gap, each in its own scale
    grad = q * r.primal + mdl.obj
    atz = np.zeros(n)
    np.add.at(atz, idx.reshape(-1), (a * r.dual_row[:, None]).reshape(-1))
    scale = max(1.0, np.abs(mdl.obj).max() + np.abs(q * r.primal).max())
    assert np.abs(grad - atz).max() <= 1e-9 * scale
    slack = ((a * r.primal[idx]).sum(axis=1) - mdl.rhs) * np.where(mdl.sense == abi.GE, 1.0, -1.0)
    assert slack.min() >= -1e-9 * max(1.0, np.abs(mdl.rhs).max())
    assert np.abs(slack @ np.abs(r.dual_row)) <= 1e-9 * (1.0 + abs(r.objective_value)) * 10
    monkeypatch.setenv("SOVEREIGN_XBAND_SEGMENTS", "1")
    nat = QpInteriorPointSolver().solve(mdl)
    assert nat.status_name == "OPTIMAL" and nat.iterations == r.iterations
    assert np.linalg.norm(r.primal - nat.primal) <= 1e-11 * np.linalg.norm(nat.primal)
    assert np.linalg.norm(r.dual_row - nat.dual_row) <= 1e-11 * np.linalg.norm(nat.dual_row)


@pytest.mark.parametrize("n", [1023, 1024, 1025])
def test_cluster_sizes_agree_with_natural_order_at_their_line(n, monkeypatch):
    mdl = band_qp(n, 2, n)[0]
    r = QpInteriorPointSolver().solve(mdl)
    monkeypatch.setenv("SOVEREIGN_XBAND_SEGMENTS", "1")
    nat = QpInteriorPointSolver().solve(mdl)
    assert r.status_name == nat.status_name == "OPTIMAL" and nat.iterations == r.iterations
    assert np.linalg.norm(r.primal - nat.primal) <= 1e-11 * np.linalg.norm(nat.primal)
