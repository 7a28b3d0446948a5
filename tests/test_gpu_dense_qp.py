"""GPU: coupled-Hessian QPs on the dense path (H factored, its forward substitution over all rows of
A at once) against the sparse KKT path, at orders and row counts around the edges of the tiles."""
import os

import numpy as np
import pytest

from sovereign_b200 import abi
from sovereign_b200.ipm import QpInteriorPointOptions, QpInteriorPointSolver
from sovereign_b200.model import Model
from sovereign_b200.problems import INF

pytestmark = pytest.mark.gpu


def coupled_qp(n, m, seed):
    """Q = B B' + diag (sparse B), m rows (<= and =) that x0 >= 0 satisfies, x >= 0."""
    rng = np.random.default_rng(seed)
    b = np.where(rng.random((n, n)) < min(1.0, 3.0 / n), rng.standard_normal((n, n)), 0.0)
    Q = b @ b.T + np.diag(rng.uniform(0.5, 2.0, n))
    A = np.where(rng.random((m, n)) < 0.4, rng.standard_normal((m, n)), 0.0)
    A[np.arange(m), rng.integers(0, n, m)] = 1.0
    x0 = rng.uniform(0.1, 1.0, n)
    sense = np.array([abi.EQ if i % 3 == 0 and i < n // 2 else abi.LE for i in range(m)], dtype=np.int8)
    rhs = A @ x0 + np.where(sense == abi.LE, rng.uniform(0.0, 0.5, m), 0.0)

    def csc(M):
        cols = [np.flatnonzero(M[:, j]) for j in range(M.shape[1])]
        ptr = np.concatenate([[0], np.cumsum([c.size for c in cols])]).astype(np.int32)
        return ptr, np.concatenate(cols).astype(np.int32), np.concatenate([M[c, j] for j, c in enumerate(cols)])

    ap, ai, av = csc(A)
    mdl = Model(n=n, m=m, col_ptr=ap, row_idx=ai, values=av, obj=rng.standard_normal(n), rhs=rhs, sense=sense,
                lb=np.zeros(n), ub=np.full(n, INF))
    mdl.q_col_ptr, mdl.q_row_idx, mdl.q_values = csc(Q)
    return mdl


@pytest.mark.parametrize("n,m", [(2, 1), (40, 31), (40, 32), (64, 33), (63, 1), (65, 4), (129, 65), (200, 5),
                                 (300, 97), (448, 130)])
def test_dense_hessian_path_matches_kkt_path(n, m, monkeypatch):
    mdl = coupled_qp(n, m, 100 * n + m)
    opt = QpInteriorPointOptions()
    opt.optimality_tol = opt.feasibility_tol = 1e-9
    dense = QpInteriorPointSolver(opt).solve(mdl)
    assert dense.status_name == "OPTIMAL" and "H %d" % dense.n_ipm in dense.message, dense.message
    monkeypatch.setenv("SOVEREIGN_QP_KKT", "sparse")
    kkt = QpInteriorPointSolver(opt).solve(mdl)
    assert kkt.status_name == "OPTIMAL" and "quasi-definite" in kkt.message, kkt.message
    # both stop at 1e-9 relative; Q's smallest eigenvalue is at least 0.5
    assert abs(dense.objective_value - kkt.objective_value) <= 1e-8 * max(1.0, abs(kkt.objective_value))
    assert np.linalg.norm(dense.primal - kkt.primal) <= 1e-4 * max(1.0, np.linalg.norm(kkt.primal))
