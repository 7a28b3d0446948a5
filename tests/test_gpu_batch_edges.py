"""GPU: the batched kernel at orders around the edges of its 8-column blocks and 32-row groups, at
every CTA width, with dependent rows among them, against the oracle."""
import numpy as np
import pytest

import oracle
from sovereign_b200 import problems as P
from sovereign_b200.ipm import solve_batch

pytestmark = pytest.mark.gpu

ORDERS = [1, 2, 7, 8, 9, 15, 16, 17, 31, 32, 33, 40, 63, 64, 65, 96, 97, 120, 127, 128]


def with_copy(mdl):
    """The LP with its last row repeated (a dependent row)."""
    last = mdl.m - 1
    cols, vals, ptr = [], [], [0]
    for j in range(mdl.n):
        r, v = mdl.row_idx[mdl.col_ptr[j]:mdl.col_ptr[j + 1]], mdl.values[mdl.col_ptr[j]:mdl.col_ptr[j + 1]]
        extra = v[r == last]
        cols.append(np.concatenate([r, np.full(extra.size, mdl.m)]))
        vals.append(np.concatenate([v, extra]))
        ptr.append(ptr[-1] + cols[-1].size)
    mdl.col_ptr, mdl.row_idx = np.array(ptr, np.int32), np.concatenate(cols).astype(np.int32)
    mdl.values, mdl.m = np.concatenate(vals), mdl.m + 1
    mdl.rhs = np.append(mdl.rhs, mdl.rhs[-1])
    mdl.sense = np.append(mdl.sense, mdl.sense[-1]).astype(np.int8)
    return mdl


@pytest.mark.parametrize("width", ["", "128", "129", "256", "257", "512"])
def test_orders_match_oracle(width, monkeypatch):
    if width:
        monkeypatch.setenv("SOVEREIGN_BATCH_THREADS", width)
    models = [P.random_sparse_lp(m, 3 * m + 5, min(m, 4), 50 + m) for m in ORDERS]
    models += [P.transport(a, b, 3) for a, b in ((2, 3), (4, 4), (30, 34), (60, 60), (64, 64))]
    # a repeated row changes nothing (and the oracle's dense factor does not take one): the oracle solves
    # the LP without it
    pairs = [(mdl, mdl) for mdl in models]
    pairs += [(with_copy(P.random_sparse_lp(*a)), P.random_sparse_lp(*a))
              for a in ((m, 3 * m + 5, min(m, 4), 90 + m) for m in (7, 8, 31, 64, 100, 127))]
    for (mdl, plain), r in zip(pairs, solve_batch([p[0] for p in pairs])):
        ref = oracle.solve(plain, kind="restatement")
        assert r.status_name == ref.status_name == "OPTIMAL", (mdl.name, r.message, ref.message)
        # both stop at a relative gap of 1e-9
        assert abs(r.objective_value - ref.objective_value) <= 1e-8 * max(1.0, abs(ref.objective_value)), mdl.name
