"""GPU: the batched kernel at orders around the edges of its 8-column blocks and 32-row groups, at
every CTA width, with dependent rows among them, against the oracle."""
import concurrent.futures as cf

import numpy as np
import pytest

import oracle
from sovereign_b200 import problems as P
from sovereign_b200.ipm import InteriorPointOptions, InteriorPointSolver, autotune, solve_batch

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


def both_routes(mdl, monkeypatch, warm=None, **options):
    """sov_lp_solve by size (one CTA) and through the general engine (a factorization asked for)."""
    solver = InteriorPointSolver(InteriorPointOptions(**options))
    auto = solver.solve(mdl, with_ipm=True, warm_start=warm)
    monkeypatch.setenv("SOVEREIGN_IPM_NORMAL_EQUATIONS", "dense")
    general = InteriorPointSolver(InteriorPointOptions(**options)).solve(mdl, with_ipm=True, warm_start=warm)
    monkeypatch.delenv("SOVEREIGN_IPM_NORMAL_EQUATIONS")
    return auto, general


def scaled_bounds(mdl):
    """Nonzero lower bounds and finite upper bounds on some columns (bound rows), a constant, maximize."""
    mdl.lb = np.where(np.arange(mdl.n) % 4 == 0, 0.05, 0.0)
    mdl.ub = np.where(np.arange(mdl.n) % 3 == 0, 300.0, P.INF)
    mdl.obj, mdl.maximize, mdl.obj_constant = -mdl.obj, True, 2.5
    return mdl


@pytest.mark.parametrize("make,batched", [
    (lambda: P.bounded_lp_example(), False),                       # two rows share two columns
    (lambda: P.transport(5, 6, 1), True),
    (lambda: P.transport(64, 64, 2), True),
    (lambda: P.transport(64, 65, 2), False),                       # 129 rows
    (lambda: scaled_bounds(P.transport(8, 9, 5)), True),           # 17 + 24 IPM rows
    (lambda: scaled_bounds(P.transport(20, 20, 6)), False),        # 40 + 134 IPM rows
    (lambda: scaled_bounds(P.random_sparse_lp(30, 90, 4, 5)), False),
    (lambda: P.random_sparse_lp(100, 300, 1, 7), True),            # no off-diagonal entries at all
])
def test_single_solve_routes_agree(make, batched, monkeypatch):
    auto, general = both_routes(make(), monkeypatch)
    assert ("batched" in auto.message) == batched and "dense Cholesky" in general.message
    assert auto.status_name == general.status_name == "OPTIMAL"
    assert auto.iterations == general.iterations and (auto.n_ipm, auto.m_ipm) == (general.n_ipm, general.m_ipm)
    # the same iteration in another order of summation: within the stopping tolerance of 1e-9
    assert abs(auto.objective_value - general.objective_value) <= 1e-9 * max(1.0, abs(general.objective_value))
    assert np.linalg.norm(auto.primal - general.primal) <= 1e-8 * max(1.0, np.linalg.norm(general.primal))
    assert np.linalg.norm(auto.ipm_x - general.ipm_x) <= 1e-8 * max(1.0, np.linalg.norm(general.ipm_x))


def test_single_solve_routes_agree_when_stopped_early_or_warm_started(monkeypatch):
    mdl = P.transport(9, 11, 4)
    auto, general = both_routes(mdl, monkeypatch, max_iterations=4)
    assert auto.status_name == general.status_name != "OPTIMAL"
    assert auto.iterations == general.iterations and auto.message == general.message
    start = InteriorPointSolver(InteriorPointOptions(ipm_iterate_at=6)).solve(mdl, with_ipm=True)
    assert "batched" not in start.message  # an iterate on the way: the general engine
    auto, general = both_routes(mdl, monkeypatch, warm=(start.ipm_x, start.ipm_y, start.ipm_s))
    assert "batched" in auto.message and auto.status_name == general.status_name == "OPTIMAL"
    assert auto.iterations == general.iterations < InteriorPointSolver().solve(mdl).iterations
    # two calls give the same bits
    first, second = (InteriorPointSolver().solve(P.transport(31, 29, 8)) for _ in range(2))
    assert first.objective_value == second.objective_value and np.array_equal(first.primal, second.primal)
    # infeasible bounds are refused with the general path's message
    bad = P.transport(3, 3, 1)
    bad.lb, bad.ub = np.full(9, 2.0), np.full(9, 1.0)
    auto, general = both_routes(bad, monkeypatch)
    assert auto.status_name == general.status_name and auto.message == general.message


@pytest.mark.parametrize("make,count", [(lambda s: P.transport(18, 18, s), 3072), (lambda s: P.transport(18, 18, s), 500),
                                        (lambda s: P.transport(30, 12 + s % 9, s), 700)])
def test_parts_give_the_bits_of_one_batch(make, count, monkeypatch):
    # each normal-matrix entry has one term here, so an LP's bits depend on its CTA width alone, and that on
    # the call, not on the part an LP is in
    pool = [make(s) for s in range(40)]
    models = [pool[k % 40] for k in range(count)]
    monkeypatch.setenv("SOVEREIGN_BATCH_PARTS", "1")
    one = solve_batch(models)
    monkeypatch.setenv("SOVEREIGN_BATCH_PARTS", "7")
    parts = solve_batch(models)
    monkeypatch.delenv("SOVEREIGN_BATCH_PARTS")
    auto = solve_batch(models)
    for a, b, c in zip(one, parts, auto):
        assert a.status_name == "OPTIMAL"
        assert a.objective_value == b.objective_value == c.objective_value
        assert np.array_equal(a.primal, b.primal) and np.array_equal(a.primal, c.primal)


def test_an_autotune_leaves_other_batch_sizes_and_single_solves_alone():
    one, few = P.transport(50, 50, 1), P.transport_batch(24, seed=3)
    before = [InteriorPointSolver().solve(one)] + solve_batch(few)
    autotune(P.transport_batch(700, seed=5))
    after = [InteriorPointSolver().solve(one)] + solve_batch(few)
    autotune(few)  # one LP per SM or less: the single solve's own class
    after.append(InteriorPointSolver().solve(one))
    for a, b in zip(before + before[:1], after):
        assert a.objective_value == b.objective_value and np.array_equal(a.primal, b.primal)


def test_single_solves_from_several_threads_give_the_bits_of_one():
    models = [P.transport(12 + k % 5, 9 + k % 7, k) for k in range(48)] + [P.transport(3, 4, k) for k in range(16)]
    alone = [InteriorPointSolver().solve(mdl) for mdl in models]
    with cf.ThreadPoolExecutor(max_workers=8) as ex:
        together = list(ex.map(InteriorPointSolver().solve, models))
    for a, b in zip(alone, together):
        assert "batched" in a.message and a.status_name == "OPTIMAL"
        assert a.objective_value == b.objective_value and a.iterations == b.iterations
        assert np.array_equal(a.primal, b.primal) and np.array_equal(a.dual_row, b.dual_row)


def complete(m, singles, seed):
    """Every pair of m rows shares one column; `singles` columns of one entry beyond them."""
    g = np.random.default_rng(seed)
    i, j = np.tril_indices(m, -1)
    cols = np.concatenate([np.repeat(np.arange(i.size), 2), np.arange(i.size, i.size + singles)])
    rows = np.concatenate([np.stack([j, i], 1).ravel(), g.integers(0, m, singles)]).astype(np.int32)
    vals, n = g.uniform(0.5, 1.5, cols.size), i.size + singles
    rhs = np.bincount(rows, weights=vals * g.uniform(0.5, 2.0, n)[cols], minlength=m)
    return P.Model(n=n, m=m, col_ptr=np.concatenate([[0], np.cumsum(np.bincount(cols, minlength=n))]).astype(np.int32),
                   row_idx=rows, values=vals, obj=g.uniform(0.5, 2.0, n), rhs=rhs, sense=np.full(m, 2, np.int8),
                   lb=np.zeros(n), ub=np.full(n, P.INF))


@pytest.mark.parametrize("m,singles,batched", [(128, 10000, True), (128, 30000, False), (32, 60000, True)])
def test_single_solve_route_by_rows_and_entries(m, singles, batched, monkeypatch):
    # either side of the line beyond which one SM streams the columns slower than the whole GPU
    auto, general = both_routes(complete(m, singles, 3), monkeypatch)
    assert ("batched" in auto.message) == batched and "batched" not in general.message
    assert auto.status_name == general.status_name == "OPTIMAL" and auto.iterations == general.iterations
    assert abs(auto.objective_value - general.objective_value) <= 1e-9 * abs(general.objective_value)


def test_batch_matches_the_general_engine():
    # with diagnostics a single solve takes the general engine, so two codes are compared (a solve without
    # them would be a batch of one)
    models = P.transport_batch(8, seed=9) + [P.transport(64, 64, 2), P.random_sparse_lp(40, 90, 3, 4)]
    for limit in (250, 5):
        options = InteriorPointOptions(max_iterations=limit)
        for mdl, b in zip(models, solve_batch(models, options)):
            s = InteriorPointSolver(options).solve(mdl, with_diag=True)
            assert "batched" not in s.message and s.diagnostics["history_iterations"][:2] == [1, 2]
            assert b.status_name == s.status_name and b.iterations == s.iterations
            # the same iteration, another order of sums; both stop at a relative gap of 1e-9
            assert abs(b.objective_value - s.objective_value) <= 1e-9 * abs(s.objective_value)
            assert np.linalg.norm(b.primal - s.primal) <= 1e-6 * np.linalg.norm(s.primal)
