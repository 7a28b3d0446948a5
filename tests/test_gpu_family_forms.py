"""GPU: the family path's solves with a CTA per LP against the grid's form, bit for bit: with and without a
dense block, fewer LPs than a launch's slots, more than one launch, long rows cut into pieces, and an order
that only the grid's form takes."""
import dataclasses

import numpy as np
import pytest

from sovereign_b200 import problems as P
from sovereign_b200.ipm import InteriorPointOptions, InteriorPointSolver, solve_family

pytestmark = pytest.mark.gpu


def joined_rows(m, block, arm, seed):
    """m equality rows, one single entry each, neighbouring rows of a block joined by columns of two entries;
    with `arm` the last row is joined to every other (a row of L of m - 1 entries)."""
    g = np.random.default_rng(seed)
    links = [(i, i + 1) for i in range(m - 1) if (i + 1) % block]
    links += [(i, m - 1) for i in range(m - 2)] if arm else []
    n = m + len(links)
    cols = np.concatenate([np.arange(m), np.repeat(np.arange(m, n), 2)])
    rows = np.concatenate([np.arange(m), np.array(links, int).ravel()]).astype(np.int32)
    vals = g.uniform(0.5, 1.5, rows.size)
    rhs = np.bincount(rows, weights=vals * g.uniform(0.5, 2.0, n)[cols], minlength=m)
    return P.Model(n=n, m=m, col_ptr=np.concatenate([[0], np.cumsum(np.bincount(cols, minlength=n))]).astype(np.int32),
                   row_idx=rows, values=vals, obj=g.uniform(0.5, 2.0, n), rhs=rhs, sense=np.full(m, 2, np.int8),
                   lb=np.zeros(n), ub=np.full(n, P.INF))


def around(mdl, count):
    g = np.random.default_rng(count)
    return [dataclasses.replace(mdl, obj=mdl.obj * g.uniform(0.9, 1.1, mdl.n), _keep=[]) for _ in range(count)]


def instances(fam, count):
    return [fam.instance_from_seed(40 + k)[0] for k in range(count)]


@pytest.mark.parametrize("make", [
    lambda: instances(P.MulticommodityFamily(nodes=200, arcs=1000), 3),
    lambda: instances(P.MulticommodityFamily(nodes=60, arcs=300), 67),
    lambda: instances(P.TransportFamily(), 5),               # the dense block is nearly all of it
    lambda: around(P.grid_network_lp(20), 2),
    lambda: around(joined_rows(1, 1, False, 1), 2),
    lambda: around(joined_rows(513, 4, False, 2), 33),       # a row more than the CTA has threads
    lambda: around(joined_rows(1500, 3, True, 3), 2),
    lambda: around(joined_rows(14000, 8, False, 4), 2),
])
def test_solves_of_both_forms_give_the_same_bits(make, monkeypatch):
    models, out = make(), []
    for form in ("grid", "cta", ""):
        if form:
            monkeypatch.setenv("SOVEREIGN_FAMILY_SOLVE", form)
        else:
            monkeypatch.delenv("SOVEREIGN_FAMILY_SOLVE")
        out.append(solve_family(models, InteriorPointOptions(max_iterations=30), with_ipm=True))
    for grid, cta, auto in zip(*out):
        assert grid.status_name == "OPTIMAL", grid.message
        for r in (cta, auto):
            assert r.iterations == grid.iterations and r.objective_value == grid.objective_value
            assert np.array_equal(r.primal, grid.primal) and np.array_equal(r.ipm_y, grid.ipm_y)


def test_order_beyond_the_shared_memory_of_a_cta():
    models = around(joined_rows(15000, 60, False, 5), 2)
    for mdl, r in zip(models, solve_family(models)):
        single = InteriorPointSolver().solve(mdl)
        assert r.status_name == single.status_name == "OPTIMAL", (r.message, single.message)
        # the same iteration, another order of sums: within the stopping tolerance of 1e-9
        assert abs(r.objective_value - single.objective_value) <= 2e-9 * abs(single.objective_value)
