"""Sparse factor and solves: which form a matrix takes (host), and the two forms against each other and
against the dense factor (GPU)."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from sovereign_b200 import problems as P
from sovereign_b200.ipm import InteriorPointOptions, InteriorPointSolver, QpInteriorPointSolver

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_form_by_columns_levels_terms_and_entries(tmp_path):
    exe = tmp_path / "sparse_walk_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(ROOT, "sovereign_b200", "csrc"),
                    os.path.join(ROOT, "tests", "sparse_walk_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and "failures 0" in r.stdout, r.stdout + r.stderr


def joined_rows(m, block, arm, seed):
    """An LP of m equality rows, one single entry each, neighbouring rows of a block joined by columns of two
    entries; with `arm` the last row is joined to every other (a row of L of m - 1 entries, cut into pieces)."""
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


def by_form(solve, monkeypatch):
    out = []
    for form in ("grid", "cta"):
        monkeypatch.setenv("SOVEREIGN_SPARSE_WALK", form)
        out.append(solve())
        monkeypatch.delenv("SOVEREIGN_SPARSE_WALK")
    return out


# one level; a row per thread, one more, and several rounds of them; short and long chains; long rows
@pytest.mark.gpu
@pytest.mark.parametrize("m,block,arm", [(1, 1, False), (33, 4, False), (33, 33, True), (1023, 1, False), (1024, 2, False),
                                         (1025, 3, True), (3000, 40, False), (3000, 3, True), (9000, 1, False),
                                         (28000, 2, False), (30000, 2, False)])
def test_forms_give_the_same_bits_on_lps(m, block, arm, monkeypatch):
    mdl = joined_rows(m, block, arm, m + block)
    monkeypatch.setenv("SOVEREIGN_IPM_NORMAL_EQUATIONS", "sparse")
    grid, cta = by_form(lambda: InteriorPointSolver().solve(mdl, with_ipm=True), monkeypatch)
    auto = InteriorPointSolver().solve(mdl, with_ipm=True)
    assert grid.status_name == "OPTIMAL" and "sparse LDL^T" in grid.message, grid.message
    for r in (cta, auto):
        assert r.iterations == grid.iterations and r.objective_value == grid.objective_value
        assert np.array_equal(r.primal, grid.primal) and np.array_equal(r.ipm_y, grid.ipm_y)
    if m <= 3000:  # the dense factor: another order of sums, within the stopping tolerance of 1e-9
        monkeypatch.setenv("SOVEREIGN_IPM_NORMAL_EQUATIONS", "dense")
        dense = InteriorPointSolver().solve(mdl)
        assert dense.status_name == "OPTIMAL" and "dense Cholesky" in dense.message
        assert abs(dense.objective_value - grid.objective_value) <= 1e-9 * abs(dense.objective_value)


@pytest.mark.gpu
@pytest.mark.parametrize("limit", [4, 250])
def test_forms_give_the_same_bits_on_a_grid_network(limit, monkeypatch):
    mdl = P.grid_network_lp(30)
    monkeypatch.setenv("SOVEREIGN_IPM_NORMAL_EQUATIONS", "sparse")
    grid, cta = by_form(lambda: InteriorPointSolver(InteriorPointOptions(max_iterations=limit)).solve(mdl), monkeypatch)
    assert grid.iterations == cta.iterations and np.array_equal(grid.primal, cta.primal)
    assert grid.objective_value == cta.objective_value and np.array_equal(grid.dual_row, cta.dual_row)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [40, 700, 2000])
def test_forms_give_the_same_bits_on_quasi_definite_systems(n, monkeypatch):
    mdl = P.coupled_chain_qp(n, 3)
    monkeypatch.setenv("SOVEREIGN_QP_KKT", "sparse")
    grid, cta = by_form(lambda: QpInteriorPointSolver().solve(mdl), monkeypatch)
    assert grid.status_name == "OPTIMAL" and "quasi-definite" in grid.message, grid.message
    assert grid.iterations == cta.iterations and grid.objective_value == cta.objective_value
    assert np.array_equal(grid.primal, cta.primal)
