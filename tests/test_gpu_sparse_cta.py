"""GPU: the sparse factor and solves on one CTA against the oracle's dense factor, on matrices that
the rules send there and on one whose right-hand side does not fit its shared memory: leaves only, one
level, long rows that are cut into pieces, and more columns in a level than the CTA has threads."""
import numpy as np
import pytest

from sovereign_b200 import abi
from sovereign_b200.ipm import normal_factor_solve

pytestmark = pytest.mark.gpu


def arrow(m, arms, extra, seed):
    """m x n: one entry per row, `extra` columns that join neighbouring rows, `arms` columns that join
    row m - 1 to every row (a long last row of L)."""
    rng = np.random.default_rng(seed)
    cols = [[(i, 1.0 + rng.random())] for i in range(m)]
    cols += [[(i, rng.standard_normal()), (i + 1, rng.standard_normal())] for i in rng.integers(0, max(1, m - 1), extra)
             if i + 1 < m]
    if arms:
        cols += [[(i, rng.standard_normal()), (m - 1, rng.standard_normal())] for i in range(0, m - 1)]
    ptr = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.int32)
    idx = np.array([r for c in cols for r, _ in c], dtype=np.int32)
    val = np.array([v for c in cols for _, v in c])
    return len(cols), ptr, idx, val


@pytest.mark.parametrize("m,arms,extra", [(1, 0, 0), (5, 0, 3), (33, 1, 10), (1025, 0, 900), (1500, 1, 1400),
                                          (5000, 1, 2500), (29500, 0, 20000)])
def test_sparse_solve_matches_normal_equations(m, arms, extra):
    n, ptr, idx, val = arrow(m, arms, extra, m + arms)
    rng = np.random.default_rng(m)
    d = rng.uniform(0.5, 2.0, n)
    rhs = rng.standard_normal((m, 2))
    z, dropped = normal_factor_solve(m, n, ptr, idx, val, d, rhs, factorization=abi.FACTOR_SPARSE)
    assert dropped == 0
    # M z = A (d * (A' z)) + 1e-12 z: the residual of a backward stable solve is a small multiple of
    # 2^-53 |M| |z|, and |M|_inf |z| bounds the longest row's sum (5000 terms of size below 100)
    cols = np.repeat(np.arange(n), np.diff(ptr))
    for q in range(2):
        at = np.bincount(cols, weights=val * z[idx, q], minlength=n)
        r = np.bincount(idx, weights=val * (d * at)[cols], minlength=m) + 1e-12 * z[:, q] - rhs[:, q]
        absm = np.bincount(idx, weights=np.abs(val) * (d * np.bincount(cols, weights=np.abs(val * z[idx, q]),
                                                                      minlength=n))[cols], minlength=m)
        assert np.all(np.abs(r) <= 1e-12 * (absm + np.abs(rhs[:, q])) + 1e-12 * np.abs(rhs).max())
