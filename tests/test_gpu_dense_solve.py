"""GPU: dense factor and dataflow triangular solves at the edges of their 64-row blocks, up to more blocks
than CTAs, several right-hand sides through the same hand-over buffers."""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg

from sovereign_b200 import abi, problems as P
from sovereign_b200.ipm import normal_factor_solve

pytestmark = pytest.mark.gpu


EDGES = [1, 63, 64, 65, 128, 129, 193, 257]


# 9537 rows are 150 blocks; at that size this matrix is singular to FP32 (a pivot is dropped)
@pytest.mark.parametrize("m,precision,bound", [(m, abi.PRECISION_FP64, 1e-12) for m in EDGES + [9537]]
                         + [(m, abi.PRECISION_MIXED, 1e-4) for m in EDGES])
def test_factor_and_solves_at_block_edges(m, precision, bound):
    n = 2 * m + 3
    mdl = P.random_sparse_lp(m, n, min(3, m), 7 + m)
    rng = np.random.default_rng(m)
    d = rng.uniform(0.5, 2.0, n)
    rhs = rng.standard_normal((m, 3))
    z, dropped = normal_factor_solve(m, n, mdl.col_ptr, mdl.row_idx, mdl.values, d, rhs, precision=precision)
    A = sp.csc_matrix((mdl.values, mdl.row_idx, mdl.col_ptr), shape=(m, n))
    N = A @ sp.diags(d) @ A.T
    assert dropped == 0
    # backward error: order x unit roundoff (9537 x 1.1e-16, 9537 x 6e-8 at worst, sums of random signs far less)
    scale = sp.linalg.norm(N) * np.linalg.norm(z, axis=0) + np.linalg.norm(rhs, axis=0)
    assert np.all(np.linalg.norm(N @ z - rhs, axis=0) <= bound * scale)
