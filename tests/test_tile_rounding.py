"""The first column of a factor, whose entries are a square root and divisions and
nothing else: correctly rounded in either precision, as LAPACK's unblocked Cholesky
has them (in FP32 in the first block of 16 rows; further down the entries are products
with the block's inverse)."""
import numpy as np
import pytest
import scipy.sparse as sp

import rank_structured_cholesky_gb300 as rs


@pytest.mark.gpu
@pytest.mark.parametrize("precision,rows", [("fp64", 32), ("mixed", 16)])
@pytest.mark.parametrize("n", [2, 9, 16, 32])
def test_first_column(n, precision, rows):
    rng = np.random.default_rng(n)
    for _ in range(8):
        A = np.tril(rng.uniform(-1, 1, (n, n)), -1)
        A = A + A.T
        A[np.diag_indices(n)] = 2.0 * np.abs(A).sum(axis=1) + 1.0
        ft = np.float64 if precision == "fp64" else np.float32
        A = A.astype(ft)
        M = sp.csc_matrix(A.astype(np.float64))
        M.sort_indices()
        ctx = rs.Context(precision=precision, max_dense_block=10 ** 6, max_diag_block=10 ** 6, nd_leaf=n)
        F = rs.GpuFactor(ctx, M.indptr, M.indices, M.data)
        assert F.num_nodes() == 1
        B = A[np.ix_(F.perm(), F.perm())]
        d = np.sqrt(B[0, 0])
        want = np.concatenate([[d], B[1:, 0] / d])
        assert np.array_equal(F.node_l11(0)[:rows, 0].astype(ft), want[:rows])
