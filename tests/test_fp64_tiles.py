"""FP64 factorisation tiles at their edges: panels and row tiles around the
16-wide blocks and 32-wide tiles, one panel and several, with and without rows
below, and long inner products.

A dense block of p columns under a dense border of r, so that a front of
exactly p + r rows, p of them eliminated, is factored; uncompressed, so one
application is the solution of A x = b.  The matrices have condition number below
4 (diagonally dominant), so the FP64 solve is within 1e-13 n of numpy's.
"""
import numpy as np
import pytest
import scipy.sparse as sp

import rank_structured_cholesky_gb300 as rs

SIZES = [(1, 0), (15, 1), (16, 16), (17, 15), (31, 33), (32, 0), (32, 32), (33, 31), (48, 17), (63, 65), (64, 64),
         (65, 1), (97, 40), (128, 129), (161, 250)]


@pytest.mark.gpu
@pytest.mark.parametrize("p,r", SIZES)
def test_fp64_tiles(p, r):
    rng = np.random.default_rng(100 * p + r)
    n = 2 * p + r   # two blocks of p under the border
    A = np.zeros((n, n))
    A[:p, :p] = rng.uniform(-1, 1, (p, p))
    A[p:2 * p, p:2 * p] = rng.uniform(-1, 1, (p, p))
    A[2 * p:, :] = rng.uniform(-1, 1, (r, n))
    A = np.tril(A, -1)
    A = A + A.T
    A[np.diag_indices(n)] = 2.0 * np.abs(A).sum(axis=1) + 1.0
    M = sp.csc_matrix(A)
    M.sort_indices()
    ctx = rs.Context(precision="fp64", max_dense_block=10 ** 6, max_diag_block=10 ** 6, nd_leaf=max(p, r))
    F = rs.GpuFactor(ctx, M.indptr.astype(np.int32), M.indices.astype(np.int32), M.data)
    b = rng.standard_normal(n)
    want = np.linalg.solve(A, b)
    assert np.linalg.norm(F.apply(b) - want) <= 1e-13 * n * np.linalg.norm(want)
