"""Blocks of right-hand sides at the widths and chunk heights where a pass over
them changes: 1, 2 and 4 vectors of columns and remainders, chunks of few rows (K
split over threads) and of many, sums of many partial rows.  And the SpMV at the
row lengths where its threads per row change.

Exact factors: an application is the direct solve, to the tolerances of the
single-vector test (FP64 1e-10; mixed 2e-5 times the grid's condition number).
"""
import math

import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spla

import rank_structured_cholesky_gb300 as rs

pytestmark = pytest.mark.gpu
WIDE = dict(max_dense_block=10 ** 6, max_diag_block=10 ** 6)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("k", [2, 5, 8, 17, 33, 64])
def test_block_is_the_direct_solve(k, precision):
    prob = rs.diffusion(3, 21, 20, 19, sigma=0.5, seed=7)   # separators of up to 400 columns
    F = rs.GpuFactor(rs.Context(precision=precision, **WIDE), prob.colptr, prob.rowind, prob.vals, prob.xyz)
    b = np.random.default_rng(k).standard_normal((k, prob.n))
    want = spla.splu(prob.scipy().tocsc()).solve(b.T).T
    tol = 1e-10 if precision == "fp64" else 2e-5 * 4 * 22 ** 2 / math.pi ** 2
    x = F.apply(b)
    err = np.linalg.norm(x - want, axis=1) / np.linalg.norm(want, axis=1)
    assert err.max() <= tol
    assert np.array_equal(x, F.apply(b))
    assert np.array_equal(x[:2], F.apply(b[:2]))   # a column's sums do not depend on the block's width


@pytest.mark.parametrize("n,width", [(50, 3), (700, 12), (700, 13), (5000, 40), (90000, 20)])
def test_spmv_rows(n, width):
    """The true residual that PCG reports is one SpMV: against scipy's."""
    rng = np.random.default_rng(n + width)
    offs = np.unique(rng.integers(1, min(n, 4 * width), width // 2))
    A = sp.diags([rng.uniform(-1, 0, n - o) for o in offs], [-int(o) for o in offs], shape=(n, n)).tocsc()
    A = A + A.T
    A = (A + sp.diags(np.asarray(abs(A).sum(axis=1)).ravel() + 1.0)).tocsc()
    A.sort_indices()
    G = rs.GpuFactor(rs.Context(precision="fp64"), A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data)
    b = rng.standard_normal(n)
    x, info = G.pcg(b, 1e-3, 1)
    r = np.linalg.norm(b - A @ x) / np.linalg.norm(b)
    # both residuals carry the rounding of a row's sum: 4 width eps |A| |x| / |b|
    slack = 4 * width * 2.0 ** -52 * np.linalg.norm(abs(A) @ abs(x)) / np.linalg.norm(b)
    assert abs(info["true_residual"] - r) <= 1e-10 * r + slack
