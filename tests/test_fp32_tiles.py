"""Mixed precision at the edges of its tiles, on well-conditioned matrices where a
tight bound holds: the FP32 tile factor's blocks of 16 and tiles of 64, the work items
of the application, the per-panel schedule's lower updates in tiles of 128 x 64.

Dense blocks: p columns under a border of r, as in the FP64 test; condition below 4.
Grids: the diffusion matrix plus its largest diagonal entry, condition below 3.
Exact factors: the solution's error is the condition number times the rounding errors
of sums of as many terms as the widest supernode has columns, which grow as a random
walk, times 4; with separators compressed at full rank the split products' 1e-5
takes their place.  (A wrong or lost entry is 1e-4 and more.)
"""
import math

import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spla

import rank_structured_cholesky_gb300 as rs
from tests.test_apply_items import FULL, WIDE

pytestmark = pytest.mark.gpu

SIZES = [(1, 0), (15, 1), (16, 0), (16, 16), (17, 15), (31, 33), (32, 32), (33, 31), (47, 1), (48, 17), (49, 16), (63, 65),
         (64, 0), (64, 64), (65, 1), (97, 40), (127, 2), (128, 129), (129, 0), (161, 250)]


def _tol(cond, columns):
    return 4 * cond * math.sqrt(columns) * 2.0 ** -24


@pytest.mark.parametrize("p,r", SIZES)
def test_dense_blocks(p, r):
    rng = np.random.default_rng(100 * p + r)
    n = 2 * p + r
    A = np.zeros((n, n))
    A[:p, :p] = rng.uniform(-1, 1, (p, p))
    A[p:2 * p, p:2 * p] = rng.uniform(-1, 1, (p, p))
    A[2 * p:, :] = rng.uniform(-1, 1, (r, n))
    A = np.tril(A, -1)
    A = A + A.T
    A[np.diag_indices(n)] = 2.0 * np.abs(A).sum(axis=1) + 1.0
    M = sp.csc_matrix(A)
    M.sort_indices()
    F = rs.GpuFactor(rs.Context(precision="mixed", nd_leaf=max(p, r), **WIDE), M.indptr, M.indices, M.data)
    b = rng.standard_normal((3, n))
    want = np.linalg.solve(A, b.T).T
    tol = _tol(4, n) * np.linalg.norm(want)
    assert np.linalg.norm(np.array([F.apply(v) for v in b]) - want) <= tol
    assert np.linalg.norm(F.apply(b) - want) <= tol


def _grid(dims):
    prob = rs.diffusion(3 if dims[2] > 1 else 2, *dims, sigma=0.5, seed=7)
    A = prob.scipy()
    return prob, (A + A.diagonal().max() * sp.identity(prob.n)).tocsc()


def _check_grid(dims, params, tol):
    prob, A = _grid(dims)
    A.sort_indices()
    F = rs.GpuFactor(rs.Context(precision="mixed", **params), A.indptr, A.indices, A.data, prob.xyz)
    b = np.random.default_rng(3).standard_normal((3, prob.n))
    want = spla.splu(A).solve(b.T).T
    assert np.linalg.norm(np.array([F.apply(v) for v in b]) - want) <= tol * np.linalg.norm(want)
    assert np.linalg.norm(F.apply(b) - want) <= tol * np.linalg.norm(want)


@pytest.mark.parametrize("dims", [(17, 16, 1), (33, 31, 1), (65, 64, 1), (130, 129, 1), (13, 11, 12), (24, 24, 25)])
def test_grids(dims):
    _check_grid(dims, WIDE, _tol(3, sorted(dims)[-1] * (sorted(dims)[-2] if dims[2] > 1 else 1)))


@pytest.mark.parametrize("dims", [(90, 83, 1), (18, 17, 19), (25, 24, 26)])
def test_full_ranks(dims):
    _check_grid(dims, FULL, 2e-5 * 3)


def test_lower_updates_in_tall_tiles(monkeypatch, capfd):
    """Per-panel schedule: launches of several tasks, lower triangles, tiles of 128 x 64
    (large fronts; by the residual, which is the error times at most the condition)."""
    monkeypatch.setenv("RSCHOL_FUSED_CHOL", "0")
    monkeypatch.setenv("RSCHOL_PLAN_LOG", "1")
    prob, A = _grid((44, 40, 42))
    A.sort_indices()
    F = rs.GpuFactor(rs.Context(precision="mixed", **WIDE), A.indptr, A.indices, A.data, prob.xyz)
    b = np.random.default_rng(3).standard_normal(prob.n)
    assert np.linalg.norm(b - A @ F.apply(b)) <= 3 * _tol(3, 40 * 42) * np.linalg.norm(b)
    tall = [line.split() for line in capfd.readouterr().err.splitlines()
            if line.startswith("plan gemm") and line.endswith("maxK 64 tc -1")]
    assert any(int(t[t.index("tasks") + 1]) > 1 for t in tall)
