"""The preconditioner application's work items at their edges: group members
and chunks around 16 / 32 / 64 columns, chunks of several row counts, supernodes
and ranks too wide for a stage, tiles of X with remainders.

Every case is an exact factor (no compression, or full ranks), so one
application is the solution of A x = b, checked against scipy's direct solver.
Tolerances: FP64 1e-10 (condition number below 1e4, n eps growth); mixed: the
split products' 1e-5 times the condition number 4 (N + 1)^2 / pi^2 of the grid's
longest side, sigma <= 0.5 doubling it.
"""
import math

import numpy as np
import pytest
import scipy.sparse.linalg as spla

import rank_structured_cholesky_gb300 as rs

WIDE = dict(max_dense_block=10 ** 6, max_diag_block=10 ** 6)
# separators compressed at full rank: V U^T is exact
FULL = dict(max_dense_block=60, max_diag_block=200, rank_constant=50.0, diag_rank_constant=50.0)

CASES = [
    ("2d_17", (2, 17, 16, 1), {}),            # one or two levels of groups
    ("2d_33", (2, 33, 31, 1), {}),
    ("2d_65_wide", (2, 65, 64, 1), WIDE),     # chunk items, the root without rows
    ("2d_130", (2, 130, 129, 1), {}),
    ("3d_13", (3, 13, 11, 12), WIDE),         # chunks of a few rows
    ("3d_24_wide", (3, 24, 24, 25), WIDE),    # 576 columns: read in place (FP32 above 512, FP64 above 256)
    ("2d_90_full", (2, 90, 83, 1), FULL),     # compressed, ranks up to 90
    ("3d_18_full", (3, 18, 17, 19), FULL),    # ranks above 256: W and V read in place (FP64)
    ("3d_25_full", (3, 25, 24, 26), FULL),    # above 512 (FP32); several tiles of X with remainders
]


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("name,grid,params", CASES, ids=[c[0] for c in CASES])
def test_apply_is_the_direct_solve(name, grid, params, precision):
    dim, nx, ny, nz = grid
    prob = rs.diffusion(dim, nx, ny, nz, sigma=0.5, seed=7)
    F = rs.GpuFactor(rs.Context(precision=precision, **params), prob.colptr, prob.rowind, prob.vals, prob.xyz)
    b = np.random.default_rng(3).standard_normal((3, prob.n))
    want = spla.splu(prob.scipy().tocsc()).solve(b.T).T
    tol = 1e-10 if precision == "fp64" else 2e-5 * 4 * (max(nx, ny, nz) + 1) ** 2 / math.pi ** 2
    for k in range(3):
        x = F.apply(b[k])
        assert np.linalg.norm(x - want[k]) <= tol * np.linalg.norm(want[k])
        assert np.array_equal(x, F.apply(b[k]))   # counters start over; fixed order of every sum
    block = F.apply(b)
    assert np.linalg.norm(block - want) <= tol * np.linalg.norm(want)
