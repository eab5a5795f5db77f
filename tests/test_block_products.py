"""Blocks of right-hand sides on compressed supernodes: the products with V and W at the
ranks where the rows of an item, and with them the split of K, change -- and what a
column's sums must not depend on, the width of the block.

Full ranks, so an application is the direct solve, to the tolerances of the
single-vector test (FP64 1e-10; mixed 2e-5 times the grid's condition number).  And a
block of two columns takes no longer than two applications to one, plus a tenth: at
large ranks it took three (a thread for all of K).
"""
import math
import time

import numpy as np
import pytest
import scipy.sparse.linalg as spla

import rank_structured_cholesky_gb300 as rs

pytestmark = pytest.mark.gpu
FULL = dict(max_diag_block=200, rank_constant=50.0, diag_rank_constant=50.0)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("grid,dense", [((2, 60, 55, 1), 20), ((2, 90, 83, 1), 40), ((3, 14, 13, 15), 60), ((3, 18, 17, 19), 60),
                                        ((3, 25, 24, 26), 100)])
def test_widths(grid, dense, precision):
    prob = rs.diffusion(*grid, sigma=0.5, seed=7)
    F = rs.GpuFactor(rs.Context(precision=precision, max_dense_block=dense, **FULL), prob.colptr, prob.rowind, prob.vals,
                     prob.xyz)
    b = np.random.default_rng(3).standard_normal((17, prob.n))
    x = F.apply(b)
    want = spla.splu(prob.scipy().tocsc()).solve(b.T).T
    tol = 1e-10 if precision == "fp64" else 2e-5 * 4 * (max(grid[1:]) + 1) ** 2 / math.pi ** 2
    assert np.linalg.norm(x - want) <= tol * np.linalg.norm(want)
    for k in (2, 3, 5, 8):
        assert np.array_equal(x[:k], F.apply(b[:k]))


def test_two_columns_cost_no_more_than_two_applications():
    import torch
    prob = rs.diffusion(3, 32, 32, 32, sigma=1.0, seed=1)
    F = rs.GpuFactor(rs.Context(precision="fp64", rank_constant=3.0), prob.colptr, prob.rowind, prob.vals, prob.xyz)
    b = torch.randn(2, prob.n, dtype=torch.float64, device="cuda")
    x = torch.zeros_like(b)
    best = {}
    for k in (1, 2):
        for _ in range(25):
            t = time.perf_counter()
            assert rs.load_library().rschol_precond_apply_device(F.h, b.data_ptr(), x.data_ptr(), k) == 0
            best[k] = min(best.get(k, 1.0), time.perf_counter() - t)
    assert best[2] <= 2.2 * best[1]
