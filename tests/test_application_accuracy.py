"""How accurate an exact factor's application is: dense matrices of a given condition
number, as one supernode and as two under a border, against LAPACK's Cholesky in the
same precision and against a bound.

The measure is the backward error |b - A x| / (|A| |x|), single and in a block.
"""
import math

import numpy as np
import pytest
import scipy.linalg as sl
import scipy.sparse as sp

import rank_structured_cholesky_gb300 as rs

pytestmark = pytest.mark.gpu
WIDE = dict(max_dense_block=10 ** 6, max_diag_block=10 ** 6)


def _spd(n, cond, rng):
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    A = (Q * np.exp(np.linspace(0, -np.log(cond), n))) @ Q.T
    return (A + A.T) / 2


def _matrix(p, r, cond):
    """p dense columns; with r > 0 two such blocks under a border of r rows."""
    rng = np.random.default_rng(1000 * p + r)
    if r == 0:
        return _spd(p, cond, rng)
    n = 2 * p + r
    L = np.zeros((n, n))
    for at, size in ((0, p), (p, p), (2 * p, r)):
        L[at:at + size, at:at + size] = np.linalg.cholesky(_spd(size, cond, rng))
    L[2 * p:, :2 * p] = rng.standard_normal((r, 2 * p)) / n
    A = L @ L.T
    A[:p, p:2 * p] = A[p:2 * p, :p] = 0
    return (A + A.T) / 2


def _factor(A, p, r, precision):
    M = sp.csc_matrix(A)
    M.sort_indices()
    return rs.GpuFactor(rs.Context(precision=precision, nd_leaf=max(p, r), **WIDE), M.indptr, M.indices, M.data)


def _backward(A, x, b):
    return np.linalg.norm(b - x @ A) / (np.linalg.norm(A, 2) * np.linalg.norm(x))


@pytest.mark.parametrize("p,r", [(100, 0), (300, 0), (700, 0), (150, 120), (300, 250)])
def test_mixed_is_as_accurate_as_lapack_in_fp32(p, r):
    """Condition number 10, random right-hand sides, 4 times LAPACK's error: sums in
    other orders, and products with inverses in place of substitutions.  (Products
    of 22 bits, a split of two TF32 operands, have 4 times the rounding of FP32 ones
    each, and it does not average out.)"""
    A = _matrix(p, r, 10.0)
    F = _factor(A, p, r, "mixed")
    b = np.random.default_rng(5).standard_normal((8, A.shape[0]))
    lapack = sl.cho_solve(sl.cho_factor(A.astype(np.float32), lower=True), b.T.astype(np.float32)).T.astype(np.float64)
    tol = 4 * _backward(A, lapack, b)
    assert _backward(A, np.array([F.apply(v) for v in b]), b) <= tol
    assert _backward(A, F.apply(b), b) <= tol


DENSE = [(n, 0) for n in (7, 20, 33, 50, 64, 65, 100, 300, 700)]
BORDERED = [(30, 20), (60, 50), (150, 120), (300, 250)]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("p,r", DENSE + BORDERED)
def test_smooth_right_hand_sides(p, r, precision):
    """b = A x of a random x: ill-conditioned blocks must not show in the residual
    (an inverse of A's block would leave the condition number in it).  Condition
    numbers 1e10 and, mixed, 1e4; under a border blocks of 1e6 and 1e3, which make a
    matrix of 1e9 and 1e4.  The bound: rounding errors of sums of up to 2 p + r terms,
    which grow as a random walk, times 4."""
    A = _matrix(p, r, {"fp64": 1e6 if r else 1e10, "mixed": 1e3 if r else 1e4}[precision])
    F = _factor(A, p, r, precision)
    b = np.random.default_rng(5).standard_normal((8, A.shape[0])) @ A
    tol = 4 * math.sqrt(A.shape[0]) * 2.0 ** (-53 if precision == "fp64" else -24)
    assert _backward(A, np.array([F.apply(v) for v in b]), b) <= tol
    assert _backward(A, F.apply(b), b) <= tol
