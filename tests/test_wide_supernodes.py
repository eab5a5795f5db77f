"""Uncompressed supernodes of any width: f of a chunk item goes through shared memory
in tiles of 4096 bytes (1024 columns in FP32, 512 in FP64), so that no width is too
wide for it.

Tiles: a dense matrix, one supernode; diagonally dominant, condition number below 4.
Planes: a grid of nx x ny points in three planes, far apart, so that dissection takes
the middle plane for the top separator, one dense supernode of nx * ny columns and
more; the 7-point stencil with 7 on the diagonal, eigenvalues 1 to 13.

The factors are exact, so one application solves A x = b: the residual is the
condition number times the rounding errors of sums of as many terms as the
supernode has columns, which grow as a random walk, times 4.
"""
import math

import numpy as np
import pytest
import scipy.sparse as sp

import rank_structured_cholesky_gb300 as rs

WIDE = dict(max_dense_block=10 ** 6, max_diag_block=10 ** 6)


def _planes(nx, ny):
    def path(k):
        return sp.diags([np.ones(k - 1), np.ones(k - 1)], [-1, 1], shape=(k, k))

    ex, ey, ez = sp.identity(nx), sp.identity(ny), sp.identity(3)
    adj = sp.kron(sp.kron(path(nx), ey), ez) + sp.kron(sp.kron(ex, path(ny)), ez) + sp.kron(sp.kron(ex, ey), path(3))
    A = (7.0 * sp.identity(3 * nx * ny) - adj).tocsc()
    A.sort_indices()
    i = np.arange(3 * nx * ny)
    xyz = np.stack([i // (3 * ny), i // 3 % ny, 10.0 * max(nx, ny) * (i % 3)], axis=1)
    return A, np.ascontiguousarray(xyz, np.float64).ravel()


def _dense(width):
    rng = np.random.default_rng(width)
    A = np.tril(rng.uniform(-1, 1, (width, width)), -1)
    A = A + A.T
    A[np.diag_indices(width)] = 2.0 * np.abs(A).sum(axis=1) + 1.0
    M = sp.csc_matrix(A)
    M.sort_indices()
    return M


def _check(A, xyz, precision, width, cond, **params):
    F = rs.GpuFactor(rs.Context(precision=precision, **WIDE, **params), A.indptr, A.indices, A.data, xyz)
    b = np.random.default_rng(width).standard_normal(A.shape[0])
    x = F.apply(b)
    eps = 2.0 ** -52 if precision == "fp64" else 2.0 ** -23
    assert np.linalg.norm(b - A @ x) <= 4 * cond * math.sqrt(width) * eps * np.linalg.norm(b)
    assert np.array_equal(x, F.apply(b))


def test_the_widths_are_reached():
    M = _dense(700)
    why = rs.check_structure(M.indptr, M.indices, max_dense_block=10 ** 6, max_diag_block=699, nd_leaf=700)[1]
    assert "has 700 columns" in why
    for nx, ny in ((23, 22), (102, 102), (143, 143)):
        A, xyz = _planes(nx, ny)
        why = rs.check_structure(A.indptr, A.indices, xyz, max_dense_block=10 ** 6, max_diag_block=nx * ny - 1)[1]
        assert "columns, more than max_diag_block" in why


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("width", [511, 512, 513, 1023, 1024, 1025, 2048, 2051])
def test_tiles_of_f(width, precision):
    _check(_dense(width), None, precision, width, 4, nd_leaf=width)


@pytest.mark.gpu
@pytest.mark.parametrize("precision,nx,ny", [("fp64", 23, 22), ("mixed", 23, 22), ("fp64", 33, 31), ("mixed", 33, 31),
                                             ("mixed", 46, 45), ("fp64", 102, 102), ("mixed", 143, 143)])
def test_planes(precision, nx, ny):
    A, xyz = _planes(nx, ny)
    _check(A, xyz, precision, nx * ny, 13)
