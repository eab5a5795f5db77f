"""One Householder QR launch of tasks of different shapes: the panel kernel is chosen
by the tallest task and meets a shorter and narrower one beside it.

Planes of points far apart, so that dissection takes whole planes for separators: one
of 46 x 45 points (above the 2048 rows that a cluster holds with one row a thread) and
one of 20 x 30 are compressed in the same level, at full rank, so that the factor is
exact.  7 on the diagonal and -1 to every neighbour: condition below 13.  FP64: the
direct solve to 1e-12; mixed: the split products' 1e-5 times 13.
"""
import numpy as np
import pytest
import scipy.sparse as sp

import rank_structured_cholesky_gb300 as rs

PARAMS = dict(max_dense_block=200, max_diag_block=10 ** 6, rank_constant=50.0, diag_rank_constant=50.0)


def _system():
    points = [(x, y, z) for z in range(7) for x in range(46) for y in range(45) if z > 2 or (x < 20 and y < 30)]
    at = {p: i for i, p in enumerate(points)}
    edges = [(i, at[q]) for (x, y, z), i in at.items() for q in ((x + 1, y, z), (x, y + 1, z), (x, y, z + 1)) if q in at]
    r, c = np.array(edges).T
    n = len(points)
    A = sp.coo_matrix((-np.ones(2 * len(r)), (np.r_[r, c], np.r_[c, r])), shape=(n, n)) + 7.0 * sp.identity(n)
    A = A.tocsc()
    A.sort_indices()
    xyz = np.array(points, np.float64) * (1, 1, 1000)
    return A, xyz.ravel()


@pytest.mark.gpu
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("mixed", 1.3e-4)])
def test_launch_of_different_shapes(precision, tol):
    A, xyz = _system()
    F = rs.GpuFactor(rs.Context(precision=precision, **PARAMS), A.indptr, A.indices, A.data, xyz)
    nodes = [F.node_info(j) for j in range(F.num_nodes())]
    shapes = sorted((v["c1"] - v["c0"] + 1, v["rank"]) for v in nodes if v["compressed"] and v["m"] > 0)
    assert shapes[0][0] < 1024 < 2048 < shapes[-1][0] and all(rank >= 500 for _, rank in shapes)
    b = np.random.default_rng(3).standard_normal(A.shape[0])
    assert np.linalg.norm(b - A @ F.apply(b)) <= tol * np.linalg.norm(b)
