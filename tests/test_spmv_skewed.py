"""SpMV of rows of very different lengths: one row of 3,000 entries among rows of 15
or 50.  As quick, to a factor of 1.5, as with 16 threads a row (two of them take more
than twice as long for the long row), and right: the true residual that PCG reports
against scipy's product."""
import numpy as np
import pytest
import scipy.sparse as sp

import rank_structured_cholesky_gb300 as rs


def _matrix(n, width):
    rng = np.random.default_rng(width)
    offs = range(1, width // 2)
    A = sp.diags([rng.uniform(-1, 0, n - o) for o in offs], [-o for o in offs], shape=(n, n)).tocsc()
    near = np.arange(n // 2 - 3000, n // 2)   # of the long row
    A = A + sp.csc_matrix((rng.uniform(-1, 0, 3000), (np.full(3000, n // 2), near)), shape=(n, n))
    A = A + A.T
    A = (A + sp.diags(np.asarray(abs(A).sum(axis=1)).ravel() + 1.0)).tocsc()
    A.sort_indices()
    return A


@pytest.mark.gpu
@pytest.mark.parametrize("width", [16, 50])
def test_one_long_row(width, monkeypatch):
    n = 60000
    A = _matrix(n, width)
    xyz = np.zeros((n, 3))
    xyz[:, 0] = np.arange(n)
    b = np.random.default_rng(1).standard_normal(n)
    ms = {}
    for threads in ("", "16"):
        if threads:
            monkeypatch.setenv("RSCHOL_SPMV_TPR", threads)
        F = rs.GpuFactor(rs.Context(precision="fp64"), A.indptr, A.indices, A.data, xyz.ravel())
        x, info = F.pcg(b, 1e-3, 1)
        r = np.linalg.norm(b - A @ x) / np.linalg.norm(b)
        slack = 4 * n * 2.0 ** -52 * np.linalg.norm(abs(A) @ abs(x)) / np.linalg.norm(b)
        assert abs(info["true_residual"] - r) <= 1e-10 * r + slack
        ms[threads] = min(_spmv_ms(F, b) for _ in range(3))
    assert ms[""] <= 1.5 * ms["16"]


def _spmv_ms(F, b):
    import torch
    out = np.zeros(16)
    d = torch.from_numpy(b).cuda()
    assert rs.load_library().rschol_profile(F.h, d.data_ptr(), out.ctypes.data) == 0
    return out[2]
