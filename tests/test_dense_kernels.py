"""The dense kernels at their edges: the FP64 GEMM around its 16-wide blocks and
32-wide tiles, whole and split along K, the FP32 one around its tiles of 64 and
128 rows and slices of 16 K, with odd and even leading dimensions, and the Householder QR around the row
counts where its panel kernel changes (512; 2048, 4096 and 8192 rows of a
cluster's registers) and its 16-column panels.

GEMM: a sum of K products in any order is within K eps of sum |a b|.  QR:
Householder's Q is orthogonal, and the columns are reproduced, to a modest
multiple of r sqrt(n) eps.
"""
import ctypes
import math

import pytest

import rank_structured_cholesky_gb300 as rs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tA,tB", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("M,N,K,slices", [(1, 1, 1, 1), (15, 17, 31, 1), (16, 16, 32, 1), (33, 32, 33, 1),
                                          (64, 65, 129, 2), (31, 48, 200, 3), (97, 40, 1006, 16), (70, 33, 65, 65)])
def test_gemm_fp64(M, N, K, slices, tA, tB):
    out = (ctypes.c_double * 1)()
    assert rs.load_library().rschol_selftest_gemm64(M, N, K, tA, tB, slices, out) == 0
    assert out[0] <= (K + 4) * 2.0 ** -52


@pytest.mark.parametrize("rows", [64, 128])
@pytest.mark.parametrize("tA,tB", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (63, 65, 15), (64, 64, 16), (127, 63, 17), (128, 64, 31), (129, 130, 33),
                                   (200, 97, 112), (257, 66, 70)])
def test_gemm_fp32(M, N, K, tA, tB, rows):
    out = (ctypes.c_double * 1)()
    assert rs.load_library().rschol_selftest_gemm32(M, N, K, tA, tB, rows, out) == 0
    assert out[0] <= (K + 4) * 2.0 ** -23


@pytest.mark.parametrize("fp64", [0, 1])
@pytest.mark.parametrize("n,r", [(1, 1), (16, 16), (17, 5), (100, 33), (512, 16), (513, 17), (2048, 20), (2049, 31),
                                 (4096, 16), (4097, 18), (8192, 3), (8193, 33)])
def test_householder_qr(n, r, fp64):
    out = (ctypes.c_double * 2)()
    assert rs.load_library().rschol_selftest_qr(n, r, 3, fp64, out) == 0
    tol = 4 * r * math.sqrt(n) * 2.0 ** (-52 if fp64 else -23)
    assert out[0] <= tol and out[1] <= tol
