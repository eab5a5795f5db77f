"""Two factors in use at once: what one of them plans leaves the other's calls as they
were, in either order of creation, and calls on both at the same time (a thread and a
stream each) give what they give alone, bit for bit.

The wide factor has supernodes above 128 columns, worked off in chunks; the narrow
one has groups of small supernodes only.  Exact factors: one application solves
A x = b (FP64 1e-10; mixed 2e-5 times the grid's condition number, as in the tests of
the work items).
"""
import math
import threading

import numpy as np
import pytest
import scipy.sparse.linalg as spla

import rank_structured_cholesky_gb300 as rs

pytestmark = pytest.mark.gpu
WIDE = dict(max_dense_block=10 ** 6, max_diag_block=10 ** 6)
GRIDS = {"wide": (3, 13, 12, 14), "narrow": (2, 20, 19, 1)}


class _System:
    def __init__(self, which, precision):
        grid = GRIDS[which]
        self.prob = rs.diffusion(*grid, sigma=0.5, seed=11)
        self.F = rs.GpuFactor(rs.Context(precision=precision, **WIDE), self.prob.colptr, self.prob.rowind,
                              self.prob.vals, self.prob.xyz)
        self.b = np.random.default_rng(5).standard_normal(self.prob.n)
        self.want = spla.splu(self.prob.scipy().tocsc()).solve(self.b)
        self.tol = 1e-10 if precision == "fp64" else 2e-5 * 4 * (max(grid[1:]) + 1) ** 2 / math.pi ** 2

    def check(self):
        x = self.F.apply(self.b)
        assert np.linalg.norm(x - self.want) <= self.tol * np.linalg.norm(self.want)
        y, info = self.F.pcg(self.b, 1e-8, 50)
        assert info["true_residual"] <= 1e-8
        return x, y


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("order", [("wide", "narrow"), ("narrow", "wide")])
def test_second_factor_leaves_the_first(order, precision):
    systems = [_System(w, precision) for w in order]
    for s in systems:
        s.check()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_two_factors_at_the_same_time(precision):
    systems = [_System(w, precision) for w in ("wide", "narrow")]
    alone = [s.check() for s in systems]
    got = [[], []]

    def work(q):
        for _ in range(40):
            got[q].append(systems[q].check())

    threads = [threading.Thread(target=work, args=(q,)) for q in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(60)
    for q in range(2):
        assert len(got[q]) == 40
        for x, y in got[q]:
            assert np.array_equal(x, alone[q][0]) and np.array_equal(y, alone[q][1])
