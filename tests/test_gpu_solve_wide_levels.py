"""Solves of small fronts, a CTA each against warps (a level of at most
8 x 148 takes CTAs): every level of the forest here is wide and every level
of the single matrix narrow, which the test reads off the plan, so each front
size is solved both ways.  The operations and their order are the same:
FP64 solutions must be bitwise equal, with fronts of at most 16, 32 and 96
rows and of at most 64 columns over a longer separator among them.  The
forest takes its fronts of at most 32 rows 16 or 32 lanes each, and (with
MF_TINY_SOLVE=0) a warp each like the others."""
import numpy as np
import pytest

import multifrontal as mf
from multifrontal import testmatrices as tm
from multifrontal._native import check, ptr64
from multifrontal.batch import block_symbolic

from test_gpu_tile_heights import repeat

pytestmark = pytest.mark.gpu

LIMIT = 8 * 148


def small_fronts_by_level(F):
    """Per tree level of the plan: rows of its small fronts (nj <= 96, or nn <= 64 and na <= 256)."""
    lib, h = F._handle.lib, F._handle.h
    info = np.zeros(9, np.int64)
    check(lib.mf_info(h, ptr64(info)), "mf_info")
    nn, na, parent = (np.zeros(info[8], np.int64) for _ in range(3))
    check(lib.mf_exec_sizes(h, ptr64(nn), ptr64(na)), "mf_exec_sizes")
    check(lib.mf_exec_parents(h, ptr64(parent)), "mf_exec_parents")
    level = np.zeros(nn.size, np.int64)
    for e in range(nn.size):  # children come before their parents
        if parent[e] >= 0:
            assert parent[e] > e
            level[parent[e]] = max(level[parent[e]], level[e] + 1)
    small = (nn + na <= 96) | ((nn <= 64) & (na <= 256))
    assert info[7] == level.max() + 1
    return [(nn + na)[small & (level == v)] for v in range(info[7])]


@pytest.mark.parametrize("tiny", ["1", "0"])
@pytest.mark.parametrize("ldlt", [False, True])
def test_every_level_both_ways(ldlt, tiny, monkeypatch):
    monkeypatch.setenv("MF_TINY_SOLVE", tiny)
    copies = LIMIT + 6
    A = tm.grid_laplacian(9, 9, 16, seed=83, lo=1e-1, hi=10.0)
    P, S = mf.symbolic(A, alg=mf.grid_nd_order(9, 9, 16))
    PB, SB, off = block_symbolic([(P, S)] * copies)
    cls, fac = (mf.ChordalLDLt, mf.ldlt_) if ldlt else (mf.ChordalCholesky, mf.cholesky_)
    alone = fac(cls(A, P, S))
    forest = fac(cls(repeat(A, np.ones(copies)), PB, SB))
    one, many = small_fronts_by_level(alone), small_fronts_by_level(forest)
    assert all(v.size <= LIMIT for v in one) and all(v.size == 0 or v.size > LIMIT for v in many)
    rows = np.concatenate(one)
    assert [np.any((rows > lo) & (rows <= hi)) for lo, hi in ((0, 16), (16, 32), (32, 96), (96, 320))] == [True] * 4
    for nrhs in (1, 4, 16):
        B = tm.rhs(S.n, nrhs, seed=96 + nrhs)
        X = mf.ldiv(alone, B)
        XB = mf.ldiv(forest, np.tile(B, (copies, 1)))
        for c in (0, 1, copies // 2, copies - 1):
            assert np.array_equal(XB[off[c]:off[c + 1]], X), (nrhs, c)
        assert tm.backward_error(A, X, B).max() <= 1e-13
    alone.close()
    forest.close()
