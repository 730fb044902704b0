"""Solves of a level's small fronts: a CTA per front where the level holds few
(at most 8 x 148), warps where it holds many.  The same matrix alone and as
every member of a large forest takes the two paths at every level, and their
operations are the same in the same order: the FP64 solutions must be bitwise
equal.  Right-hand-side counts cover each width the kernels are compiled for
and one in between; the sizes cover fronts of one column, of at most 96 rows,
and of at most 64 columns over a long separator."""
import numpy as np
import pytest

import multifrontal as mf
from multifrontal import testmatrices as tm
from multifrontal.batch import block_symbolic
from oracle import oracle
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ldlt", [False, True])
@pytest.mark.parametrize("shape,copies", [((9, 8, 1), 1300), ((10, 10, 9), 620)])
def test_alone_equals_member_of_a_wide_forest(shape, copies, ldlt):
    nx, ny, nz = shape
    A = tm.grid_laplacian(nx, ny, nz, seed=81, lo=1e-1, hi=10.0)
    P, S = mf.symbolic(A, alg=mf.grid_nd_order(nx, ny, nz))
    PB, SB, off = block_symbolic([(P, S)] * copies)
    cls, fac = (mf.ChordalLDLt, mf.ldlt_) if ldlt else (mf.ChordalCholesky, mf.cholesky_)
    alone = fac(cls(A, P, S))
    forest = fac(cls(sp.block_diag([A] * copies, format="csc"), PB, SB))
    for nrhs in (1, 2, 3, 8, 16):
        B = tm.rhs(S.n, nrhs, seed=90 + nrhs)
        X = mf.ldiv(alone, B)
        XB = mf.ldiv(forest, np.tile(B, (copies, 1)))
        for c in (0, 1, copies // 2, copies - 1):
            assert np.array_equal(XB[off[c]:off[c + 1]], X), (nrhs, c)
        assert tm.backward_error(A, X, B).max() <= 1e-13
        info, Xo, _ = oracle.factor_and_solve(A, P, S, B, int(ldlt))
        assert np.abs(X - Xo).max() <= 1e-9 * np.abs(Xo).max()
    alone.close()
    forest.close()
