"""Sub-panels of a blocked front in FP64: the diagonal block's own left-looking
update beside that of the rows below it, at the widths where a last block is
one column, one short of full, full, or starts an outer block (256 columns;
512 when MF_WIDE_FRONT_NN lets these fronts take it), with no rows, one row and
a tile's worth of rows below.  Bars as everywhere: backward error <= 1e-13 and
within 1e-9 of the oracle."""
import numpy as np
import pytest

import multifrontal as mf
from multifrontal import testmatrices as tm
from oracle import oracle

from test_gpu_elimination import two_cliques

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("ldlt", [False, True])
@pytest.mark.parametrize("a,b,s", [(65, 40, 31), (127, 97, 1), (128, 70, 129), (129, 128, 33), (193, 96, 2), (255, 100, 5),
                                   (256, 131, 64), (257, 120, 7), (321, 190, 65), (513, 66, 3)])
def test_block_widths(a, b, s, ldlt, wide, monkeypatch):
    if wide:
        monkeypatch.setenv("MF_WIDE_FRONT_NN", "97")
    A = two_cliques(a, b, s, ldlt, seed=7 * a + s)
    P, S = mf.symbolic(A, alg=np.arange(A.shape[0]))
    B = tm.rhs(S.n, 3, seed=b)
    info, Xo, _ = oracle.factor_and_solve(A, P, S, B, int(ldlt))
    assert info == 0
    F = mf.ldlt_(mf.ChordalLDLt(A, P, S)) if ldlt else mf.cholesky_(mf.ChordalCholesky(A, P, S))
    X = mf.ldiv(F, B)
    assert tm.backward_error(A, X, B).max() <= 1e-13
    assert np.abs(X - Xo).max() <= 1e-9 * np.abs(Xo).max()
    F.close()
