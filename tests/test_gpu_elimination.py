"""The elimination of small fronts (nj <= 96) and of 64-column diagonal blocks
at the sizes where its tiles, quads of columns and size classes begin and end:
two cliques that share a separator give one front of nn = a residual columns
and na = s separator rows, and a root of the separator with the second
clique.  Bars as everywhere: FP64 backward error <= 1e-13 and within 1e-9 of
the oracle, refined <= 1e-12."""
import numpy as np
import pytest
import scipy.sparse as sp

import multifrontal as mf
from multifrontal import testmatrices as tm
from oracle import oracle

pytestmark = pytest.mark.gpu


def two_cliques(a, b, s, ldlt, seed):
    """Dense on [0, a) + S and on [a, a + b) + S; quasidefinite for LDLt."""
    n = a + b + s
    rng = np.random.default_rng(seed)
    A = np.zeros((n, n))
    S = np.arange(a + b, n)
    for part in (np.arange(a), np.arange(a, a + b)):
        idx = np.concatenate([part, S])
        G = rng.standard_normal((idx.size, idx.size))
        A[np.ix_(idx, idx)] += 0.5 * (G + G.T)
    sign = np.where(np.arange(n) % 3 == 1, -1.0, 1.0) if ldlt else np.ones(n)
    A[np.arange(n), np.arange(n)] = sign * (np.abs(A).sum(axis=1) + 1.0)
    return sp.csc_matrix(A)


SIZES = [(1, 1, 1), (2, 3, 2), (3, 5, 14), (5, 4, 11), (7, 8, 25), (17, 16, 15), (20, 12, 28), (33, 30, 15), (33, 5, 31),
         (40, 7, 56), (47, 1, 1), (61, 9, 3), (64, 31, 32), (65, 2, 31), (94, 30, 2), (95, 48, 1), (97, 63, 2),
         (127, 96, 5), (130, 64, 60), (190, 129, 3)]


@pytest.mark.parametrize("ldlt", [False, True])
@pytest.mark.parametrize("a,b,s", SIZES)
def test_edges_of_tiles_and_quads(a, b, s, ldlt):
    A = two_cliques(a, b, s, ldlt, seed=1000 * a + s)
    P, S = mf.symbolic(A, alg=np.arange(A.shape[0]))
    assert a in S.nn() or (a + s) in (S.nn() + S.na())
    B = tm.rhs(S.n, 2, seed=a)
    info, Xo, _ = oracle.factor_and_solve(A, P, S, B, int(ldlt))
    assert info == 0
    for mixed in (False, True):
        F = mf.ldlt_(mf.ChordalLDLt(A, P, S, mixed=mixed)) if ldlt else mf.cholesky_(mf.ChordalCholesky(A, P, S, mixed=mixed))
        X = mf.ldiv(F, B)
        assert not F.used_fp64
        assert tm.backward_error(A, X, B).max() <= (1e-12 if mixed else 1e-13)
        assert np.abs(X - Xo).max() <= 1e-9 * np.abs(Xo).max()
        F.close()
