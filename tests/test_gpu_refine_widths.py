"""Refinement's sums for each number of right-hand sides their kernels are
compiled for and ones in between: conjugate gradients (Cholesky) and GMRES
(LDLt), one matrix and a batch, with fewer rows than one pass of the
reduction grid (592 blocks of 256 rows) and with more.  Bars: backward error
<= 1e-12 as the device reports it, the oracle's solution within 1e-9; a step
with the single-precision factor gains about five digits on these matrices, so
ten steps are twice what 1e-12 can need."""
import numpy as np
import pytest

import multifrontal as mf
from multifrontal import batch, testmatrices as tm
from oracle import oracle

pytestmark = pytest.mark.gpu

WIDTHS = (1, 2, 3, 4, 5, 8, 11, 16)


@pytest.mark.parametrize("kind", ["cg", "cg_long", "gmres"])
def test_one_matrix(kind):
    if kind == "gmres":
        A = tm.config4(side=7, m=120, per_row=6, seed=5)
        P, S = mf.symbolic(A, alg="natural")
        F = mf.ldlt_(mf.ChordalLDLt(A, P, S, mixed=True))
    else:
        nx, ny = (396, 390) if kind == "cg_long" else (31, 27)
        A = tm.grid_laplacian(nx, ny, seed=6)
        P, S = mf.symbolic(A, alg=mf.grid_nd_order(nx, ny, 1))
        F = mf.cholesky_(mf.ChordalCholesky(A, P, S, mixed=True))
    for k in WIDTHS:
        B = tm.rhs(S.n, k, seed=k)
        X = mf.ldiv(F, B)
        it, eta_dev = F.last_refinement
        eta = tm.backward_error(A, X, B).max()
        assert not F.used_fp64 and it <= 10
        assert eta <= 1e-12 and abs(eta - eta_dev) <= 1e-3 * eta + 1e-16
        if k in (3, 16):
            info, Xo, _ = oracle.factor_and_solve(A, P, S, B, int(kind == "gmres"))
            assert np.abs(X - Xo).max() <= 1e-9 * np.abs(Xo).max()
    F.close()


@pytest.mark.parametrize("ldlt", [False, True])
def test_segments(ldlt):
    if ldlt:
        mats = [tm.config4(side=s, m=max(8, s ** 3 // 4), seed=20 + i) for i, s in enumerate((5, 6, 5))]
        orders = ["amf"] * 3
    else:
        sides = ((31, 27), (9, 8), (40, 38))
        mats = [tm.grid_laplacian(a, b, seed=7 + a) for a, b in sides]
        orders = [mf.grid_nd_order(a, b, 1) for a, b in sides]
    F = batch.BatchedFactorization(mats, orders, ldlt=ldlt, mixed=True)
    F.factorize()
    for k in WIDTHS:
        rhs = [tm.rhs(A.shape[0], k, seed=30 + i) for i, A in enumerate(mats)]
        X = F.solve(rhs)
        seg = F.segment_errors()
        for i, A in enumerate(mats):
            eta = tm.backward_error(A, X[i], rhs[i]).max()
            assert eta <= 1e-12 and abs(seg[i] - eta) <= 1e-3 * eta + 1e-16
    F.close()
