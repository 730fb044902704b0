"""FP64 GEMM tiles of 32, 64 and 128 rows.  A launch takes the height that its
tile counts give it, so the same front gets another height as a member of
a forest than alone; the products of an entry are added in the same order at
every height, so the factors must be bitwise equal.  Members are scaled by
powers of four (exact in the factors), so that a tile which read another
member's panel would show.  The sizes are odd and even, with every remainder of
four, at one column or row past a tile's edge and one short of it; the one of
579 columns has trailing updates in two parts (the next outer block's
columns, then the rest).  The single matrix is also compared with the oracle: backward error
<= 1e-13 and within 1e-9."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

import multifrontal as mf
from multifrontal import testmatrices as tm
from multifrontal._native import check, ptr64
from multifrontal.batch import block_symbolic
from oracle import oracle

from test_gpu_elimination import two_cliques

pytestmark = pytest.mark.gpu


def repeat(A, scales):
    n, nnz, m = A.shape[0], A.nnz, len(scales)
    data = (scales[:, None] * A.data).ravel()
    idx = (np.arange(m)[:, None] * n + A.indices).ravel()
    ptr = np.concatenate([[0], (np.arange(m)[:, None] * nnz + A.indptr[1:]).ravel()])
    return sp.csc_matrix((data, idx, ptr), shape=(m * n, m * n))


def height(small, large):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return 128 if large >= 2 * sms else 64 if small >= sms else 32


def cdiv(a, b):
    return -(-a // b)


def heights(nn, na, m):
    """Tile heights of the roles for m fronts of nn columns and na rows."""
    nj, h = nn + na, {"left": set(), "trsm": set(), "trail": set()}
    for c0 in range(0, nn, 64):
        r0 = min(nn, c0 + 64)
        now = height(m * cdiv(nj - r0, 64), m * cdiv(nj - (r0 & ~3), 128))
        h["trsm"].add(now)
        if c0 % 256:
            h["left"].add(now)
        e = (c0 // 256 + 1) * 256
        if r0 == e and e < nn:
            for far in (False, True):
                small = sum(cdiv(nj - e - 64 * t, 64) for t in range(cdiv(nn - e, 64)) if (t >= 4) == far)
                large = sum(cdiv(nj - e - 128 * t, 128) for t in range(cdiv(nn - e, 128)) if (t >= 2) == far)
                if small:
                    h["trail"].add(height(m * small, 2 * m * large))
    d, t = nn & 3, cdiv(na, 64)
    large = sum(cdiv(na + d - 128 * j, 128) for j in range(cdiv(na + d, 128)))
    h["syrk"] = {height(m * t * (t + 1) // 2, 2 * m * large)}
    return h


# columns, rows below, members, and what the case is there for
CASES = [(129, 33, 160, {"left": {64}, "trsm": {64}, "syrk": {128}}),
         (130, 65, 60, {"syrk": {64}}),
         (131, 66, 70, {"syrk": {64}}),
         (65, 64, 150, {"trsm": {64}, "syrk": {128}}),
         (129, 33, 300, {"left": {128}, "trsm": {128}}),
         (130, 61, 300, {"left": {128}, "trsm": {128}}),
         (127, 130, 300, {"left": {128}, "trsm": {128}, "syrk": {128}}),
         (323, 35, 60, {"trail": {64}}),
         (321, 32, 150, {"trail": {128}}),
         (579, 34, 60, {"trail": {64, 128}})]


@pytest.mark.parametrize("ldlt", [False, True])
@pytest.mark.parametrize("nn,na,m,want", CASES)
def test_member_equals_the_matrix_alone(nn, na, m, want, ldlt, monkeypatch):
    monkeypatch.setenv("MF_AMALGAMATE", "0")
    got = heights(nn, na, m)
    assert all(got[role] == h for role, h in want.items()), got
    A = two_cliques(1, nn, na, ldlt, seed=31 * nn + na)
    P, S = mf.symbolic(A, alg=np.arange(A.shape[0]))
    PB, SB, off = block_symbolic([(P, S)] * m)
    scales = 4.0 ** (np.arange(m) % 3 - 1)
    cls, fac = (mf.ChordalLDLt, mf.ldlt_) if ldlt else (mf.ChordalCholesky, mf.cholesky_)
    alone = fac(cls(A, P, S))
    sizes = np.empty(16, np.int64), np.empty(16, np.int64)
    check(alone._handle.lib.mf_exec_sizes(alone._handle.h, ptr64(sizes[0]), ptr64(sizes[1])), "mf_exec_sizes")
    assert (sizes[0][0], sizes[1][0]) == (nn, na)  # the plan holds the front as it is
    D, L, d = alone.factor_arrays()
    B = tm.rhs(S.n, 2, seed=nn)
    X = mf.ldiv(alone, B)
    alone.close()
    forest = fac(cls(repeat(A, scales), PB, SB))
    DB, LB, dB = forest.factor_arrays()
    forest.close()
    for c in {0, 1, 2, m // 2, m - 2, m - 1}:
        f = 1.0 if ldlt else np.sqrt(scales[c])
        assert np.array_equal(LB[c * L.size:(c + 1) * L.size], f * L), c
        Dc = DB[c * D.size:(c + 1) * D.size]
        for j in range(S.nfr):
            w = S.nn(j)
            blk = slice(S.Dptr[j], S.Dptr[j] + w * w)
            lo = np.tril(D[blk].reshape(w, w, order="F"), -1 if ldlt else 0)
            assert np.array_equal(np.tril(Dc[blk].reshape(w, w, order="F"), -1 if ldlt else 0), f * lo), (c, j)
        if ldlt:
            assert np.array_equal(dB[off[c]:off[c + 1]], scales[c] * d), c
    assert tm.backward_error(A, X, B).max() <= 1e-13
    info, Xo, _ = oracle.factor_and_solve(A, P, S, B, int(ldlt))
    assert info == 0
    assert np.abs(X - Xo).max() <= 1e-9 * np.abs(Xo).max()
