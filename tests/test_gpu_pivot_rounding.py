"""Rounding of the eliminations of small fronts (a warp or a CTA each) and of
64-column diagonal blocks.

Reciprocal pivots: the entry below a pivot p is a times the correctly rounded
reciprocal of the stored diagonal entry (sqrt(p) rounded, or p), over the
exponent range in FP64, and in single precision over what the scaled matrix can
hold; there the diagonal blocks' Cholesky takes a reciprocal square root of at
most 2 ulp.  The expected values are numpy's, each operation of which rounds
correctly, so all but that last one must be equal bit for bit.

Order of sums: a pivot's updates in a diagonal block are summed four columns
at a time before they are subtracted.  With entries in [1, 2) every subtraction
adds a rounding error of variance 2^-104 / 12, so the 64th pivot of a block has
an error of sqrt(18 / 12) 2^-52 in the root mean square (fifteen groups, then
three columns of its own group); subtracted one by one it would be
sqrt(63 / 12) 2^-52.  The bar lies between, at 1.6 x 2^-52."""
import numpy as np
import pytest
import scipy.sparse as sp

import multifrontal as mf

pytestmark = pytest.mark.gpu

# columns of a member, members: warp per front, the CTA size classes, diagonal block
PATHS = [(3, 700), (3, 400), (40, 300), (60, 300), (90, 300), (98, 300)]


def dense_members(blocks):
    """Block-diagonal matrix of dense members."""
    m, n, _ = blocks.shape
    idx = (np.arange(m)[:, None, None] * n + np.arange(n)[None, None, :] + np.zeros((m, n, 1), np.int64)).ravel()
    ptr = np.arange(m * n + 1) * n
    return sp.csc_matrix((blocks.transpose(0, 2, 1).ravel(), idx, ptr), shape=(m * n, m * n))


def factor(blocks, ldlt, mixed):
    """Per member the strictly lower part of L and the pivots (LDLt)."""
    m, n, _ = blocks.shape
    A = dense_members(blocks)
    P, S = mf.symbolic(dense_members(np.ones_like(blocks)), alg=np.arange(A.shape[0]))
    # the ordering may move members, not the columns inside one
    perm = np.asarray(P.perm).reshape(m, n)
    at = np.argsort(perm[:, 0])
    assert S.nfr == m and np.array_equal(perm[at].ravel(), np.arange(m * n))
    F = (mf.ChordalLDLt if ldlt else mf.ChordalCholesky)(A, P, S, mixed=mixed)
    (mf.ldlt_ if ldlt else mf.cholesky_)(F)
    assert F.info == 0 and not F.used_fp64 and F.rescued == 0
    D, _, d, *scale = F.factor_arrays_mixed() if mixed else F.factor_arrays()
    F.close()
    assert all(np.all(s == 1.0) for s in scale)
    return D.reshape(m, n, n).transpose(0, 2, 1)[at], d.reshape(m, n)[at]


@pytest.mark.parametrize("ldlt", [False, True])
@pytest.mark.parametrize("n,m", PATHS)
def test_fp64_reciprocal_pivot(n, m, ldlt):
    rng = np.random.default_rng(n + m)
    p = 10.0 ** np.linspace(-300, 300, m) * rng.uniform(1, 10, m)
    p[:4] = [3e-308, 1.0, 2.0, 1.0e308] if ldlt else [7e-310, 1.0, 2.0, 1.7e308]
    mant = rng.uniform(0.25, 0.5, m)
    a = p * mant if ldlt else np.sqrt(p) * mant
    blocks = np.zeros((m, n, n))
    blocks[:, np.arange(n), np.arange(n)] = 2.0
    blocks[:, 0, 0] = p
    blocks[:, 1, 0] = blocks[:, 0, 1] = a
    if ldlt:
        blocks[:, 1, 1] = -p  # the second pivot stays of the first one's size
    L, d = factor(blocks, ldlt, False)
    assert np.array_equal(L[:, 1, 0], a * (1.0 / (p if ldlt else np.sqrt(p))))
    assert np.array_equal(d[:, 0] if ldlt else L[:, 0, 0], p if ldlt else np.sqrt(p))


@pytest.mark.parametrize("ldlt", [False, True])
@pytest.mark.parametrize("n,m", PATHS)
def test_single_precision_reciprocal_pivot(n, m, ldlt):
    # unit diagonal (so the scaling is 1) and b = k / 2^11: the second pivot 1 - b^2 is exact
    rng = np.random.default_rng(2 * n + m)
    b = rng.permutation(2047)[:m] / 2048.0
    p = (1.0 - b * b).astype(np.float32)
    c = (np.sqrt(p) * rng.uniform(0.25, 0.5, m)).astype(np.float32)
    blocks = np.zeros((m, n, n))
    blocks[:, np.arange(n), np.arange(n)] = 1.0
    blocks[:, 1, 0] = blocks[:, 0, 1] = b
    blocks[:, 2, 1] = blocks[:, 1, 2] = c
    L, d = factor(blocks, ldlt, True)
    want = c * (np.float32(1) / (p if ldlt else np.sqrt(p)))
    if n > 96 and not ldlt:
        exact = c.astype(np.float64) / np.sqrt(p.astype(np.float64))
        assert np.all(np.abs(L[:, 2, 1] - exact) <= 2.5 * 2.0 ** -23 * exact)  # 2 ulp, then the product's rounding
    else:
        assert np.array_equal(L[:, 2, 1], want.astype(np.float64))
    if ldlt:
        assert np.array_equal(d[:, 1], p.astype(np.float64))


@pytest.mark.parametrize("ldlt", [False, True])
def test_block_sums_updates_by_fours(ldlt):
    n, m, k = 98, 400, 63
    rng = np.random.default_rng(17)
    G = rng.uniform(-0.05, 0.05, (m, 64, 64))
    blocks = np.zeros((m, n, n))
    blocks[:, np.arange(n), np.arange(n)] = 1.0
    blocks[:, :64, :64] = np.tril(G, -1) + np.tril(G, -1).transpose(0, 2, 1)
    blocks[:, np.arange(64), np.arange(64)] = rng.uniform(1.5, 1.9, (m, 64))
    X = blocks[:, :64, :64].astype(np.longdouble)
    for j in range(k):
        col = X[:, j + 1:, j].copy()
        X[:, j + 1:, j + 1:] -= col[:, :, None] * (col / X[:, j, j][:, None])[:, None, :]
    want = X[:, k, k]
    assert want.min() > 1.0 and want.max() < 2.0
    L, d = factor(blocks, ldlt, False)
    have = d[:, k] if ldlt else L[:, k, k].astype(np.longdouble) ** 2
    rms = 2.0 ** 52 * float(np.sqrt(np.mean((have - want) ** 2)))
    # the stored square root's rounding: variance 2^-104 / 12, times (2 sqrt(p))^2 in its square
    assert rms <= np.sqrt(1.6 ** 2 + (0 if ldlt else 4 * 1.9 / 12))
