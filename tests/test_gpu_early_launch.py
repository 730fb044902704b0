"""Factorizations whose short launches start before the launch ahead of them
has finished (MF_PANEL_PDL=1, the default) against stream-ordered launches
(MF_PANEL_PDL=0), as graphs and as direct launches (MF_GRAPHS=0).  The kernels
and the order of every sum are the same, so factors and solutions must be
bitwise equal, on a first factorization and on ones with new values, which
find another matrix's pivots and panels in every cache.  The members'
widths put a front's first column (and so its pivots) at any place in a cache
line and give fronts of one to nine 64-column sub-panels, last blocks of
one column, of an odd width and full ones, with rows below them and without.

Queued passes: assembly, factorization and solve of alternating values with
no synchronisation in between, as graphs and as direct launches.  The first
launch of a factorization or solve waits for all that was queued before it,
so each pass must give what it gives by itself."""
import ctypes

import numpy as np
import pytest
import scipy.sparse as sp
import torch

import multifrontal as mf
from multifrontal import testmatrices as tm
from multifrontal._native import check
from multifrontal.sparse import lower_triangle

from test_gpu_elimination import two_cliques

pytestmark = pytest.mark.gpu

MEMBERS = [(321, 190, 65), (7, 5, 3), (129, 97, 31), (513, 257, 2), (50, 30, 9), (256, 131, 64), (41, 66, 77)]


def forest(ldlt, seed):
    return sp.block_diag([two_cliques(a, b, s, ldlt, seed=seed + a) for a, b, s in MEMBERS], format="csc")


def passes(A0, A1, P, S, B, ldlt, mixed):
    F = (mf.ChordalLDLt if ldlt else mf.ChordalCholesky)(A0, P, S, mixed=mixed)
    out = []
    for A in (A0, A1, A0, A1):
        F.refresh(lower_triangle(A).data)
        (mf.ldlt_ if ldlt else mf.cholesky_)(F)
        assert not F.used_fp64
        out.append((*(F.factor_arrays_mixed() if mixed else F.factor_arrays()), mf.ldiv(F, B)))
    F.close()
    return out


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("ldlt", [False, True])
def test_early_launches_equal_stream_order(monkeypatch, ldlt, mixed):
    A0, A1 = forest(ldlt, 100), forest(ldlt, 900)
    P, S = mf.symbolic(A0, alg=np.arange(A0.shape[0]))
    B = tm.rhs(S.n, 3, seed=5)
    got = {}
    for pdl, graphs in (("0", "1"), ("1", "1"), ("1", "0")):
        monkeypatch.setenv("MF_PANEL_PDL", pdl)
        monkeypatch.setenv("MF_GRAPHS", graphs)
        got[pdl, graphs] = passes(A0, A1, P, S, B, ldlt, mixed)
    for how in (("1", "1"), ("1", "0")):
        for k, (want, have) in enumerate(zip(got["0", "1"], got[how])):
            for w, g in zip(want, have):
                assert np.array_equal(w, g), (how, k)
    for A, p in ((A0, 0), (A1, 1)):
        assert tm.backward_error(A, got["1", "1"][p][-1], B).max() <= (1e-12 if mixed else 1e-13)
        for w, g in zip(got["1", "1"][p], got["1", "1"][p + 2]):
            assert np.array_equal(w, g)


@pytest.mark.parametrize("graphs", ["1", "0"])
@pytest.mark.parametrize("ldlt", [False, True])
def test_queued_passes_equal_single_ones(monkeypatch, ldlt, graphs):
    monkeypatch.setenv("MF_GRAPHS", graphs)
    mats = [forest(ldlt, 100), forest(ldlt, 900)]
    P, S = mf.symbolic(mats[0], alg=np.arange(mats[0].shape[0]))
    F = (mf.ChordalLDLt if ldlt else mf.ChordalCholesky)(mats[0], P, S)
    lib, h, vp = F._handle.lib, F._handle.h, ctypes.c_void_p
    stream = torch.cuda.Stream()
    check(lib.mf_set_stream(h, vp(stream.cuda_stream)), "mf_set_stream")
    nz = [torch.from_numpy(np.ascontiguousarray(lower_triangle(A).data)).cuda() for A in mats]
    B = torch.from_numpy(tm.rhs(S.n, 3, seed=6).ravel(order="F").copy()).cuda()
    perm = torch.from_numpy(np.ascontiguousarray(P.perm, dtype=np.int64)).cuda()
    X = [B.clone() for _ in range(6)]
    torch.cuda.synchronize()

    def one(values, x):
        check(lib.mf_assemble_device(h, vp(values.data_ptr())), "mf_assemble_device")
        check(lib.mf_factorize(h, None, None), "mf_factorize")
        check(lib.mf_solve_device(h, vp(x.data_ptr()), 3, S.n, vp(perm.data_ptr())), "mf_solve_device")

    want = []
    for values in nz:
        x = B.clone()
        torch.cuda.synchronize()
        one(values, x)
        torch.cuda.synchronize()
        want.append(x)
    for k, x in enumerate(X):
        one(nz[k % 2], x)
    torch.cuda.synchronize()
    for k, x in enumerate(X):
        assert torch.equal(x, want[k % 2]), k
    for A, x in zip(mats, want):
        x = x.cpu().numpy().reshape(3, S.n).T
        assert tm.backward_error(A, x, B.cpu().numpy().reshape(3, S.n).T).max() <= 1e-13
    F.close()


@pytest.mark.parametrize("nrhs", [2, 8, 16])
def test_solves_of_wide_levels_equal_stream_order(monkeypatch, nrhs):
    """48^3: levels whose forward gather has fewer CTAs than SMs and levels
    where it has more, with vectors narrow and wide (both launch rules)."""
    A = tm.grid_laplacian(48, 48, 48, seed=74)
    P, S = mf.symbolic(A, alg=mf.grid_nd_order(48, 48, 48))
    B = tm.rhs(S.n, nrhs, seed=15)
    X = {}
    for v in ("0", "1"):
        monkeypatch.setenv("MF_STEP_PDL", v)
        F = mf.cholesky_(mf.ChordalCholesky(A, P, S))
        X[v] = mf.ldiv(F, B)
        F.close()
    assert np.array_equal(X["0"], X["1"])
    assert tm.backward_error(A, X["1"], B).max() <= 1e-13
