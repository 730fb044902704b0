"""Performance cases of the multifrontal numeric phase.

A case is one pass that a user's program makes over and over: new values of a
matrix whose pattern was analysed once, factored and solved on the handle
that the program keeps for that pattern (value refresh, or one request of a
served stream), or one more block of right-hand sides against a kept factor.
Most cases take the device-resident calls of the C ABI (values and right-hand
sides already in HBM, as ``bench.py`` does); the ``host`` ones take the Python
objects with host arrays.

Keys of a case: ``kind`` (pattern: ``grid2d`` 5-point, ``grid3d`` 7-point,
``kkt`` quasidefinite, ``batch`` of 9-point grids), ``nx, ny, nz`` (or
``side`` / ``count``), ``nrhs``, ``mixed`` (single-precision fronts with FP64
refinement; else FP64 throughout), ``op`` (``factor_solve``, ``solve``,
``host``).
"""
import ctypes
import functools
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "cliquetrees.jl_b200"))
import multifrontal as mf  # noqa: E402
from multifrontal import _native, testmatrices as tm  # noqa: E402
from multifrontal.batch import block_symbolic  # noqa: E402
from multifrontal.sparse import lower_triangle  # noqa: E402

TOL, MAXIT = 1e-12, 100  # the library's default backward error and step limit


def _g2(name, nx, ny, nrhs, mixed, op="factor_solve"):
    return {"name": name, "kind": "grid2d", "nx": nx, "ny": ny, "nz": 1, "nrhs": nrhs, "mixed": mixed, "op": op}


def _g3(name, nx, ny, nz, nrhs, mixed, op="factor_solve"):
    return {"name": name, "kind": "grid3d", "nx": nx, "ny": ny, "nz": nz, "nrhs": nrhs, "mixed": mixed, "op": op}


def listed():
    return [
        # the smallest call: a few hundred unknowns, where launches and host work are all there is
        _g2("2d 24x24 fp64", 24, 24, 1, False),
        # one small system through the Python objects with host arrays (the smallest served pattern)
        _g2("2d 64x64 fp64 host", 64, 64, 1, False, "host"),
        # the benchmark's plain 2D system
        _g2("2d 100x100 fp64", 100, 100, 1, False),
        # the largest served 2D pattern: long thin elimination tree, narrow fronts at the top
        _g2("2d 512x512 mixed", 512, 512, 4, True),
        # small 3D system with a full block of right-hand sides
        _g3("3d 16x16x16 fp64 16rhs", 16, 16, 16, 16, False),
        # the largest served 3D pattern, odd sides
        _g3("3d 47x49x45 mixed", 47, 49, 45, 3, True),
        # more right-hand sides against a kept factor (time stepping, sensitivities)
        _g3("3d 48x48x48 fp64 solve", 48, 48, 48, 8, False, "solve"),
        # the benchmark's large 3D system in both forms
        _g3("3d 80x80x80 fp64", 80, 80, 80, 4, False),
        _g3("3d 80x80x80 mixed", 80, 80, 80, 4, True),
        # many independent small systems as one forest
        {"name": "batch 512 mixed", "kind": "batch", "count": 512, "nrhs": 4, "mixed": True, "op": "factor_solve"},
        # quasidefinite LDLt: a few very large dense fronts under many tiny ones
        {"name": "kkt 24 fp64", "kind": "kkt", "side": 24, "nrhs": 8, "mixed": False, "op": "factor_solve"},
        {"name": "kkt 24 mixed", "kind": "kkt", "side": 24, "nrhs": 8, "mixed": True, "op": "factor_solve"},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["grid2d", "grid2d", "grid3d", "grid3d", "batch", "kkt"])
    mixed = rng.random() < 0.5
    nrhs = rng.randint(1, 16)
    if kind == "grid2d":
        op = rng.choice(["factor_solve", "factor_solve", "host", "solve"])
        nx, ny = _log_int(rng, 16, 512), _log_int(rng, 16, 512)
        c = _g2("", nx, ny, nrhs, mixed, op)
    elif kind == "grid3d":
        op = rng.choice(["factor_solve", "factor_solve", "solve"])
        c = _g3("", *(_log_int(rng, 8, 60) for _ in range(3)), nrhs, mixed, op)
    elif kind == "batch":
        c = {"kind": "batch", "count": _log_int(rng, 16, 512), "nrhs": nrhs, "mixed": mixed, "op": "factor_solve"}
    else:
        c = {"kind": "kkt", "side": _log_int(rng, 8, 24), "nrhs": min(nrhs, 8), "mixed": mixed, "op": "factor_solve"}
    c.pop("name", None)
    return c


# -- inputs ------------------------------------------------------------------

def _sides(count):
    r = random.Random(count)
    return [r.randint(8, 48) for _ in range(count)]


def _members(case, seed):
    """The matrices of a case with the seed's values (one, or a batch's)."""
    k = case["kind"]
    if k in ("grid2d", "grid3d"):
        # log-uniform [0.1, 10] edge weights, diagonal = row sum + 1e-2
        return [tm.grid_laplacian(case["nx"], case["ny"], case["nz"], stencil=5 if k == "grid2d" else 7, seed=seed)]
    if k == "batch":
        return [tm.config3_matrix(s, 100003 * seed + i) for i, s in enumerate(_sides(case["count"]))]
    # the constraint block keeps its pattern (and so the handle); its values
    # and H's are scaled by the seed's congruence D K D below
    K = tm.config4(side=case["side"], m=max(8, 16000 * case["side"] ** 3 // 64000), delta=1e-2, seed=4).tocsc()
    d = np.exp(np.random.default_rng(seed).uniform(-0.5, 0.5, K.shape[0]))
    K.data *= d[K.indices] * np.repeat(d, np.diff(K.indptr))
    return [K]


def _lower_values(mats):
    """The stored lower-triangle values in the order the handle expects
    (a block-diagonal matrix's are its members', one after the other)."""
    return np.concatenate([lower_triangle(A).data for A in mats])


def _rhs(n, nrhs, seed):
    return np.asfortranarray(np.random.default_rng([seed, 1]).standard_normal((n, nrhs)))


def _order(case):
    if case["kind"] == "grid3d":
        return mf.grid_nd_order(case["nx"], case["ny"], case["nz"])
    return "amf"


def _key(case):
    return tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "nrhs", "op", "mixed")))


@functools.lru_cache(maxsize=4)
def _symbolic(key):
    """Pattern analysis, once per pattern (as every program does)."""
    case = dict(key)
    mats = _members(case, 0)
    parts = [mf.symbolic(A, alg=_order(case)) for A in mats]
    return block_symbolic(parts) if case["kind"] == "batch" else (*parts[0], None)


class _Handle:
    """A kept handle: pattern, plan and device storage, on its own stream."""

    def __init__(self, case, mats):
        P, S, offsets = _symbolic(_key(case))
        cls = mf.ChordalLDLt if case["kind"] == "kkt" else mf.ChordalCholesky
        A = mats[0] if len(mats) == 1 else _block_diag(mats)
        self.F = cls(A, P, S, mixed=bool(case["mixed"]))
        self.lib, self.h, self.n = self.F._handle.lib, self.F._handle.h, S.n
        if offsets is not None:
            _native.check(self.lib.mf_set_segments(self.h, len(offsets) - 1, _native.ptr64(offsets)),
                          "mf_set_segments")
        self.perm = torch.from_numpy(np.ascontiguousarray(P.perm, dtype=np.int64)).cuda()
        self.stream = torch.cuda.Stream()
        if case["op"] != "host":
            _native.check(self.lib.mf_set_stream(self.h, ctypes.c_void_p(self.stream.cuda_stream)), "mf_set_stream")


def _block_diag(mats):
    """Block-diagonal CSC matrix of the members."""
    off = np.concatenate([[0], np.cumsum([A.shape[0] for A in mats])])
    nz = np.concatenate([[0], np.cumsum([A.nnz for A in mats])])
    data = np.concatenate([A.data for A in mats])
    idx = np.concatenate([A.indices + off[i] for i, A in enumerate(mats)])
    ptr = np.concatenate([[0]] + [A.indptr[1:] + nz[i] for i, A in enumerate(mats)])
    return type(mats[0])((data, idx, ptr), shape=(int(off[-1]), int(off[-1])))


_kept = {}


def _handle(case, mats):
    """The handle of this pattern, kept by the program across new values; a
    solve-only state has one of its own, which holds its factor."""
    if case["op"] == "solve":
        return _Handle(case, mats)
    key = (_key(case), case["mixed"], case["op"])
    if key not in _kept:
        _kept.clear()
        _kept[key] = _Handle(case, mats)
    return _kept[key]


class _State:
    pass


def prepare(case, seed):
    mats = _members(case, seed)
    s = _State()
    s.case = case
    s.H = _handle(case, mats)
    s.values = np.ascontiguousarray(_lower_values(mats))
    B = _rhs(s.H.n, case["nrhs"], seed)
    if case["op"] == "host":
        s.B = B
        return s
    s.nz = torch.from_numpy(s.values).cuda()
    s.B = torch.from_numpy(B.ravel(order="F")).cuda()
    s.X = torch.empty_like(s.B)
    torch.cuda.synchronize()
    if case["op"] == "solve":
        _factor(s)
        torch.cuda.synchronize()
    return s


# -- one pass ----------------------------------------------------------------

def _factor(s):
    H = s.H
    lib, vp = H.lib, ctypes.c_void_p
    _native.check(lib.mf_assemble_device(H.h, vp(s.nz.data_ptr())), "mf_assemble_device")
    if s.case["mixed"]:
        info, fp64 = ctypes.c_int64(0), ctypes.c_int(0)
        _native.check(lib.mf_factorize_mixed(H.h, None, ctypes.byref(info), ctypes.byref(fp64)), "mf_factorize_mixed")
        if info.value:
            raise RuntimeError("factorization failed")
    else:
        _native.check(lib.mf_factorize(H.h, None, None), "mf_factorize")


def _solve(s):
    H = s.H
    lib, vp, k = H.lib, ctypes.c_void_p, s.case["nrhs"]
    with torch.cuda.stream(H.stream):
        s.X.copy_(s.B)
    if s.case["mixed"]:
        it, eta = ctypes.c_int(0), ctypes.c_double(0.0)
        _native.check(lib.mf_solve_refined_device(H.h, vp(s.X.data_ptr()), k, H.n, vp(H.perm.data_ptr()), TOL, MAXIT,
                                                  ctypes.byref(it), ctypes.byref(eta)), "mf_solve_refined_device")
    else:
        _native.check(lib.mf_solve_device(H.h, vp(s.X.data_ptr()), k, H.n, vp(H.perm.data_ptr())), "mf_solve_device")


def run(state):
    s = state
    if s.case["op"] == "host":
        F = s.H.F
        F.refresh(s.values)
        mf.cholesky_(F)
        return mf.ldiv(F, s.B)
    if s.case["op"] == "factor_solve":
        _factor(s)
    _solve(s)
    return s.X


# -- what a pass cannot do without -------------------------------------------

def work(case):
    """Flops of the factorization and of the two triangular solves; bytes of
    the values, right-hand sides and solution, plus the factor: written once
    when it is made, read by each of the two sweeps of a solve-only pass."""
    P, S, _ = _symbolic(_key(case))
    nn, na = np.diff(S.resptr).astype(np.float64), np.diff(S.sepptr).astype(np.float64)
    k = case["nrhs"]
    entries = float((nn * (nn + 1) / 2 + nn * na).sum())
    nnz = sum(lower_triangle(A).nnz for A in _members(case, 0))
    w = 4 if case["mixed"] else 8
    io = 16.0 * S.n * k
    if case["op"] == "solve":
        return {"bytes": io + 2 * w * entries, "flops": 4.0 * entries * k}
    flops = float((nn ** 3 / 3 + nn * nn * na + nn * na * na).sum())
    return {"bytes": 8.0 * nnz + io + w * entries, "flops": flops + 4.0 * entries * k}


# -- the answer in 64 bits ---------------------------------------------------

def exact(case, seed):
    mats = _members(case, seed)
    A = mats[0] if len(mats) == 1 else _block_diag(mats)
    n = A.shape[0]
    B = torch.from_numpy(_rhs(n, case["nrhs"], seed)).cuda()
    M = torch.sparse_csr_tensor(torch.from_numpy(A.indptr.astype(np.int64)), torch.from_numpy(A.indices.astype(np.int64)),
                                torch.from_numpy(A.data), (n, n)).cuda()
    X = _dense_solve(M, B) if case["kind"] == "kkt" else _cg(M, B, torch.from_numpy(A.diagonal()).cuda())
    if case["op"] == "host":
        X = X.cpu().numpy()
        return X
    return X.t().contiguous().reshape(-1)


def _dense_solve(M, B):
    D = M.to_dense()
    LU, piv = torch.linalg.lu_factor(D)
    X = torch.linalg.lu_solve(LU, piv, B)
    for _ in range(2):
        X = X + torch.linalg.lu_solve(LU, piv, B - D @ X)
    return X


def _cg(M, B, diag):
    """Jacobi-preconditioned conjugate gradients on every column, restarted
    from the true residual until it stops falling."""
    X, best = torch.zeros_like(B), None
    w = (1.0 / diag).unsqueeze(1)
    for _ in range(8):
        R = B - M @ X
        now = float((R.norm(dim=0) / B.norm(dim=0)).max())
        if best is not None and now > 0.25 * best:
            break
        best = now
        scale = R.norm(dim=0)
        Z = w * R
        Q, rz, dX = Z.clone(), (R * Z).sum(0), torch.zeros_like(B)
        for it in range(6000):
            AQ = M @ Q
            a = rz / (Q * AQ).sum(0).clamp_min(1e-300)
            dX += a * Q
            R -= a * AQ
            Z = w * R
            new = (R * Z).sum(0)
            Q = Z + (new / rz.clamp_min(1e-300)) * Q
            rz = new
            if it % 50 == 49 and bool((R.norm(dim=0) <= 1e-14 * scale).all()):
                break
        X = X + dX
    return X
