// Numeric factorization kernels (FP64) for the B200 multifrontal solver.
//
// Per tree level (see mf_plan.cu):
//   k_small   : fronts with nj <= kSmallMax.  One CTA holds the whole frontal
//               matrix: load the assembled panel, extend-add the children's
//               update matrices, partial LDL^T/Cholesky of the first nn
//               columns, write panel + update matrix.  This fuses
//               chol_loop_snd!/chol_loop_nod! (cholesky.jl:434-692) for the
//               many tiny fronts of a maximal-supernode tree.
//   k_ea      : extend-add for larger fronts, one CTA per (front, 16 parent
//               columns, 1024 parent rows); each CTA owns its target entries,
//               so the children are added in a fixed order without atomics
//               (addscattertri!, utils.jl:555-579 via chol_send!,
//               cholesky.jl:950-983).  The panel columns are done before the
//               front is factored, the update-matrix columns after the SYRK.
//   k_diag    : per 64-column sub-panel, one CTA per front factors the
//               diagonal block in shared memory, writes it back and stores
//               the inverse of the factored block (potrf! of chol_factor!,
//               cholesky.jl:694-737);
//   k_gemm64  : grouped DMMA (mma.sync m8n8k4 f64) tile GEMM, 128 x 64 or
//               64 x 64 tiles (FP32: mf_tc.cu, or k_gemm), in four roles: left-looking
//               update of a sub-panel from its outer block, trailing update
//               of the panel after an outer block (K = 256), the TRSM of a
//               sub-panel as a product with the inverse of its diagonal
//               block, and M = -L21 D L21^T with K = nn (syrk!,
//               blas/syrk.jl:137-159; the children's F22 is added to M
//               after it, which reorders the reference's sum F22 - L21 L21^T).
#include <climits>
#include <cstdio>
#include <type_traits>

#include "mf_internal.cuh"

namespace mf {

// ---------------------------------------------------------------------------
// helpers
// ---------------------------------------------------------------------------

// pivot acceptance of NoRegularization (no_regularization.jl:27-42):
// a pivot whose sign disagrees with a nonzero requested sign is rejected,
// and a zero pivot is always rejected.
__device__ __forceinline__ bool pivot_ok(double s, double p) {
    if (s != 0.0 && !(s * p > 0.0)) return false;
    return p != 0.0;
}

__device__ __forceinline__ double reg_pivot(const Reg& r, double s, double p) {
    return (s * p < r.eps) ? r.delta * s : p;
}

__device__ __forceinline__ double pivot_sign(const double* signs, int ldlt, int64_t col) {
    if (!ldlt) return 1.0;
    return signs ? signs[col] : 0.0;
}

__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(c0), "+d"(c1)
                 : "d"(a), "d"(b));
}

// ---------------------------------------------------------------------------
// assembly and layout conversion
// ---------------------------------------------------------------------------

template <typename T>
__global__ void k_scatter(T* __restrict__ P, const int64_t* __restrict__ slot, const double* __restrict__ v,
                          int64_t nnz, const int32_t* __restrict__ rowi, const int32_t* __restrict__ coli,
                          const double* __restrict__ scale) {
    pdl_prologue();
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (; i < nnz; i += stride) {
        double x = v[i];
        if (scale) x *= scale[rowi[i]] * scale[coli[i]];
        P[slot[i]] = (T)x;
    }
}

// scale[i] = 1/sqrt(|a_ii|) (1 where a_ii = 0) from the assembled values
__global__ void k_diag_scale(double* __restrict__ scale, const int64_t* __restrict__ dslot,
                             const double* __restrict__ v, int64_t n) {
    pdl_prologue();
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    int64_t k = dslot[i];
    double a = k >= 0 ? fabs(v[k]) : 0.0;
    scale[i] = a > 0.0 ? 1.0 / sqrt(a) : 1.0;
}

// one warp per column: copy between the reference layout (Dval nn x nn,
// Lval na x nn of reference front j) and the panel of the execution front
// that holds j (nj x nn, ld nj): the D rows keep their order, the L rows go
// to sepmap positions.
template <bool TO_PANEL>
__global__ void k_dl_panel(const Front* __restrict__ fronts, const RefFront* __restrict__ ref,
                           const int32_t* __restrict__ colref, const int32_t* __restrict__ sepmap,
                           double* __restrict__ Dv, double* __restrict__ Lv, double* __restrict__ P, int64_t n) {
    pdl_prologue();
    int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    int lane = threadIdx.x & 31;
    if (warp >= n) return;
    const RefFront rf = ref[colref[warp]];
    const Front f = fronts[rf.exec];
    const int c = (int)(warp - rf.res0);
    const int off = rf.res0 - f.col0;
    double* pc = P + f.poff + (int64_t)(off + c) * f.ldp;
    double* dc = Dv + rf.Dptr + (int64_t)c * rf.nn;
    double* lc = Lv + rf.Lptr + (int64_t)c * rf.na;
    const int32_t* map = sepmap + rf.sep0;
    for (int r = lane; r < rf.nn; r += 32) {
        if (TO_PANEL) pc[off + r] = dc[r]; else dc[r] = pc[off + r];
    }
    for (int r = lane; r < rf.na; r += 32) {
        if (TO_PANEL) pc[map[r]] = lc[r]; else lc[r] = pc[map[r]];
    }
}

// single-precision panels -> reference layout (mixed-mode factor download)
__global__ void k_panel32_to_dl(const Front* __restrict__ fronts, const RefFront* __restrict__ ref,
                                const int32_t* __restrict__ colref, const int32_t* __restrict__ sepmap,
                                double* __restrict__ Dv, double* __restrict__ Lv, const float* __restrict__ P,
                                int64_t n) {
    pdl_prologue();
    int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    int lane = threadIdx.x & 31;
    if (warp >= n) return;
    const RefFront rf = ref[colref[warp]];
    const Front f = fronts[rf.exec];
    const int c = (int)(warp - rf.res0);
    const int off = rf.res0 - f.col0;
    const float* pc = P + f.poff + (int64_t)(off + c) * f.ldp;
    double* dc = Dv + rf.Dptr + (int64_t)c * rf.nn;
    double* lc = Lv + rf.Lptr + (int64_t)c * rf.na;
    const int32_t* map = sepmap + rf.sep0;
    for (int r = lane; r < rf.nn; r += 32) dc[r] = pc[off + r];
    for (int r = lane; r < rf.na; r += 32) lc[r] = pc[map[r]];
}

// ---------------------------------------------------------------------------
// small fronts: whole frontal matrix in shared memory
// ---------------------------------------------------------------------------
// Thresholds of the single-precision factorization's pivot check (mixed form,
// whose matrix is scaled to unit diagonal): a pivot that lost more than five
// of FP32's seven digits to cancellation against its diagonal entry, or grew
// beyond 1e7 times the largest diagonal entry of its block, flags the front
// (or 64 x 64 diagonal block), which is then factored again in FP64.
constexpr double kRescueSmall = 1e-5;
constexpr double kRescueGrowth = 1e7;
constexpr int kSmallKids = 16;  // children whose records k_small fetches up front

// The reciprocal ik that scales the column of an accepted pivot p: one over the
// stored diagonal entry (sqrt(p) for Cholesky, p for LDLt), both correctly
// rounded.  BLOCK, single-precision Cholesky: the hardware's reciprocal square
// root (rsqrtf, at most 2 ulp) in the diagonal blocks, whose factor only
// preconditions the FP64 refinement and whose pivots are one long chain.
template <int LDLT, bool BLOCK, typename TC>
__device__ __forceinline__ TC pivot_recip(TC p) {
    if (BLOCK && !LDLT && sizeof(TC) == 4) return rsqrtf((float)p);
    return TC(1) / (LDLT ? p : sqrt(p));
}
template <typename TC, int LDLT>
__device__ __forceinline__ TC pivot_stored(TC p) {
    return LDLT ? p : sqrt(p);
}

// ---------------------------------------------------------------------------
// Elimination of the first `nel` columns of a symmetric matrix of at most
// NR = TD * R rows by one CTA of TD x TD threads: k_small's partial
// factorization and k_diag's block with its inverse.  Thread (tx, ty) holds
// the entries (tx + TD i, ty + TD j), i >= j, in registers; columns go four
// at a time:
//   publish  the owners of columns k .. k + 3 write them to shared memory;
//   solve    thread t < NR factors the 4 x 4 pivot block (every one the same,
//            in registers) and solves row t's four entries against it; they go
//            to F and, as one quad a row, to lb (LDLt: times the pivots to rq,
//            the right factor);
//   update   every thread subtracts the four rank-1 products from its
//            entries: one by one, columns in order, in k_small; as one sum of
//            four in k_diag.  Entries of finished rows and columns take junk:
//            nothing reads them again.
// The pivots are checked, and the diagonal stored, after the last quad.
// INV: the same steps applied to the identity give X = L^-1 (unit diagonal
// for LDLt) in the registers of the finished columns: a second group of NR
// threads solves X's four pivot rows beside the row group, one column each,
// into rq and X, and the update is the same for A's and X's entries.
// What bounds it is the chain of pivots (square root and reciprocal, scale and
// update within the quad, two barriers around it), then shared-memory reads of
// the quads in the update (two rows a warp: 128 bytes a cycle and SM).  So
// nothing else is on the chain, its code is straight-line, and one rolled
// loop of a few hundred instructions serves all quads: a CTA runs it once, and
// its instructions come from L2.  64 x 64 block with its inverse, one CTA, per
// launch (medians over the blocks of a 1,024-column front): FP64 Cholesky 36 ->
// 23 us, LDLt 36 -> 21 us, FP32 17.7 -> 12.3 us and 21.7 -> 14.9 us (before:
// panels of sixteen columns factored by one warp's shuffles, the inverse after
// them).  A small front's launch in a narrow level: 44 -> 12 to 16 us (before: a
// right-looking loop in shared memory, two divisions an entry, a barrier a
// column and a memory trip a child).
// Measured slower: the matrix in shared memory instead of registers (29 us for
// the FP64 LDLt block: aliased loads and stores wait for one another), the
// panel one quad ahead of the update in warps of its own (26 us: the panel
// threads then redo part of the update), a copy of the step per 16 columns
// (23 us: instruction fetches).
// Each entry gets the right-looking order's operations, whatever TD and R are.
// The sums of four keep k_diag's error at that of the panels of sixteen it
// replaced: a 64-column block's last pivots take 18 roundings of their own size
// then, not 63.  Solutions of 47 x 49 x 45 mixed come out 6.9e-14 (relative, ten
// sets of values) from the exact ones, 7.1e-14 with those panels; products
// subtracted one by one gave 1.4 times as much, there and at 80^3 mixed.
// ---------------------------------------------------------------------------
template <typename TC>
struct __align__(16) Quad {
    TC v[4];
};

// shared-memory scratch of eliminate()
template <typename TC, int NR, bool INV>
struct __align__(16) ElimBufs {
    Quad<TC> lb[NR + 1], rq[NR];
    TC cb[4 * NR];
    TC xb[INV ? 4 * NR : 1];
    TC diag0[NR];    // |a_kk| on entry (single-precision pivot check)
    TC piv[NR + 4];  // pivots, then stored diagonal entries
    double sgn[NR];  // requested pivot signs (LDLt)
    int bad;
};

template <typename TC, int LDLT, int TD, int R, bool INV, bool REG>
__device__ __forceinline__ int eliminate(TC (&a)[R][R], int nrow, int nel, TC* F, int ldf, TC* X, int ldx,
                                         ElimBufs<TC, TD * R, INV>& s, const Reg& reg, bool check, int* flag) {
    constexpr int NR = TD * R;
    static_assert(TD * TD >= (INV ? 2 : 1) * NR, "one thread per row (and per inverse column)");
    const int tid = threadIdx.x, tx = tid % TD, ty = tid / TD;
    if (tid == 0) s.bad = INT_MAX;
#pragma unroll 1
    for (int k = 0; k < nel; k += 4) {
        const int jb = k / TD, kk = k % TD, nc = nel - k;  // columns of the quad past nc take pivot 1 and zero factors
        {
            const int c = ty - kk, r = tx - kk;
#pragma unroll
            for (int j = 0; j < R; ++j)
                if (j == jb) {  // uniform
                    if (c >= 0 && c < 4)
#pragma unroll
                        for (int i = j; i < R; ++i) {
                            s.cb[c * NR + tx + TD * i] = a[i][j];
                            if (INV) a[i][j] = TC(0);
                        }
                    if (INV && r >= 0 && r < 4)
#pragma unroll
                        for (int j2 = 0; j2 <= j; ++j2) s.xb[INV ? r * NR + ty + TD * j2 : 0] = a[j][j2];
                }
        }
        __syncthreads();
        if (tid < (INV ? 2 : 1) * NR) {
            // straight-line: a branch in here would sit on the pivot chain
            const bool row = !INV || tid < NR;
            const int t = row ? tid : tid - NR;
            TC p[4][4], v[4], raw[4];
#pragma unroll
            for (int c = 0; c < 4; ++c)
#pragma unroll
                for (int r = c; r < 4; ++r) p[r][c] = s.cb[c * NR + k + r];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                v[c] = INV && !row ? s.xb[INV ? c * NR + t : 0] : s.cb[c * NR + t];
                if (INV && !row && t >= k) v[c] = t == k + c ? TC(1) : TC(0);
            }
            Quad<TC> q, q2;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                TC piv = p[c][c];
                if (REG) piv = (TC)reg_pivot(reg, LDLT ? s.sgn[min(k + c, NR - 1)] : 1.0, (double)piv);
                if (c > 0) piv = c < nc ? piv : TC(1);
                raw[c] = piv;
                // after a rejected pivot the remaining steps run on junk and are discarded
                const TC ik = pivot_recip<LDLT, INV>(piv);
                TC lv = (LDLT && INV && !row) ? v[c] : v[c] * ik;
                if (c > 0) lv = c < nc ? lv : TC(0);
#pragma unroll
                for (int r = c + 1; r < 4; ++r) p[r][c] *= ik;
#pragma unroll
                for (int c2 = c + 1; c2 < 4; ++c2) {
                    const TC l = p[c2][c];
                    const TC lc = LDLT ? l * piv : l;
#pragma unroll
                    for (int r = c2; r < 4; ++r) p[r][c2] -= p[r][c] * lc;
                    v[c2] -= lv * ((LDLT && INV && !row) ? l : lc);
                }
                q.v[c] = lv;
                if (LDLT) q2.v[c] = lv * piv;
            }
            s.lb[INV && !row ? NR : t] = q;  // (the inverse's threads write a spare slot)
            if (INV) {
                // right factors: the inverse's rows in finished columns, the factor's in the rest
                if (row == (t >= k + 4)) s.rq[t] = (LDLT && row) ? q2 : q;
            } else if (LDLT) {
                s.rq[t] = q2;
            }
            if (row) {
                if (t > k + 3 && t < nrow) {
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        if (c < nc) F[t + (k + c) * ldf] = q.v[c];
                } else if (t < nrow) {  // the quad's own rows
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        if (c < nc && t > k + c) F[t + (k + c) * ldf] = q.v[c];
                }
            } else if (t < k + 4) {
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if (c < nc && t <= k + c) X[(k + c) + t * ldx] = q.v[c];
            }
            if (tid == 0)
#pragma unroll
                for (int c = 0; c < 4; ++c) s.piv[k + c] = raw[c];
        }
        __syncthreads();
        Quad<TC> lr[R];
#pragma unroll
        for (int i = 0; i < R; ++i) lr[i] = s.lb[tx + TD * i];
#pragma unroll
        for (int j = 0; j < R; ++j) {
            if (INV || j >= jb) {  // uniform
                const Quad<TC> u = (LDLT || INV) ? s.rq[ty + TD * j] : s.lb[ty + TD * j];
#pragma unroll
                for (int i = j; i < R; ++i) {
                    if (INV) {
                        TC t = lr[i].v[0] * u.v[0];
#pragma unroll
                        for (int c = 1; c < 4; ++c) t += lr[i].v[c] * u.v[c];
                        a[i][j] -= t;
                    } else {
#pragma unroll
                        for (int c = 0; c < 4; ++c) a[i][j] -= lr[i].v[c] * u.v[c];
                    }
                }
            }
        }
    }
    __syncthreads();
    // the pivots: the first rejected one, and the stored diagonal
    if (tid < nel) {
        const TC piv = s.piv[tid];
        const double sg = LDLT ? s.sgn[tid] : 1.0;
        const bool bad = REG ? piv == TC(0) : !pivot_ok(sg, (double)piv) || (!LDLT && !(piv > TC(0)));
        if (bad) atomicMin(&s.bad, tid);
        const TC dk = pivot_stored<TC, LDLT>(piv);
        F[tid + tid * ldf] = dk;
        s.piv[tid] = dk;
        if (check) {
            const double a0 = (double)s.diag0[tid], ap = fabs((double)piv);
            if (ap < kRescueSmall * a0 || ap > kRescueGrowth * fmax(a0, 1.0)) *flag = 1;
        }
    }
    __syncthreads();
    return s.bad == INT_MAX ? -1 : s.bad;
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}

// A small front assembled in shared memory (F, leading dimension f.ldp): the
// panel, zeros in the update part, then the children in the reference's
// reverse order (cholesky.jl:506-514).  The panel and every child's update
// matrix are contiguous 16-byte-aligned blocks (leading dimensions and
// offsets are multiples of four entries), so they stream into shared memory
// as 16-byte asynchronous copies, as many children at a time as `stage`
// entries hold (at least the largest one), and the adds wait for one memory
// trip per group instead of one per child.  The panel (the assembled matrix)
// and the children's records come before the wait for the level below.  Ends
// with a block barrier.
template <typename T>
__device__ __forceinline__ void small_assemble(T* F, T* S, int stage, const Front& f,
                                               const Front* __restrict__ fronts, const int32_t* __restrict__ reltgt,
                                               const int32_t* __restrict__ chdtgt, const T* P, const T* M) {
    constexpr int V = 16 / (int)sizeof(T);
    const int nn = f.nn, nj = nn + f.na, ld = f.ldp;
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
    // the children's records, kSmallKids at a time, in the order they are added
    __shared__ int kid_na[kSmallKids], kid_lm[kSmallKids], kid_sep0[kSmallKids], kid_at[kSmallKids + 1];
    __shared__ int64_t kid_moff[kSmallKids];
    __shared__ int32_t kid_rel[kSmallKids * kSmallMax];
    __shared__ int kid_end;
    const int nch = f.chd1 - f.chd0;
    for (int i = V * tid; i < ld * nn; i += V * nt) cp_async16(F + i, P + f.poff + i);
    for (int i = ld * nn + tid; i < ld * nj; i += nt) F[i] = T(0);
    for (int k0 = 0; k0 < nch; k0 += kSmallKids) {
        const int m = min(kSmallKids, nch - k0);
        for (int q = tid; q < m; q += nt) {
            const Front fc = fronts[chdtgt[f.chd1 - 1 - k0 - q]];
            kid_na[q] = fc.na;
            kid_lm[q] = fc.ldm;
            kid_sep0[q] = fc.sep0;
            kid_moff[q] = fc.moff;
        }
        // the level below has written the children (and read what this front writes)
        if (k0 == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
        __syncthreads();
        for (int q0 = 0; q0 < m;) {
            if (tid == 0) {  // the children of this group and where they land
                int at = 0, q = q0;
                while (q < m && (q == q0 || at + kid_lm[q] * kid_na[q] <= stage)) {
                    kid_at[q] = at;
                    at += kid_lm[q] * kid_na[q];
                    ++q;
                }
                kid_end = q;
            }
            __syncthreads();
            const int q1 = kid_end;
            for (int q = q0; q < q1; ++q) {
                const int n = kid_lm[q] * kid_na[q];
                const T* src = M + kid_moff[q];
                T* dst = S + kid_at[q];
                for (int i = V * tid; i < n; i += V * nt) cp_async16(dst + i, src + i);
                const int32_t* rel = reltgt + kid_sep0[q];
                for (int i = tid; i < kid_na[q]; i += nt) cp_async4(kid_rel + q * kSmallMax + i, rel + i);
            }
            cp_async_wait_all();
            __syncthreads();
            for (int q = q0; q < q1; ++q) {
                const int ma = kid_na[q], lm = kid_lm[q];
                const int32_t* rel = kid_rel + q * kSmallMax;
                const T* Mc = S + kid_at[q];
                // a child's entries land on distinct entries of F, so a lane
                // reads four columns' worth before it writes the first
                for (int b0 = warp; b0 < ma; b0 += 4 * nw) {
                    int col[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) col[u] = b0 + u * nw < ma ? rel[b0 + u * nw] * ld : 0;
                    for (int r = (b0 & ~31) + lane; r < ma; r += 32) {
                        const int rr = rel[r];
                        T v[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const int b = b0 + u * nw;
                            v[u] = (b <= r && b < ma) ? F[col[u] + rr] + Mc[r + b * lm] : T(0);
                        }
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const int b = b0 + u * nw;
                            if (b <= r && b < ma) F[col[u] + rr] = v[u];
                        }
                    }
                }
                __syncthreads();
            }
            q0 = q1;
        }
    }
    if (nch == 0) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        cp_async_wait_all();
        __syncthreads();
    }
}

// The FP64 redo of a flagged single-precision small front (rare): assembled
// and factored right-looking in shared memory as doubles (F, leading
// dimension nj).  Returns the first rejected pivot (front-local) or -1,
// uniform across the block.
template <int LDLT>
__device__ __noinline__ int small_redo(double* F, const Front& f, const Front* __restrict__ fronts,
                                       const int32_t* __restrict__ reltgt, const int32_t* __restrict__ chdtgt,
                                       const float* __restrict__ P, const float* __restrict__ M,
                                       const double* __restrict__ signs) {
    const int nn = f.nn, nj = nn + f.na;
    const int tid = threadIdx.x, nt = blockDim.x;
    for (int i = tid; i < nj * nj; i += nt) {
        const int r = i % nj, c = i / nj;
        F[i] = c < nn ? (double)P[f.poff + r + (int64_t)c * f.ldp] : 0.0;
    }
    __syncthreads();
    for (int q = f.chd1 - 1; q >= f.chd0; --q) {
        const Front fc = fronts[chdtgt[q]];
        const int32_t* rel = reltgt + fc.sep0;
        for (int i = tid; i < fc.na * fc.na; i += nt) {
            const int a = i % fc.na, b = i / fc.na;
            if (a >= b) F[rel[a] + rel[b] * nj] += (double)M[fc.moff + a + b * fc.ldm];
        }
        __syncthreads();
    }
    for (int k = 0; k < nn; ++k) {
        const double piv = F[k + k * nj];
        const double s = pivot_sign(signs, LDLT, f.col0 + k);
        if (!pivot_ok(s, piv) || (!LDLT && !(piv > 0.0))) return k;  // uniform across the block
        const double inv = pivot_recip<LDLT, false>(piv);
        __syncthreads();
        if (tid == 0) F[k + k * nj] = pivot_stored<double, LDLT>(piv);
        for (int i = k + 1 + tid; i < nj; i += nt) F[i + k * nj] *= inv;
        __syncthreads();
        const int m = nj - k - 1;
        for (int i = tid; i < m * m; i += nt) {
            const int r = k + 1 + i % m, c = k + 1 + i / m;
            if (r >= c) {
                double lc = F[c + k * nj];
                if (LDLT) lc *= piv;
                F[r + c * nj] -= F[r + k * nj] * lc;
            }
        }
        __syncthreads();
    }
    return -1;
}

// Write a factored small front's panel (F, leading dimension lf) and LDLt
// pivots back (the panel diagonal holds them: the unit diagonal of L is
// implied).
template <typename TC, typename T, int LDLT>
__device__ __forceinline__ void small_panel_store(const TC* F, int lf, const Front& f, T* __restrict__ P,
                                                  T* __restrict__ d) {
    const int nn = f.nn, nj = nn + f.na;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int c = warp; c < nn; c += nw) {
        T* dst = P + f.poff + (int64_t)c * f.ldp;
        for (int r = c + lane; r < nj; r += 32) dst[r] = (T)F[r + c * lf];
    }
    if (LDLT)
        for (int k = threadIdx.x; k < nn; k += blockDim.x) d[f.col0 + k] = (T)F[k + k * lf];
}

// small fronts (nj <= kSmallMax): one CTA of TD x TD threads assembles the
// front in shared memory and eliminates it in registers (eliminate()).  Single precision: a
// front whose factorization rejects a pivot or flags a small or grown pivot
// is factored again from its inputs in FP64 in the same shared memory (fronts
// of nj <= kSmallRescue; the panel and the children's update matrices are
// only read before the final store, so the inputs are intact), and the FP64
// result is stored rounded to FP32.  A rejection in FP64 -- or in FP32 for a
// larger front -- is reported through info.
constexpr int kSmallRescue = 67;

template <typename T, int LDLT, int TD, int R, bool REG>
__global__ void __launch_bounds__(TD * TD) k_small(const Front* __restrict__ fronts, const Item* __restrict__ items,
                                                   int stage, const int32_t* __restrict__ reltgt,
                                                   const int32_t* __restrict__ chdtgt, T* P, T* M, T* d,
                                                   const double* __restrict__ signs, long long* __restrict__ info,
                                                   int* __restrict__ rescued, Reg reg) {
    pdl_trigger();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ ElimBufs<T, TD * R, false> s;
    __shared__ int flag;
    T* S = reinterpret_cast<T*>(smem_raw);  // staged children
    T* F = S + stage;
    const Item it = items[blockIdx.x];
    const Front f = fronts[it.front];
    const int nn = f.nn, na = f.na, nj = nn + na;
    const int tid = threadIdx.x, tx = tid % TD, ty = tid / TD;
    constexpr bool single = sizeof(T) == 4;
    if (tid == 0) flag = 0;
    for (int k = tid; k < nn; k += TD * TD) {
        if (LDLT) s.sgn[k] = pivot_sign(signs, LDLT, f.col0 + k);
        // the pivot check compares against the entry before the children's updates
        if (single) s.diag0[k] = (T)fabs((double)P[f.poff + k + (int64_t)k * f.ldp]);
    }
    small_assemble<T>(F, S, stage, f, fronts, reltgt, chdtgt, P, M);
    T a[R][R];
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j <= i; ++j) {
            const int r = tx + TD * i, c = ty + TD * j;
            a[i][j] = (r < nj && c <= r) ? F[r + c * f.ldp] : T(0);
        }
    int bad = eliminate<T, LDLT, TD, R, false, REG>(a, nj, nn, F, f.ldp, nullptr, 0, s, reg, single, &flag);
    if constexpr (single) {
        if ((bad >= 0 || flag) && nj <= kSmallRescue) {
            double* F64 = reinterpret_cast<double*>(smem_raw);
            __syncthreads();
            bad = small_redo<LDLT>(F64, f, fronts, reltgt, chdtgt, P, M, signs);
            if (bad < 0) {
                if (tid == 0) atomicAdd(rescued, 1);
                small_panel_store<double, T, LDLT>(F64, nj, f, P, d);
                for (int i = tid; i < na * na; i += TD * TD) {
                    const int r = i % na, c = i / na;
                    if (r >= c) M[f.moff + r + c * f.ldm] = (T)F64[(nn + r) + (nn + c) * nj];
                }
                return;
            }
        }
    }
    if (bad >= 0) {
        if (tid == 0) atomicMin(info, (long long)(f.col0 + bad + 1));
        return;
    }
    small_panel_store<T, T, LDLT>(F, f.ldp, f, P, d);
    T* Mj = M + f.moff - nn - (int64_t)nn * f.ldm;
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j <= i; ++j) {
            const int r = tx + TD * i, c = ty + TD * j;
            if (r < nj && c <= r && c >= nn) Mj[r + (int64_t)c * f.ldm] = a[i][j];
        }
}

// ---------------------------------------------------------------------------
// Tiny fronts (nj <= ROWS, ROWS = 16 or 32): one WARP per front, kWarpFronts
// fronts per CTA, warp-synchronous (no block barriers).  Lane r holds row r of
// the front in the warp's slice of shared memory (leading dimension ROWS + 1,
// sized for FP64 so a flagged single-precision front can be redone in place).  The
// arithmetic is k_small's: the children added in the reference's reverse
// order, one addition per entry and child, then the right-looking partial
// factorization with the same update expression.
// ---------------------------------------------------------------------------
// ROWS = 16 (nj <= kWarpSmallNJ: lanes 16..31 idle, registers and shared
// memory small) or 32 (kWarpSmallNJ < nj <= kWarpSmallNJ2)
constexpr int kWarpFronts = 8;
template <int ROWS>
constexpr int warp_slice() { return (ROWS + 1) * ROWS * (int)sizeof(double); }  // bytes per warp

template <typename TC, typename T, int LDLT, int ROWS>
__device__ int warp_front(TC* F, const Front& f, const Front* __restrict__ fronts,
                          const int32_t* __restrict__ reltgt, const int32_t* __restrict__ chdtgt,
                          const T* __restrict__ P, const T* __restrict__ M, const double* __restrict__ signs,
                          bool check, bool* flag, Reg reg, int lane) {
    const int nn = f.nn, na = f.na, nj = nn + na, ld = f.ldp;
    const T* Pj = P + f.poff;
    const bool row = lane < nj;
    // lane q fetches the record of the q-th child to add (children past 32
    // are read in the loop), beside the panel loads
    const int nch = f.chd1 - f.chd0;
    int kna = 0, klm = 0, ksep = 0;
    int64_t kmoff = 0;
    if (lane < nch) {
        const Front fc = fronts[chdtgt[f.chd1 - 1 - lane]];
        kna = fc.na, klm = fc.ldm, ksep = fc.sep0, kmoff = fc.moff;
    }
    {
        // every panel load of the lane in flight at once, then the stores
        T v[ROWS];
#pragma unroll
        for (int c = 0; c < ROWS; ++c) v[c] = (row && c < nn) ? Pj[lane + (int64_t)c * ld] : T(0);
#pragma unroll
        for (int c = 0; c < ROWS; ++c)
            if (row && c < nj) F[lane + c * (ROWS + 1)] = (TC)v[c];
    }
    __syncwarp();
    // extend-add, children popped in reverse (cholesky.jl:506-514)
    for (int q = 0; q < nch; ++q) {
        int ma = __shfl_sync(0xffffffffu, kna, q & 31), lm = __shfl_sync(0xffffffffu, klm, q & 31);
        int sep0 = __shfl_sync(0xffffffffu, ksep, q & 31);
        int64_t moff = __shfl_sync(0xffffffffu, kmoff, q & 31);
        if (q >= 32) {
            const Front fc = fronts[chdtgt[f.chd1 - 1 - q]];
            ma = fc.na, lm = fc.ldm, sep0 = fc.sep0, moff = fc.moff;
        }
        const int32_t* rel = reltgt + sep0;
        const T* Mc = M + moff;
        const int ra = lane < ma ? rel[lane] : 0;
        T mv[ROWS];
#pragma unroll
        for (int b = 0; b < ROWS; ++b) mv[b] = (b < ma && lane >= b && lane < ma) ? Mc[lane + b * lm] : T(0);
#pragma unroll
        for (int b = 0; b < ROWS; ++b) {
            const int rb = __shfl_sync(0xffffffffu, ra, b);
            if (b < ma && lane >= b && lane < ma) F[ra + rb * (ROWS + 1)] += (TC)mv[b];
        }
        __syncwarp();
    }
    // right-looking partial factorization of the first nn columns
    for (int k = 0; k < nn; ++k) {
        TC piv = F[k + k * (ROWS + 1)];
        const double s = pivot_sign(signs, LDLT, f.col0 + k);
        if (reg.delta >= 0.0) {
            piv = (TC)reg_pivot(reg, s, (double)piv);
            if (piv == TC(0)) return k;  // uniform across the warp
        } else if (!pivot_ok(s, (double)piv) || (!LDLT && !(piv > TC(0)))) {
            return k;  // uniform across the warp
        }
        if (check) {
            const double a0 = fabs((double)Pj[k + (int64_t)k * ld]);
            const double ap = fabs((double)piv);
            if (ap < kRescueSmall * a0 || ap > kRescueGrowth * fmax(a0, 1.0)) *flag = true;
        }
        const TC inv = pivot_recip<LDLT, false>(piv);
        __syncwarp();
        if (lane == k) F[k + k * (ROWS + 1)] = pivot_stored<TC, LDLT>(piv);
        if (lane > k && row) F[lane + k * (ROWS + 1)] *= inv;
        __syncwarp();
        if (lane > k && row) {
            const TC lr = F[lane + k * (ROWS + 1)];
            for (int c = k + 1; c <= lane; ++c) {
                TC lc = F[c + k * (ROWS + 1)];
                if (LDLT) lc *= piv;
                F[lane + c * (ROWS + 1)] -= lr * lc;
            }
        }
        __syncwarp();
    }
    return -1;
}

template <typename TC, typename T, int LDLT, int ROWS>
__device__ void warp_front_store(const TC* F, const Front& f, T* __restrict__ P, T* __restrict__ M,
                                 T* __restrict__ d, int lane) {
    const int nn = f.nn, na = f.na, nj = nn + na, ld = f.ldp;
    T* Pj = P + f.poff;
    if (lane < nj)
        for (int c = 0; c < nn; ++c) Pj[lane + (int64_t)c * ld] = (T)F[lane + c * (ROWS + 1)];
    if (LDLT && lane < nn) d[f.col0 + lane] = (T)F[lane + lane * (ROWS + 1)];
    T* Mj = M + f.moff;
    const int lm = f.ldm;
    if (lane < na)
        for (int b = 0; b < na; ++b) Mj[lane + b * lm] = (T)F[(nn + lane) + (nn + b) * (ROWS + 1)];
}

template <typename T, int LDLT, int ROWS>
__global__ void __launch_bounds__(kWarpFronts * 32) k_small_warp(const Front* __restrict__ fronts,
                                                                const Item* __restrict__ items, int64_t cnt,
                                                                const int32_t* __restrict__ reltgt,
                                                                const int32_t* __restrict__ chdtgt,
                                                                T* __restrict__ P, T* __restrict__ M,
                                                                T* __restrict__ d, const double* __restrict__ signs,
                                                                long long* __restrict__ info,
                                                                int* __restrict__ rescued, Reg reg) {
    pdl_prologue();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int64_t w = (int64_t)blockIdx.x * kWarpFronts + wib;
    if (w >= cnt) return;  // whole warps only
    unsigned char* slice = smem_raw + (size_t)wib * warp_slice<ROWS>();
    const Front f = fronts[items[w].front];
    constexpr bool single = sizeof(T) == 4;
    bool flag = false;
    T* F = reinterpret_cast<T*>(slice);
    int bad = warp_front<T, T, LDLT, ROWS>(F, f, fronts, reltgt, chdtgt, P, M, signs, single, &flag, reg, lane);
    if (single && (bad >= 0 || flag)) {
        // the panel and the children's update matrices are only read before
        // the final store: refactor from the same inputs in FP64
        double* F64 = reinterpret_cast<double*>(slice);
        __syncwarp();
        bool unused = false;
        bad = warp_front<double, T, LDLT, ROWS>(F64, f, fronts, reltgt, chdtgt, P, M, signs, false, &unused, reg, lane);
        if (bad < 0) {
            if (lane == 0) atomicAdd(rescued, 1);
            __syncwarp();
            warp_front_store<double, T, LDLT, ROWS>(F64, f, P, M, d, lane);
            return;
        }
    }
    if (bad >= 0) {
        if (lane == 0) atomicMin(info, (long long)(f.col0 + bad + 1));
        return;
    }
    __syncwarp();
    warp_front_store<T, T, LDLT, ROWS>(F, f, P, M, d, lane);
}

// ---------------------------------------------------------------------------
// extend-add for blocked fronts
// ---------------------------------------------------------------------------

// One CTA per (front, 16 parent columns, kEArows parent rows); warp w owns
// parent columns c0 + w and c0 + w + 8.  The plan lists, per child in the
// reference's order (reverse, cholesky.jl:506-514), the child columns b0..b1
// and rows a0..a1 whose relative indices fall in the item's columns and rows,
// so the kernel does no searching.  Every parent entry belongs to one CTA and
// one warp, and the children are added in a fixed order: no atomics, no block
// barrier, deterministic sums.  PART 0 adds into the panel columns (before
// the front is factored), PART 1 into the update matrix, which the SYRK has
// already set to -L21 L21^T (so it is never zeroed or read twice).  A child
// column streams in chunks of up to 4 x 32 rows (ea_chunk).
// a chunk of U x 32 rows of a child column: the relative indices and child
// values of the chunk first, then the U parent entries they address, so U
// independent gather chains are in flight per lane; PRED drops rows >= a1
template <typename T, int U, bool PRED>
__device__ __forceinline__ void ea_chunk(const int32_t* __restrict__ rel, const T* mc, T* dst, int a, int a1) {
    int r[U];
    T v[U], o[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int aa = a + 32 * u;
        const bool in = !PRED || aa < a1;
        r[u] = in ? __ldg(rel + aa) : -1;
        v[u] = in ? mc[aa] : T(0);
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
        if (r[u] >= 0) o[u] = dst[r[u]];
#pragma unroll
    for (int u = 0; u < U; ++u)
        if (r[u] >= 0) dst[r[u]] = o[u] + v[u];
}

//
// A front may have hundreds of children that miss an item, and a small front's
// item is a chain of dependent loads (child list, child record, relative
// index, entry), so the lanes of a warp fetch the segments and records of 32
// children at once -- and the first children's relative indices before the
// kernel waits for the work below it -- and only children that reach the item
// are visited.
template <typename T, int PART>
__global__ void __launch_bounds__(256) k_ea(const Front* __restrict__ fronts, const Item* __restrict__ items,
                                            const Item* __restrict__ all_items, const int32_t* __restrict__ reltgt,
                                            T* P, T* M) {
    pdl_trigger();
    constexpr unsigned kAll = 0xffffffffu;
    const Item it = items[blockIdx.x];
    const Front f = fronts[it.front];
    const int nn = f.nn, ld = f.ldp, lm = f.ldm;
    const int c0 = it.a * kEAcols;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T* Pj = P + f.poff;
    T* Mj = M + f.moff;
    const Item* seg = all_items + it.pad;  // segment offsets index the whole item buffer
    const int nch = f.chd1 - f.chd0;
    bool waited = false;
    for (int s0 = 0; s0 < nch; s0 += 32) {
        // lane q holds child s0 + q's segment and record
        Item s1{}, s2{};
        int sep0 = 0, ldm = 0;
        int64_t moff = 0;
        bool hit = false;
        if (s0 + lane < nch) {
            s1 = seg[2 * (s0 + lane)], s2 = seg[2 * (s0 + lane) + 1];
            hit = s1.a < s1.b && s2.front < s2.a;
            if (hit) {
                const Front& fc = fronts[s1.front];
                sep0 = fc.sep0, ldm = fc.ldm, moff = fc.moff;
            }
        }
        unsigned todo = __ballot_sync(kAll, hit);
        int cn = -1;  // lane j: the parent column of the next child's column b0 + j
        auto columns = [&](unsigned left) {
            if (!left) return;
            const int q = __ffs(left) - 1;
            const int b0 = __shfl_sync(kAll, s1.a, q), b1 = __shfl_sync(kAll, s1.b, q), sp = __shfl_sync(kAll, sep0, q);
            cn = b0 + lane < b1 ? __ldg(reltgt + sp + b0 + lane) : -1;
        };
        columns(todo);
        if (!waited) asm volatile("griddepcontrol.wait;" ::: "memory");
        waited = true;
        while (todo) {
            const int q = __ffs(todo) - 1;
            todo &= todo - 1;
            const int b0 = __shfl_sync(kAll, s1.a, q);
            const int a0 = __shfl_sync(kAll, s2.front, q), a1 = __shfl_sync(kAll, s2.a, q);
            const int32_t* __restrict__ rel = reltgt + __shfl_sync(kAll, sep0, q);
            const T* Mc = M + __shfl_sync(kAll, moff, q);
            const int lmc = __shfl_sync(kAll, ldm, q);
            const int cq = cn;
            columns(todo);
            // the owner warp of a parent column takes it (at most kEAcols columns of the child fall in the item)
            unsigned own = __ballot_sync(kAll, cq >= 0 && ((cq - c0) & 7) == warp);
            while (own) {
                const int j = __ffs(own) - 1;
                own &= own - 1;
                const int b = b0 + j, col = __shfl_sync(kAll, cq, j);
                const T* mc = Mc + (int64_t)b * lmc;
                T* dst = PART == 0 ? Pj + (int64_t)col * ld : Mj + (int64_t)(col - nn) * lm - nn;
                // full chunks of 4 x 32 rows, then one predicated chunk of at
                // most 4 x 32 rows (a single row per lane when the rest is that
                // short: many child columns are, and the predicated slots would
                // cost instructions for nothing).  Eight chains per lane measured
                // slower on long columns (more lines in flight than L1 keeps).
                int a = max(a0, b) + lane;
                for (; a + 96 < a1; a += 128) ea_chunk<T, 4, false>(rel, mc, dst, a, a1);
                if (a + 32 < a1) ea_chunk<T, 4, true>(rel, mc, dst, a, a1);
                else if (a < a1) dst[__ldg(rel + a)] += mc[a];
            }
            __syncwarp();
        }
    }
    if (!waited) asm volatile("griddepcontrol.wait;" ::: "memory");
}

// ---------------------------------------------------------------------------
// diagonal block: factor + inverse
// ---------------------------------------------------------------------------

// Diagonal block: factor + inverse, one CTA of 256 threads per front
// (eliminate() on the 64 x 64 block, columns >= w padded with the identity).
constexpr int LDS = kNB + 4;  // shared-memory leading dimension of the GEMM stages
constexpr int LDA = kNB + 1;  // leading dimension of the factor and inverse in the diagonal kernel
constexpr int kDiagTD = 16, kDiagR = kNB / kDiagTD;

// dynamic shared memory of k_diag: the FP64 layout in both precisions (the
// single-precision kernel refactors flagged blocks in FP64 in place)
template <typename T>
constexpr int diag_smem() { return 2 * kNB * LDA * (int)sizeof(double) + (int)sizeof(ElimBufs<double, kNB, true>); }

// Factor and invert the 64 x 64 block held in shared memory as TC: A (block,
// identity beyond column w) and X (zeros, receives the inverse); s.piv gets
// the stored diagonal.  Returns the first rejected pivot (block-local) or -1,
// uniform across the block.
template <typename TC, int LDLT, bool REG>
__device__ __forceinline__ int diag_block(TC* A, TC* X, ElimBufs<TC, kNB, true>& s, int w,
                                          const double* __restrict__ signs, int64_t colbase, const Reg& reg) {
    const int tid = threadIdx.x, tx = tid % kDiagTD, ty = tid / kDiagTD;
    if (LDLT && tid < w) s.sgn[tid] = pivot_sign(signs, LDLT, colbase + tid);
    TC a[kDiagR][kDiagR];
#pragma unroll
    for (int i = 0; i < kDiagR; ++i)
#pragma unroll
        for (int j = 0; j <= i; ++j) a[i][j] = A[(tx + kDiagTD * i) + (ty + kDiagTD * j) * LDA];
    return eliminate<TC, LDLT, kDiagTD, kDiagR, true, REG>(a, kNB, w, A, LDA, X, LDA, s, reg, false, nullptr);
}

// Write back a factored diagonal block: the factor into the panel, the LDLt
// pivots, the inverse into the inverse scratch.
template <typename TC, typename T, int LDLT>
__device__ void diag_block_store(const TC* A, const TC* X, const TC* pivs, int w, T* Pj, int64_t ld, int c0,
                                 T* __restrict__ d, int64_t dcol, T* dst) {
    const int tid = threadIdx.x;
#pragma unroll
    for (int e = tid; e < kNB * kNB; e += 256) {
        const int r = e & (kNB - 1), c = e >> 6;
        if (r >= c && r < w && c < w) Pj[(c0 + r) + (int64_t)(c0 + c) * ld] = (T)A[r + c * LDA];
    }
    if (LDLT && tid < w) d[dcol + tid] = (T)pivs[tid];
#pragma unroll
    for (int e = tid; e < kNB * kNB; e += 256) {
        const int r = e & (kNB - 1), c = e >> 6;
        dst[e] = (r < w && c < w) ? (T)X[r + c * LDA] : T(0);
    }
}

template <typename TC, typename T, bool ZERO>
__device__ __forceinline__ void diag_block_load(TC* A, TC* X, const T* Pj, int64_t ld, int c0, int w) {
    const int tid = threadIdx.x;
#pragma unroll
    for (int e = tid; e < kNB * kNB; e += 256) {
        const int r = e & (kNB - 1), c = e >> 6;
        TC v = (r == c) ? TC(1) : TC(0);
        if (r >= c && r < w && c < w) v = (TC)Pj[(c0 + r) + (int64_t)(c0 + c) * ld];
        A[r + c * LDA] = v;
        if (ZERO) X[r + c * LDA] = TC(0);
    }
}

// FP64: the block's left-looking update from the outer block's columns
// [k0, c0), sum_k (L_rk d_k) L_ck over its lower triangle, in chunks of 64
// columns staged as stage[k * DLD + row] while the next chunk is on its way in
// registers; on DMMA, the triangle's 36 8 x 8 tiles nine a pair of warps
// (w, w + 4) that share a scheduler (tile row 7 - s and tile row s).
constexpr int DLD = kNB + 4;
struct DiagAccD {
    double c[5][2] = {};
    __device__ __forceinline__ static void tile(int t, int& r, int& col, bool& ok) {
        const int warp = threadIdx.x >> 5, s = warp & 3;
        if (warp < 4) { r = 7 - s; col = t; ok = true; }
        else if (t < 3 - s) { r = 7 - s; col = 5 + t; ok = true; }
        else { r = s; col = t - (3 - s); ok = col <= s; }
    }
    template <int LDLT>
    __device__ __forceinline__ void mma(const double* S, const double* dsc) {
        const int lane = threadIdx.x & 31, fr = lane >> 2, fk = lane & 3;
        const int s = (threadIdx.x >> 5) & 3, r0 = 8 * (7 - s) + fr, r1 = 8 * s + fr;
        int co[5];
        bool first[5], ok[5];  // all uniform in a warp
#pragma unroll
        for (int t = 0; t < 5; ++t) {
            int r, col;
            tile(t, r, col, ok[t]);
            first[t] = r == 7 - s;
            co[t] = ok[t] ? 8 * col + fr : 0;
        }
#pragma unroll 4
        for (int k = 0; k < kNB; k += 4) {
            const double* Sk = S + (k + fk) * DLD;
            double a0 = Sk[r0], a1 = Sk[r1];
            if (LDLT) a0 *= dsc[k + fk], a1 *= dsc[k + fk];
#pragma unroll
            for (int t = 0; t < 5; ++t)
                if (ok[t]) dmma(c[t][0], c[t][1], first[t] ? a0 : a1, Sk[co[t]]);
        }
    }
    template <typename F>
    __device__ __forceinline__ void visit(F&& fn) {
        const int lane = threadIdx.x & 31;
#pragma unroll
        for (int t = 0; t < 5; ++t) {
            int r, col;
            bool ok;
            tile(t, r, col, ok);
            if (ok)
#pragma unroll
                for (int e = 0; e < 2; ++e) fn(8 * r + (lane >> 2), 8 * col + (lane & 3) * 2 + e, c[t][e]);
        }
    }
};
template <int LDLT>
__device__ __forceinline__ void diag_update(double* A, double* X, double* dsc, const double* Pj, const double* dj,
                                            int64_t ld, int k0, int c0, int w) {
    constexpr int PER = kNB * kNB / 256;
    const int tid = threadIdx.x, r = tid & (kNB - 1), kc = tid >> 6;
    double* stage = X;  // X's place and 1.5 KB of the elimination's buffers after it
    DiagAccD acc;
    double v[PER], dv = 0.0;
    auto fetch = [&](int k) {
#pragma unroll
        for (int u = 0; u < PER; ++u) v[u] = r < w ? Pj[(c0 + r) + (int64_t)(k + kc + 4 * u) * ld] : 0.0;
        if (LDLT && tid < kNB) dv = dj[k + tid];
    };
    fetch(k0);
    diag_block_load<double, double, false>(A, X, Pj, ld, c0, w);
    for (int k = k0; k < c0; k += kNB) {
#pragma unroll
        for (int u = 0; u < PER; ++u) stage[(kc + 4 * u) * DLD + r] = v[u];
        if (LDLT && tid < kNB) dsc[tid] = dv;
        __syncthreads();
        if (k + kNB < c0) fetch(k + kNB);
        acc.mma<LDLT>(stage, dsc);
        __syncthreads();
    }
    for (int e = tid; e < kNB * LDA; e += 256) X[e] = 0.0;
    acc.visit([&](int row, int col, double x) {
        if (row >= col && row < w) A[row + col * LDA] -= x;  // (col <= row < w)
    });
}
static_assert(kNB * DLD <= kNB * LDA + 4 * kNB, "the stage ends inside the elimination's buffers");

// Diagonal block kernel.  UPDATE (FP64, sub-panels after an outer block's
// first): applies the block's left-looking update before it factors and
// inverts it.  The rows below get theirs from the LEFT launch that follows,
// which runs beside this one: a sub-panel's chain is the longer of the two and
// the TRSM, not their sum.  For that this kernel lets the next grid go only
// after its own wait, when all that both read is complete, and LEFT waits for
// this kernel at its end.  KKT 24 10.78 -> 10.30 ms (a sub-panel's update and
// block 25 -> 23 us, and its rows' update off the chain), 80^3 81.1 -> 79.3,
// 16^3 1.182 -> 1.168 ms.  (diag_and_left in factor_impl launches the pair.)
// Not in single precision: on the chain the update costs the 64 x 64 x K
// products on one SM, about what the tensor-core launch took (KKT 24 mixed
// 9.08 -> 9.04 ms, 80^3 mixed 32.65 -> 32.80, 512^2 8.56 -> 8.55).
//
// Single precision: when the FP32 factorization rejects a pivot, or a pivot
// lost more than five digits against its diagonal entry or grew beyond 1e7
// times the block's largest diagonal entry, the block is loaded again and
// factored and inverted in FP64 (the dynamic shared memory is sized for that),
// and the FP64 result is stored rounded to FP32.  A rejection in FP64 is
// reported through info.
template <typename T, int LDLT, bool REG, bool UPDATE>
__global__ void __launch_bounds__(256, 1) k_diag(const Front* __restrict__ fronts, const Item* __restrict__ items,
                                              int obs, int c0, T* P, T* inv,
                                              T* d, const double* __restrict__ signs,
                                              long long* __restrict__ info, int* __restrict__ rescued, Reg reg) {
    if (!UPDATE) pdl_trigger();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* A = reinterpret_cast<T*>(smem_raw);  // block, then its factor, A[r + c * LDA]
    T* X = A + kNB * LDA;                   // inverse, same layout
    unsigned char* sraw = smem_raw + 2 * kNB * LDA * sizeof(double);
    ElimBufs<T, kNB, true>& s = *reinterpret_cast<ElimBufs<T, kNB, true>*>(sraw);
    const T* pivs = s.piv;  // L_kk (Cholesky) or d_k (LDLt)
    __shared__ int flag_s;
    __shared__ double dmax_s;
    const Item it = items[blockIdx.x];
    const Front f = fronts[it.front];
    const int nn = f.nn;
    const int64_t ld = f.ldp;
    const int w = min(kNB, nn - c0);
    const int tid = threadIdx.x;
    T* Pj = P + f.poff;
    T* dst = inv + f.ioff + (int64_t)(c0 / kNB) * kNB * kNB;
    constexpr bool single = sizeof(T) == 4;
    if (tid == 0) { flag_s = 0; dmax_s = 0.0; }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if constexpr (UPDATE) {
        static_assert(!single, "FP64 only");
        pdl_trigger();
        __shared__ double dsc[LDLT ? kNB : 1];
        diag_update<LDLT>(A, X, dsc, Pj, d + f.col0, ld, obs, c0, w);
    } else {
        diag_block_load<T, T, true>(A, X, Pj, ld, c0, w);
    }
    __syncthreads();
    // |a_kk| before the factorization and the block's largest (non-negative
    // doubles order like their bit patterns); the factorization has barriers
    const double a0 = tid < w ? fabs((double)A[tid + tid * LDA]) : 0.0;
    if (single && tid < w)
        atomicMax(reinterpret_cast<unsigned long long*>(&dmax_s), (unsigned long long)__double_as_longlong(a0));
    int bad = diag_block<T, LDLT, REG>(A, X, s, w, signs, (int64_t)f.col0 + c0, reg);
    if (single) {
        if (bad < 0 && tid < w) {
            const double dk = LDLT ? fabs((double)pivs[tid]) : (double)pivs[tid] * (double)pivs[tid];
            if (dk < kRescueSmall * a0 || dk > kRescueGrowth * fmax(dmax_s, 1.0)) flag_s = 1;
        }
        __syncthreads();
        if (bad >= 0 || flag_s) {
            double* A64 = reinterpret_cast<double*>(smem_raw);
            double* X64 = A64 + kNB * LDA;
            ElimBufs<double, kNB, true>& s64 = *reinterpret_cast<ElimBufs<double, kNB, true>*>(sraw);
            __syncthreads();
            diag_block_load<double, T, true>(A64, X64, Pj, ld, c0, w);
            __syncthreads();
            bad = diag_block<double, LDLT, false>(A64, X64, s64, w, signs, (int64_t)f.col0 + c0, reg);
            if (bad < 0) {
                if (tid == 0) atomicAdd(rescued, 1);
                diag_block_store<double, T, LDLT>(A64, X64, s64.piv, w, Pj, ld, c0, d, f.col0 + c0, dst);
                return;
            }
        }
    }
    if (bad >= 0) {  // uniform
        if (tid == 0) atomicMin(info, (long long)(f.col0 + c0 + bad + 1));
        return;
    }
    diag_block_store<T, T, LDLT>(A, X, pivs, w, Pj, ld, c0, d, f.col0 + c0, dst);
}

// ---------------------------------------------------------------------------
// FP32 tile GEMM without tensor cores (the autotuner's alternative to mf_tc.cu's
// tiles on levels of small fronts), with a cp.async double-buffered K loop:
// acc(64x64) += A(64 x K) * B(64 x K)^T.  Shared tiles are [k][m] with m
// contiguous (leading dimension LDS); thread t owns rows (t>>4)*4..+4 and
// columns (t&15)*4..+4.
// ---------------------------------------------------------------------------
constexpr int KC = 32;                   // K chunk per pipeline stage
constexpr int STAGE = KC * LDS;          // elements per matrix per stage

template <typename T>
constexpr int gemm_smem() { return (4 * STAGE + 2 * KC) * (int)sizeof(T); }

template <typename T>
struct Acc;
template <>
struct Acc<float> {
    float c[4][4];
};

__device__ __forceinline__ void acc_zero(Acc<float>& a) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) a.c[i][j] = 0.f;
}

__device__ __forceinline__ void cp_async_el(float* dst, const float* src, bool valid) {
    const unsigned saddr = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(saddr), "l"(src), "r"(valid ? 4 : 0));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

template <typename T>
__device__ __forceinline__ void stage_chunk(T* As, T* Bs, const T* A, int64_t lda, int ra, int amax, const T* B,
                                            int64_t ldb, int rb, int bmax, int k, int kc) {
    for (int i = threadIdx.x; i < 64 * KC; i += blockDim.x) {
        int m = i & 63, kk = i >> 6;
        bool va = (ra + m < amax) && kk < kc;
        bool vb = (rb + m < bmax) && kk < kc;
        const T* sa = A + (va ? (ra + m) + (int64_t)(k + kk) * lda : 0);
        const T* sb = B + (vb ? (rb + m) + (int64_t)(k + kk) * ldb : 0);
        cp_async_el(As + m + kk * LDS, sa, va);
        cp_async_el(Bs + m + kk * LDS, sb, vb);
    }
}

__device__ __forceinline__ void mma_chunk(Acc<float>& acc, const float* As, const float* Bs, const float* dsc,
                                          int kc) {
    const int tr = (threadIdx.x >> 4) * 4, tc = (threadIdx.x & 15) * 4;
    for (int k = 0; k < kc; ++k) {
        const float4 a4 = *reinterpret_cast<const float4*>(As + tr + k * LDS);
        const float4 b4 = *reinterpret_cast<const float4*>(Bs + tc + k * LDS);
        const float s = dsc ? dsc[k] : 1.f;
        const float a[4] = {a4.x * s, a4.y * s, a4.z * s, a4.w * s};
        const float b[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc.c[i][j] = fmaf(a[i], b[j], acc.c[i][j]);
    }
}

// acc += A[ra.., kbeg..kend) * B[rb.., kbeg..kend)^T (optionally D-scaled)
template <typename T>
__device__ void gemm_k_loop(Acc<T>& acc, T* smem, const T* A, int64_t lda, int ra, int amax, const T* B,
                            int64_t ldb, int rb, int bmax, int kbeg, int kend, const T* dvec) {
    const int nchunk = (kend - kbeg + KC - 1) / KC;
    if (nchunk <= 0) return;
    auto buf_a = [&](int st) { return smem + st * STAGE; };
    auto buf_b = [&](int st) { return smem + (2 + st) * STAGE; };
    auto buf_d = [&](int st) { return smem + 4 * STAGE + st * KC; };
    auto load = [&](int c, int st) {
        int k = kbeg + c * KC;
        int kc = min(KC, kend - k);
        stage_chunk(buf_a(st), buf_b(st), A, lda, ra, amax, B, ldb, rb, bmax, k, kc);
        if (dvec)
            for (int i = threadIdx.x; i < KC; i += blockDim.x) buf_d(st)[i] = i < kc ? dvec[k + i] : T(0);
        cp_commit();
    };
    load(0, 0);
    for (int c = 0; c < nchunk; ++c) {
        const int st = c & 1;
        if (c + 1 < nchunk) {
            load(c + 1, st ^ 1);
            cp_wait<1>();
        } else {
            cp_wait<0>();
        }
        __syncthreads();
        int kc = min(KC, kend - (kbeg + c * KC));
        mma_chunk(acc, buf_a(st), buf_b(st), dvec ? buf_d(st) : nullptr, (kc + 3) & ~3);
        __syncthreads();
    }
}

// visit every accumulator element as (row, col, value)
template <typename F>
__device__ __forceinline__ void acc_for_each(const Acc<float>& acc, F&& fn) {
    const int tr = (threadIdx.x >> 4) * 4, tc = (threadIdx.x & 15) * 4;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) fn(tr + i, tc + j, acc.c[i][j]);
}

// C(rbase+r, cbase+c) -= acc (or = acc * colscale when OVERWRITE), for
// r < rmax, c < cmax; on a diagonal tile only row >= col is written.
// Store an accumulator tile: MODE 0 C -= acc, MODE 1 C = acc (times the
// column scale if given), MODE 2 C = -acc (the SYRK writes M = -L21 L21^T;
// the children's extend-add follows it).
template <int MODE, typename T>
__device__ __forceinline__ void acc_store(const Acc<T>& acc, T* C, int64_t ldc, int rbase, int cbase, int rmax,
                                          int cmax, bool diag_tile, const T* colscale) {
    acc_for_each(acc, [&](int r, int c, T v) {
        if (r < rmax && c < cmax && (!diag_tile || rbase + r >= cbase + c)) {
            T* p = C + (rbase + r) + (int64_t)(cbase + c) * ldc;
            if (MODE == 1) *p = colscale ? v * colscale[c] : v;
            else if (MODE == 2) *p = -v;
            else *p -= v;
        }
    });
}

enum GemmRole { G_LEFT = 0, G_TRAIL = 1, G_SYRK = 2, G_TRSM = 3 };

template <typename T, int ROLE, int LDLT>
__global__ void __launch_bounds__(256) k_gemm(const Front* __restrict__ fronts, const Item* __restrict__ items,
                                              int obs, int obw, int c0, T* P, T* M, const T* d, const T* inv) {
    pdl_prologue();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* smem = reinterpret_cast<T*>(smem_raw);
    const Item it = items[blockIdx.x];
    const Front f = fronts[it.front];
    const int nn = f.nn, na = f.na, nj = nn + na, ld = f.ldp;
    T* Pj = P + f.poff;
    const T* dj = LDLT ? d + f.col0 : nullptr;
    Acc<T> acc;
    acc_zero(acc);
    if (ROLE == G_LEFT) {
        const int w = min(kNB, nn - c0);
        const int rs = c0 + it.a * kTile;
        gemm_k_loop<T>(acc, smem, Pj, ld, rs, nj, Pj, ld, c0, c0 + w, obs, c0, dj);
        acc_store<0>(acc, Pj, ld, rs, c0, nj - rs, w, it.a == 0, (const T*)nullptr);
    } else if (ROLE == G_TRAIL) {
        const int e = min(nn, obs + obw);
        const int cs = e + it.b * kTile, rs = cs + it.a * kTile;
        gemm_k_loop<T>(acc, smem, Pj, ld, rs, nj, Pj, ld, cs, nn, obs, e, dj);
        acc_store<0>(acc, Pj, ld, rs, cs, nj - rs, nn - cs, it.a == 0, (const T*)nullptr);
    } else if (ROLE == G_SYRK) {
        const int rs = it.a * kTile, cs = it.b * kTile;
        gemm_k_loop<T>(acc, smem, Pj + nn, ld, rs, na, Pj + nn, ld, cs, na, 0, nn, dj);
        acc_store<2>(acc, M + f.moff, f.ldm, rs, cs, na - rs, na - cs, it.a == it.b, (const T*)nullptr);
    } else {
        // X (rows below the diagonal block, cols [c0, c0+w)) = X * Linv^T (* D^-1)
        const int w = min(kNB, nn - c0);
        const int rs = c0 + w + it.a * kTile;
        const T* Li = inv + f.ioff + (int64_t)(c0 / kNB) * kNB * kNB;
        gemm_k_loop<T>(acc, smem, Pj + (int64_t)c0 * ld, ld, rs, nj, Li, kNB, 0, w, 0, w, (const T*)nullptr);
        __syncthreads();
        T* sc = smem;  // reuse: reciprocal pivots for LDLt
        if (LDLT) {
            for (int i = threadIdx.x; i < w; i += blockDim.x) sc[i] = T(1) / dj[c0 + i];
            __syncthreads();
        }
        acc_store<1>(acc, Pj + (int64_t)c0 * ld, ld, rs, 0, nj - rs, w, false, LDLT ? (const T*)sc : nullptr);
    }
}

// ---------------------------------------------------------------------------
// FP64 tile GEMM of the blocked fronts: acc(BM x 64) = A(BM x K) B(64 x K)^T on
// DMMA (mma.sync m8n8k4 f64; tcgen05 has no FP64 kind), a warp per 32 x 32
// (16 x 32 for BM = 32).
//   BM = 128, 8 warps: sixteen independent products per four k and eight
//     shared-memory reads for them, two CTAs per SM, so one CTA's prologue and
//     C update hide behind the other's products;
//   BM = 64, 4 warps: launches of few tiles, where the SMs would idle;
//   BM = 32, 4 warps, two CTAs a 64-row item: launches of fewer 64-row tiles
//     than SMs, which last as long as one tile's products (KKT 24: 12.26 ->
//     11.75 ms a pass, 100^2 922 -> 886 us).
// What bounds the large launches is the FP64 pipe (64 FMA a cycle and SM:
// 36.9 TFLOP/s measured for DMMA alone; 87 % active in a large SYRK launch, 79 %
// in a large trailing update, whose tiles read and write C for 256 of k); 80^3: SYRKs 40.7 -> 36.5 ms, trailing
// updates 23.1 -> 20.6, left updates 5.9 -> 4.2, KKT 24 left updates 1.56 ->
// 1.01 ms, against 64 x 64 tiles of eight warps fed by 8-byte copies, two
// barriers per 32 k.  Operands come in 16-byte asynchronous copies, three
// stages of 16 k deep, one barrier a stage.  Tiles are columns of the panel
// (rows contiguous, [k][row] in shared memory with 4 doubles of padding: a
// fragment read touches every bank once).  A copy needs an even row start;
// tiles on an odd row (a 64-row SYRK tile of an odd nn) copy 8 bytes at a time.
// ---------------------------------------------------------------------------
constexpr int GK = 16, GStages = 3;
template <int BM>
constexpr int g64_stage() { return GK * (BM + 4) + GK * (kTile + 4) + GK; }  // A, B, pivots (doubles)
template <int BM>
constexpr int g64_smem() { return GStages * g64_stage<BM>() * (int)sizeof(double); }
template <int BM>
constexpr int g64_wm() { return BM == 32 ? 16 : 32; }  // rows per warp
template <int BM>
constexpr int g64_threads() { return 32 * (BM / g64_wm<BM>()) * (kTile / 32); }

__device__ __forceinline__ double ld_l2(const double* p) {
    double v;
    asm volatile("ld.global.cg.f64 %0, [%1];\n" : "=d"(v) : "l"(p));
    return v;
}

// copy rows [row0, row0 + ROWS) x columns [k, k + GK) of a column-major matrix
// into dst[kk * (ROWS + 4) + m]; rows at or past rlim (rounded up to the next
// even one) and columns at or past kend become zeros.  L2: nothing is read
// through L1 (an 8-byte asynchronous copy would be)
template <int ROWS, int NT, bool VEC, bool L2>
__device__ __forceinline__ void g64_copy(double* dst, const double* src, int64_t ld, int row0, int rlim, int k, int kend) {
    constexpr int W = VEC ? 2 : 1, PER = ROWS / W;
    static_assert((GK * PER) % NT == 0, "whole rounds of copies");
    if constexpr (L2 && !VEC) {
        double v[GK * PER / NT];
#pragma unroll
        for (int u = 0; u < GK * PER / NT; ++u) {
            const int i = threadIdx.x + u * NT, m = i % PER, kk = i / PER;
            const bool ok = row0 + m < rlim && k + kk < kend;
            v[u] = ok ? ld_l2(src + (row0 + m) + (int64_t)(k + kk) * ld) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < GK * PER / NT; ++u) {
            const int i = threadIdx.x + u * NT;
            dst[i / PER * (ROWS + 4) + i % PER] = v[u];
        }
    } else {
#pragma unroll
        for (int u = 0; u < GK * PER / NT; ++u) {
            const int i = threadIdx.x + u * NT;
            const int m = (i % PER) * W, kk = i / PER;
            const bool ok = row0 + m < rlim && k + kk < kend;
            const double* s = src + (ok ? (row0 + m) + (int64_t)(k + kk) * ld : 0);
            const unsigned d = (unsigned)__cvta_generic_to_shared(dst + kk * (ROWS + 4) + m);
            if (VEC)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(s), "r"(ok ? 16 : 0) : "memory");
            else
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(s), "r"(ok ? 8 : 0) : "memory");
        }
    }
}

// Items of BM <= 64 are the (front, 64-row tile, 64-column tile) lists; of
// BM = 128 the tensor-core lists (128-row tiles, 128-column ones for the
// trailing update and the SYRK, which start on 4-row boundaries), two CTAs an
// item there: column half blockIdx & 1.
template <int BM, int ROLE, int LDLT>
__global__ void __launch_bounds__(g64_threads<BM>(), BM == 128 ? 2 : 4) k_gemm64(const Front* __restrict__ fronts,
                                                                 const Item* __restrict__ items, int obs, int obw,
                                                                 int c0, double* P, double* M, const double* d,
                                                                 const double* inv) {
    pdl_trigger();
    constexpr int NT = g64_threads<BM>(), LA = BM + 4, LB = kTile + 4, STG = g64_stage<BM>();
    constexpr bool PAIR = BM == 128 && (ROLE == G_TRAIL || ROLE == G_SYRK);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* smem = reinterpret_cast<double*>(smem_raw);
    constexpr int IR = BM == 32 ? kTile : BM;  // rows of an item
    const Item it = items[(PAIR || BM == 32) ? blockIdx.x >> 1 : blockIdx.x];
    const int half = PAIR ? (int)(blockIdx.x & 1) * kTile : 0;
    const Front f = fronts[it.front];
    const int nn = f.nn, na = f.na, nj = nn + na, ld = f.ldp;
    double* Pj = P + f.poff;
    const int row0 = it.a * IR + (BM == 32 ? (int)(blockIdx.x & 1) * BM : 0);
    // panel rows ra.. (A) and rb.. (B) over columns [kbeg, kend); C rows
    // [rlo, rhi) x columns [clo, chi) in panel coordinates, at C + row + col * ldc
    int ra, rb, kbeg, kend, rlo, rhi = nj, clo, chi, blim = nj;
    const double* Bm = Pj;
    int64_t ldb = ld, ldc = ld;
    double* C = Pj;
    bool tri = true;
    if (ROLE == G_LEFT) {
        const int r0 = min(nn, c0 + kNB);  // k_diag updates the rows above
        ra = (BM == 128 ? r0 & ~3 : r0) + row0, rb = c0, kbeg = obs, kend = c0;
        rlo = r0, clo = c0, chi = r0, tri = false;
    } else if (ROLE == G_TRAIL) {
        const int e = min(nn, obs + obw);
        const int cs = e + it.b * (PAIR ? 2 * kTile : kTile);
        ra = cs + row0, rb = cs + half, kbeg = obs, kend = e;
        rlo = clo = e, chi = nn;
    } else if (ROLE == G_SYRK) {
        const int x0 = PAIR ? nn & ~3 : nn;
        // 64-row tiles: item (row tile, column tile); 128-row ones: (row tile below the diagonal, column tile)
        ra = PAIR ? x0 + it.b * 2 * kTile + row0 : x0 + row0;
        rb = x0 + it.b * (PAIR ? 2 * kTile : kTile) + half;
        kbeg = 0, kend = nn, rlo = clo = nn, chi = nj;
        C = M + f.moff - nn - (int64_t)nn * f.ldm;
        ldc = f.ldm;
    } else {
        const int r0 = min(nn, c0 + kNB);
        ra = (BM == 128 ? r0 & ~3 : r0) + row0, rb = 0, kbeg = c0, kend = r0;
        rlo = r0, clo = c0, chi = r0;
        Bm = inv + f.ioff + (int64_t)(c0 / kNB) * kNB * kNB - (int64_t)c0 * kNB;
        ldb = kNB, blim = kNB, tri = false;
    }
    // past the rows, or wholly above the diagonal (the wait is still taken: the
    // next grid may rely on the one before this)
    const bool none = ra >= rhi || (tri && ra + BM <= rb);
    // LEFT runs beside the k_diag<UPDATE> that is launched directly before it
    // (diag_and_left): that kernel lets it go only once its own wait has shown
    // that the grids before are complete, and so that what they wrote is in
    // L2.  This SM's L1 may still hold lines from before those writes, which
    // only a wait of this grid's own would drop, so LEFT reads panels and
    // pivots through L2 alone.  It waits for k_diag at its end: the TRSM
    // relies on both.
    constexpr bool L2 = ROLE == G_LEFT;
    auto wait = []() { asm volatile("griddepcontrol.wait;" ::: "memory"); };
    if (none || ROLE != G_LEFT) wait();
    if (none) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int WM = g64_wm<BM>(), MI = WM / 8;
    const int wr = (warp % (BM / WM)) * WM, wc = (warp / (BM / WM)) * 32;
    const int fr = lane >> 2, fk = lane & 3;
    const double* dj = (LDLT && ROLE != G_TRSM) ? d + f.col0 : nullptr;
    const bool vec = BM == 128 || ROLE == G_TRAIL || ((ra | rb) & 1) == 0;  // (even by their lists there)
    const int nchunk = (kend - kbeg + GK - 1) / GK;
    double dn = 0.0;
    if (LDLT && L2 && tid < GK && kbeg + tid < kend) dn = ld_l2(dj + kbeg + tid);
    auto load = [&](int c) {
        if (c < nchunk) {
            double* st = smem + (c % GStages) * STG;
            const int k = kbeg + c * GK;
            if (vec) {
                g64_copy<BM, NT, true, L2>(st, Pj, ld, ra, nj, k, kend);
                g64_copy<kTile, NT, true, L2>(st + GK * LA, Bm, ldb, rb, blim, k, kend);
            } else {
                g64_copy<BM, NT, false, L2>(st, Pj, ld, ra, nj, k, kend);
                g64_copy<kTile, NT, false, L2>(st + GK * LA, Bm, ldb, rb, blim, k, kend);
            }
            if (LDLT && L2 && tid < GK) {
                st[GK * (LA + LB) + tid] = dn;  // fetched a stage ahead
                const int kn = k + GK + tid;
                dn = kn < kend ? ld_l2(dj + kn) : 0.0;
            } else if (LDLT && ROLE != G_TRSM && tid < GK) {
                const bool ok = k + tid < kend;
                const unsigned sd = (unsigned)__cvta_generic_to_shared(st + GK * (LA + LB) + tid);
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(sd), "l"(dj + (ok ? k + tid : 0)),
                             "r"(ok ? 8 : 0)
                             : "memory");
            }
        }
        cp_commit();
    };
    double acc[MI][4][2];
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
#pragma unroll
    for (int c = 0; c < GStages - 1; ++c) load(c);
    double rd[4][2];  // TRSM of LDLt: reciprocal pivots of the thread's columns, formed beside the copies
    if (LDLT && ROLE == G_TRSM)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int col = c0 + wc + j * 8 + fk * 2 + e;
                rd[j][e] = col < chi ? 1.0 / d[f.col0 + col] : 1.0;
            }
    for (int c = 0; c < nchunk; ++c) {
        cp_wait<GStages - 2>();
        __syncthreads();
        load(c + GStages - 1);  // into the stage that every warp finished before this barrier
        const double* As = smem + (c % GStages) * STG;
        const double* Bs = As + GK * LA;
        const double* Ds = Bs + GK * LB;
#pragma unroll
        for (int k = 0; k < GK; k += 4) {
            double a[MI], b[4];
            const double s = (LDLT && ROLE != G_TRSM) ? Ds[k + fk] : 1.0;
#pragma unroll
            for (int i = 0; i < MI; ++i) {
                a[i] = As[(k + fk) * LA + wr + i * 8 + fr];
                if (LDLT && ROLE != G_TRSM) a[i] *= s;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = Bs[(k + fk) * LB + wc + j * 8 + fr];
#pragma unroll
            for (int i = 0; i < MI; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) dmma(acc[i][j][0], acc[i][j][1], a[i], b[j]);
        }
    }
    // C = -acc (SYRK), acc / d (TRSM) or C - acc: eight columns' worth of C is
    // read before the first of it is written
#pragma unroll
    for (int i = 0; i < MI; ++i) {
        const int row = ra + wr + i * 8 + fr;
        const bool rok = row >= rlo && row < rhi;
        double cv[4][2];
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int col = (ROLE == G_TRSM ? c0 : rb) + wc + j * 8 + fk * 2 + e;
                const bool ok = rok && col >= clo && col < chi && (!tri || row >= col);
                cv[j][e] = 0.0;
                if (ok && L2) cv[j][e] = ld_l2(C + row + (int64_t)col * ldc);
                else if (ok && ROLE == G_TRAIL) cv[j][e] = C[row + (int64_t)col * ldc];
            }
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int col = (ROLE == G_TRSM ? c0 : rb) + wc + j * 8 + fk * 2 + e;
                const bool ok = rok && col >= clo && col < chi && (!tri || row >= col);
                if (!ok) continue;
                double v = acc[i][j][e];
                if (ROLE == G_TRSM) {
                    if (LDLT) v *= rd[j][e];
                } else {
                    v = cv[j][e] - v;
                }
                C[row + (int64_t)col * ldc] = v;
            }
    }
    if (ROLE == G_LEFT) wait();
}

// ---------------------------------------------------------------------------
// 256x256 diagonal super-block inverses for the blocked solves, once after
// the factorization.  Super-block K of a front (columns k0 = 256 K ..) is
// made of up to four 64-column blocks with stored inverses D_s; its inverse
// X follows by block forward substitution down each column block t:
//   X_tt = D_t,   X_st = -D_s sum_{u=t}^{s-1} L_su X_ut   (s > t).
// Columns of X are independent, so a CTA takes 32 of one block's: item
// (front, K, 2 t + half).  Its X_ut stay in shared memory, and the next 64 x 64
// operand is on its way in registers while the current one is multiplied:
// doubles on DMMA (a warp 16 x 16 of the 64 x 32 product), floats as 4 x 2
// FMAs a thread.  What bounds it is the chain of at most nine products (and on
// trees of many super-blocks the reads of L).  One CTA for all of a
// super-block, its scalar products bound by shared-memory reads, took 213 us
// at 16^3, 267 us at KKT 24 and 804 us at 80^3 (FP64); this takes 33, 49 and
// 612 us.
// ---------------------------------------------------------------------------
constexpr int ILD = kNB + 1;
constexpr int kInvCols = kNB / 2;

template <typename T>
constexpr int inv256_smem() { return (kNB * ILD + 5 * kInvCols * ILD) * (int)sizeof(T); }

// C(64 x 32) += A(64 x 64) B(64 x 32): A[r + k * ILD], B[k + c * ILD]; visit()
// gives a thread's entries as (row, column, accumulator)
struct InvAccD {
    double c[2][2][2] = {};
    __device__ __forceinline__ void mma(const double* A, const double* B) {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const int wr = (warp & 3) * 16, wc = (warp >> 2) * 16, fr = lane >> 2, fk = lane & 3;
#pragma unroll 4
        for (int k = 0; k < kNB; k += 4) {
            double a[2], b[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) a[i] = A[(wr + 8 * i + fr) + (k + fk) * ILD];
#pragma unroll
            for (int j = 0; j < 2; ++j) b[j] = B[(k + fk) + (wc + 8 * j + fr) * ILD];
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j) dmma(c[i][j][0], c[i][j][1], a[i], b[j]);
        }
    }
    template <typename F>
    __device__ __forceinline__ void visit(F&& fn) {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const int wr = (warp & 3) * 16, wc = (warp >> 2) * 16;
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int e = 0; e < 2; ++e) fn(wr + 8 * i + (lane >> 2), wc + 8 * j + (lane & 3) * 2 + e, c[i][j][e]);
    }
};
struct InvAccF {
    float c[4][2] = {};
    __device__ __forceinline__ void mma(const float* A, const float* B) {
        const int tr = (threadIdx.x & 15) * 4, tc = (threadIdx.x >> 4) * 2;
#pragma unroll 8
        for (int k = 0; k < kNB; ++k) {
            float a[4], b[2];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = A[(tr + i) + k * ILD];
#pragma unroll
            for (int j = 0; j < 2; ++j) b[j] = B[k + (tc + j) * ILD];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j) c[i][j] += a[i] * b[j];
        }
    }
    template <typename F>
    __device__ __forceinline__ void visit(F&& fn) {
        const int tr = (threadIdx.x & 15) * 4, tc = (threadIdx.x >> 4) * 2;
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) fn(tr + i, tc + j, c[i][j]);
    }
};

template <typename T>
__global__ void __launch_bounds__(256) k_inv256(const Front* __restrict__ fronts, const Item* __restrict__ items,
                                                const T* __restrict__ P, const T* __restrict__ inv,
                                                T* __restrict__ inv2) {
    pdl_prologue();
    using Acc2 = typename std::conditional<sizeof(T) == 8, InvAccD, InvAccF>::type;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* As = reinterpret_cast<T*>(smem_raw);
    T* Cs = As + kNB * ILD;               // the sum of a block row, as the next product's operand
    T* Xs = Cs + kInvCols * ILD;          // X_ut, u = 0 .. 3
    const Item it = items[blockIdx.x];
    const Front f = fronts[it.front];
    const int K = it.a, t = it.b >> 1, cb = (it.b & 1) * kInvCols;
    const int k0 = K * kSolveNB, wK = min(kSolveNB, f.nn - k0), ns = (wK + kNB - 1) / kNB;
    const int ld2 = super_ld(wK), ld = f.ldp, tid = threadIdx.x;
    const int nc = min(kInvCols, wK - t * kNB - cb);  // columns of the piece
    T* X = inv2 + f.i2off + (int64_t)K * kSolveNB * kSolveNB + (int64_t)(t * kNB + cb) * ld2;
    const T* Pk = P + f.poff + k0 + (int64_t)k0 * ld;
    const T* Dk = inv + f.ioff + (int64_t)(k0 / kNB) * kNB * kNB;
    // zeros above the block row t and in the padding rows
    for (int e = tid; e < ld2 * nc; e += 256) {
        const int r = e % ld2, c = e / ld2;
        if (r < t * kNB || r >= wK) X[r + (int64_t)c * ld2] = T(0);
    }
    for (int e = tid; e < kNB * kInvCols; e += 256) {
        const int r = e & (kNB - 1), c = e >> 6;
        const T v = c < nc ? Dk[(int64_t)t * kNB * kNB + r + (cb + c) * kNB] : T(0);
        Xs[t * kInvCols * ILD + r + c * ILD] = v;
        if (c < nc && t * kNB + r < wK) X[t * kNB + r + (int64_t)c * ld2] = v;
    }
    // operands in the order they are needed: L_st .. L_s,s-1, D_s for each s
    T v[16];
    auto fetch = [&](int s, int u) {
        const int ws = min(kNB, wK - s * kNB);
        const T* src = u < s ? Pk + s * kNB + (int64_t)(u * kNB) * ld : Dk + (int64_t)s * kNB * kNB;
        const int64_t l = u < s ? ld : kNB;
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            const int e = tid + 256 * q, r = e & (kNB - 1), c = e >> 6;
            v[q] = r < ws ? src[r + c * l] : T(0);
        }
    };
    if (t + 1 < ns) fetch(t + 1, t);
    for (int s = t + 1; s < ns; ++s) {
        const int ws = min(kNB, wK - s * kNB);
        Acc2 sum, prod;
        for (int u = t; u <= s; ++u) {
            __syncthreads();  // As is free, Xs and Cs are whole
#pragma unroll
            for (int q = 0; q < 16; ++q) {
                const int e = tid + 256 * q;
                As[(e & (kNB - 1)) + (e >> 6) * ILD] = v[q];
            }
            if (u < s) fetch(s, u + 1);
            else if (s + 1 < ns) fetch(s + 1, t);
            __syncthreads();
            if (u < s) {
                sum.mma(As, Xs + u * kInvCols * ILD);
                if (u == s - 1) sum.visit([&](int r, int c, T x) { Cs[r + c * ILD] = x; });
            } else {
                prod.mma(As, Cs);
                prod.visit([&](int r, int c, T x) {
                    Xs[s * kInvCols * ILD + r + c * ILD] = -x;
                    if (r < ws && c < nc) X[s * kNB + r + (int64_t)c * ld2] = -x;
                });
            }
        }
    }
}

// ---------------------------------------------------------------------------
// launch helpers
// ---------------------------------------------------------------------------
Timer::Timer(mf_handle* h_, int k_) : h(h_), k(k_) {
    if (!h->profile) return;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    cudaEventRecord(a, h->stream);
}

Timer::~Timer() {
    if (!h->profile) return;
    cudaEventRecord(b, h->stream);
    cudaEventSynchronize(b);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, a, b);
    h->times.ms[k] += ms;
    h->times.launches[k] += 1;
    cudaEventDestroy(a);
    cudaEventDestroy(b);
}

static inline unsigned grid_for(int64_t cnt) { return (unsigned)cnt; }

template <typename T>
static int assemble_impl(mf_handle* h, const double* dnz, T* P, const double* scale) {
    Timer t(h, K_ASSEMBLE);
    MF_CUDA(cudaMemsetAsync(P, 0, sizeof(T) * h->npanel, h->stream));
    if (h->nnz > 0) {
        int64_t blocks = (h->nnz + 255) / 256;
        if (blocks > 148 * 16) blocks = 148 * 16;
        launch_k(k_scatter<T>, (unsigned)blocks, 256, 0, h->stream, P, h->d_pslot, dnz, h->nnz, h->d_nzrow, h->d_nzcol,
                                                               scale);
        MF_CUDA(cudaGetLastError());
    }
    return 0;
}

int launch_assemble(mf_handle* h, const double* dnz) {
    if (!have_fp64(h)) {
        set_error("no FP64 factor storage: a mixed handle has it only after an FP64 factorization");
        return -1;
    }
    return assemble_impl<double>(h, dnz, h->d_P, nullptr);
}

int launch_assemble_mixed(mf_handle* h, const double* dnz) {
    if (h->n > 0) {
        launch_k(k_diag_scale, (unsigned)((h->n + 255) / 256), 256, 0, h->stream, h->d_scale, h->d_dslot, dnz, h->n);
        MF_CUDA(cudaGetLastError());
    }
    return assemble_impl<float>(h, dnz, h->f32.P, h->d_scale);
}

int launch_dl_to_panel(mf_handle* h, const double* dD, const double* dL) {
    if (!have_fp64(h)) {
        set_error("no FP64 factor storage: a mixed handle has it only after an FP64 factorization");
        return -1;
    }
    Timer t(h, K_OTHER);
    if (h->n == 0) return 0;
    int64_t threads = h->n * 32;
    unsigned blocks = (unsigned)((threads + 255) / 256);
    MF_CUDA(cudaMemsetAsync(h->d_P, 0, sizeof(double) * h->npanel, h->stream));
    launch_k(k_dl_panel<true>, blocks, 256, 0, h->stream, h->d_fronts, h->d_ref, h->d_colfront, h->d_sepmap,
                                                     const_cast<double*>(dD), const_cast<double*>(dL), h->d_P, h->n);
    MF_CUDA(cudaGetLastError());
    return 0;
}

int launch_panel_to_dl(mf_handle* h, double* dD, double* dL) {
    if (!have_fp64(h)) {
        set_error("no FP64 factor storage: a mixed handle has it only after an FP64 factorization");
        return -1;
    }
    if (h->mixed && !h->fp64_current) {
        set_error("the FP64 factor storage does not hold the current matrix: the last mixed factorization "
                  "stayed in FP32");
        return -1;
    }
    Timer t(h, K_OTHER);
    if (h->n == 0) return 0;
    int64_t threads = h->n * 32;
    unsigned blocks = (unsigned)((threads + 255) / 256);
    launch_k(k_dl_panel<false>, blocks, 256, 0, h->stream, h->d_fronts, h->d_ref, h->d_colfront, h->d_sepmap, dD, dL,
                                                      h->d_P, h->n);
    MF_CUDA(cudaGetLastError());
    return 0;
}

int launch_panel32_to_dl(mf_handle* h, double* dD, double* dL) {
    if (h->n == 0) return 0;
    int64_t threads = h->n * 32;
    unsigned blocks = (unsigned)((threads + 255) / 256);
    launch_k(k_panel32_to_dl, blocks, 256, 0, h->stream, h->d_fronts, h->d_ref, h->d_colfront, h->d_sepmap, dD, dL,
                                                   h->f32.P, h->n);
    MF_CUDA(cudaGetLastError());
    return 0;
}


template <int BM, int ROLE, int LDLT>
static int gemm64_go(mf_handle* h, int64_t ctas, const Item* items, int obs, int obw, int c0,
                     const FactorBufs<double>& fb) {
    const bool pdl = early(h, pdl_enabled() || (h->panel_pdl && ROLE != G_TRAIL));
    MF_CUDA(cudaFuncSetAttribute(k_gemm64<BM, ROLE, LDLT>, cudaFuncAttributeMaxDynamicSharedMemorySize, g64_smem<BM>()));
    launch_kx(pdl, k_gemm64<BM, ROLE, LDLT>, grid_for(ctas), g64_threads<BM>(), g64_smem<BM>(), h->stream, h->d_fronts,
              items, obs, obw, c0, fb.P, fb.M, fb.d, fb.inv);
    MF_CUDA(cudaGetLastError());
    return 0;
}

// one role of the FP64 factorization: 128-row tiles when they give every SM at
// least two CTAs, else 64-row ones (a launch of fewer large tiles leaves SMs
// idle for a whole tile's time), 32-row ones when even those are fewer than
// the SMs
template <int ROLE, int LDLT>
static int gemm64(mf_handle* h, const ItemList& small, const ItemList& large, int obs, int obw, int c0,
                  const FactorBufs<double>& fb) {
    if (!small.cnt) return 0;
    const int64_t big = large.cnt * (ROLE == G_TRAIL || ROLE == G_SYRK ? 2 : 1), sms = h->num_sms > 0 ? h->num_sms : 148;
    const Item* items = h->d_items;
    if (big >= 2 * sms) return gemm64_go<128, ROLE, LDLT>(h, big, items + large.off, obs, obw, c0, fb);
    if (small.cnt >= sms) return gemm64_go<64, ROLE, LDLT>(h, small.cnt, items + small.off, obs, obw, c0, fb);
    return gemm64_go<32, ROLE, LDLT>(h, 2 * small.cnt, items + small.off, obs, obw, c0, fb);
}

// one role of a level's panel steps or SYRK without the tcgen05 tiles
template <typename T, int ROLE, int LDLT>
static int gemm_role(mf_handle* h, const ItemList& small, const ItemList& large, int obs, int obw, int c0,
                     const FactorBufs<T>& fb) {
    if constexpr (std::is_same<T, double>::value) {
        return gemm64<ROLE, LDLT>(h, small, large, obs, obw, c0, fb);
    } else {
        constexpr int gs = gemm_smem<T>();
        MF_CUDA(cudaFuncSetAttribute(k_gemm<T, ROLE, LDLT>, cudaFuncAttributeMaxDynamicSharedMemorySize, gs));
        launch_kx(early(h, pdl_enabled() || (h->panel_pdl && (ROLE == G_LEFT || ROLE == G_TRSM))), k_gemm<T, ROLE, LDLT>,
                  grid_for(small.cnt), 256, gs, h->stream, h->d_fronts, h->d_items + small.off, obs, obw, c0, fb.P, fb.M,
                  fb.d, fb.inv);
        MF_CUDA(cudaGetLastError());
        return 0;
    }
}

// k_small over one run of a level's small fronts of at most mj rows: 64
// threads up to 48 rows (two warps keep the barriers of the pivot chain
// short), 256 above.  Shared memory holds `stage` staged
// entries of children and a front of mj rows (as FP64 up to kSmallRescue
// rows, for the in-place rescue of an FP32 front).
template <typename T, int LDLT, bool REG, int TD, int R>
static int small_go(mf_handle* h, const ItemList& l, int mj, int stage, const FactorBufs<T>& fb, const Reg& reg) {
    const int rj = std::min(mj, kSmallRescue), lj = (mj + 3) & ~3;
    const size_t sm = std::max<size_t>(((size_t)stage + (size_t)lj * mj) * sizeof(T), sizeof(T) == 4 ? (size_t)rj * rj * 8 : 0);
    MF_CUDA(cudaFuncSetAttribute(k_small<T, LDLT, TD, R, REG>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (kSmallStage + kSmallMax * kSmallMax) * (int)sizeof(T)));
    launch_kx(early(h, h->panel_pdl || pdl_enabled()), k_small<T, LDLT, TD, R, REG>, grid_for(l.cnt), TD * TD, sm, h->stream, h->d_fronts,
             h->d_items + l.off, stage, h->d_reltgt, h->d_chdtgt, fb.P, fb.M, fb.d, h->d_signs, h->d_info,
             h->d_rescued, reg);
    MF_CUDA(cudaGetLastError());
    return 0;
}

template <typename T, int LDLT, bool REG>
static int launch_small(mf_handle* h, const ItemList& l, int mj, int stage, const FactorBufs<T>& fb, const Reg& reg) {
    if (mj <= 32) return small_go<T, LDLT, REG, 8, 4>(h, l, mj, stage, fb, reg);
    if (mj <= 48) return small_go<T, LDLT, REG, 8, 6>(h, l, mj, stage, fb, reg);
    if (mj <= 64) return small_go<T, LDLT, REG, 16, 4>(h, l, mj, stage, fb, reg);
    return small_go<T, LDLT, REG, 16, 6>(h, l, mj, stage, fb, reg);
}

template <typename T, int LDLT, bool REG>
static int factor_impl(mf_handle* h, const FactorBufs<T>& fb) {
    // the pivot rule applies to the FP64 factorization; the mixed form keeps
    // NoRegularization (its single-precision factor only preconditions)
    const Reg reg = std::is_same<T, double>::value ? h->reg : Reg();
    MF_CUDA(cudaFuncSetAttribute(k_small_warp<T, LDLT, kWarpSmallNJ>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 kWarpFronts * warp_slice<kWarpSmallNJ>()));
    MF_CUDA(cudaFuncSetAttribute(k_small_warp<T, LDLT, kWarpSmallNJ2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 kWarpFronts * warp_slice<kWarpSmallNJ2>()));
    // sub-panels after an outer block's first: the diagonal block's update in k_diag (FP64), or in LEFT's first tile
    constexpr bool upd = std::is_same<T, double>::value;
    MF_CUDA(cudaFuncSetAttribute(k_diag<T, LDLT, REG, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, diag_smem<T>()));
    MF_CUDA(cudaFuncSetAttribute(k_diag<T, LDLT, REG, upd>, cudaFuncAttributeMaxDynamicSharedMemorySize, diag_smem<T>()));
    MF_CUDA(cudaFuncSetAttribute(k_inv256<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, inv256_smem<T>()));
    const Item* items = h->d_items;
    // per-level timing while autotuning (profile mode: no graph, synchronised)
    cudaEvent_t tev[3] = {nullptr, nullptr, nullptr};
    if (h->tuning) {
        for (auto& e : tev) MF_CUDA(cudaEventCreate(&e));
        h->tune_steps_ms.assign(h->levels.size(), 0.0);
        h->tune_syrk_ms.assign(h->levels.size(), 0.0);
    }
    h->seq_begun = false;
    for (size_t L = 0; L < h->levels.size(); ++L) {
        const Level& lv = h->levels[L];
        if (lv.small_warp.cnt) {
            Timer t(h, K_SMALL);
            const unsigned g = (unsigned)((lv.small_warp.cnt + kWarpFronts - 1) / kWarpFronts);
            launch_k(k_small_warp<T, LDLT, kWarpSmallNJ>, g, kWarpFronts * 32, kWarpFronts * warp_slice<kWarpSmallNJ>(),
                h->stream, h->d_fronts, items + lv.small_warp.off, lv.small_warp.cnt, h->d_reltgt, h->d_chdtgt, fb.P,
                fb.M, fb.d, h->d_signs, h->d_info, h->d_rescued, reg);
            MF_CUDA(cudaGetLastError());
        }
        if (lv.small_warp2.cnt) {
            Timer t(h, K_SMALL);
            const unsigned g = (unsigned)((lv.small_warp2.cnt + kWarpFronts - 1) / kWarpFronts);
            launch_k(k_small_warp<T, LDLT, kWarpSmallNJ2>, g, kWarpFronts * 32,
                kWarpFronts * warp_slice<kWarpSmallNJ2>(), h->stream, h->d_fronts, items + lv.small_warp2.off,
                lv.small_warp2.cnt, h->d_reltgt, h->d_chdtgt, fb.P, fb.M, fb.d, h->d_signs, h->d_info, h->d_rescued,
                reg);
            MF_CUDA(cudaGetLastError());
        }
        if (lv.small_warp.cnt || lv.small_warp2.cnt) h->seq_begun = true;
        if (lv.small.cnt) {
            Timer t(h, K_SMALL);
            // one launch sized for the level's largest front; a level that
            // fills the SMs several times over takes one launch per size
            // class (a class of less than one front per SM joins the next)
            int64_t off = lv.small.off, cnt = 0;
            int stage = 0;
            for (int c = 0; c < kSmallClasses; ++c) {
                cnt += lv.small_cls[c];
                stage = std::max(stage, lv.small_stage[c]);
                const bool last = off + cnt == lv.small.off + lv.small.cnt;
                if (!cnt || (!last && (lv.small.cnt < kSmallWideLevel || cnt < 148))) continue;
                if (int rc = launch_small<T, LDLT, REG>(h, ItemList{off, cnt}, last ? lv.small_maxnj : kSmallClassNJ[c],
                                                   stage, fb, reg))
                    return rc;
                off += cnt;
                cnt = 0;
                stage = 0;
            }
        }
        if (lv.ea.cnt) {
            Timer t(h, K_EA);
            launch_kx(early(h, h->panel_pdl || pdl_enabled()), k_ea<T, 0>, grid_for(lv.ea.cnt), 256, 0, h->stream, h->d_fronts, items + lv.ea.off, items,
                                                                   h->d_reltgt, fb.P, fb.M);
            MF_CUDA(cudaGetLastError());
        }
        if (h->tuning) MF_CUDA(cudaEventRecord(tev[0], h->stream));
        // Look-ahead: an outer block's trailing update runs its tiles of the
        // next outer block's columns on `stream` and the rest on `side`,
        // beside the next block's sub-panels (which touch only their own
        // columns); `stream` waits for `side` before the next trailing update
        // (its columns overlap, and it reuses the split operands) and before
        // the SYRK.  The persistent tensor-core kernel on `side` leaves
        // side_free_sms SMs to the sub-panel kernels.  Profile and tuning runs
        // stay on one stream.
        const bool la_on = h->lookahead && h->side && !h->profile && !h->tuning;
        bool pending = false;
        auto join = [&]() -> int {
            if (pending) MF_CUDA(cudaStreamWaitEvent(h->stream, h->ev_join, 0));
            pending = false;
            return 0;
        };
        // launch `body` on `side` after the work queued on `stream` so far
        auto on_side = [&](const std::function<int()>& body) -> int {
            MF_CUDA(cudaEventRecord(h->ev_fork, h->stream));
            MF_CUDA(cudaStreamWaitEvent(h->side, h->ev_fork, 0));
            cudaStream_t main = h->stream;
            h->stream = h->side;
            h->grid_cap = std::max(1, (h->num_sms > 0 ? h->num_sms : 148) - h->side_free_sms);
            const int rc = body();
            h->grid_cap = 0;
            h->stream = main;
            if (rc) return rc;
            MF_CUDA(cudaEventRecord(h->ev_join, h->side));
            pending = true;
            return 0;
        };
        for (const PanelStep& st : lv.steps) {
            const int obs = st.b * lv.kob, obw = lv.kob;
            const int c0 = obs + st.s * kNB;
            auto launch_diag = [&](auto update) {
                launch_kx(early(h, h->panel_pdl || pdl_enabled()), k_diag<T, LDLT, REG, decltype(update)::value>,
                          grid_for(st.diag.cnt), 256, diag_smem<T>(), h->stream, h->d_fronts, items + st.diag.off, obs,
                          c0, fb.P, fb.inv, fb.d, h->d_signs, h->d_info, h->d_rescued, reg);
            };
            if (std::is_same<T, float>::value && h->use_tc && lv.tc_steps) {
                // single precision: the GEMM roles run on the tcgen05 tensor cores
                const FactorBufs<float>& f32b = reinterpret_cast<const FactorBufs<float>&>(fb);
                int rc;
                if (st.left_tc.cnt) {
                    Timer t(h, K_LEFT);
                    if ((rc = tc_launch(h, 0, st.left_tc, obs, obw, c0, f32b))) return rc;
                }
                if (st.diag.cnt) {
                    Timer t(h, K_DIAG);
                    launch_diag(std::false_type{});
                    MF_CUDA(cudaGetLastError());
                }
                if (st.panel_tc.cnt) {
                    Timer t(h, K_PANEL);
                    if ((rc = tc_launch(h, 3, st.panel_tc, obs, obw, c0, f32b))) return rc;
                }
                if (st.trail_tc.cnt) {
                    Timer t(h, K_UPDATE);
                    if ((rc = join())) return rc;
                    const bool la = la_on && st.trail_tc_ncrit > 0 && st.trail_tc_ncrit < st.trail_tc.cnt;
                    const ItemList crit{st.trail_tc.off, la ? st.trail_tc_ncrit : st.trail_tc.cnt};
                    rc = h->tc_split ? tc_launch_split(h, 1, crit, st.split_tc, obs, obw, c0, f32b)
                                     : tc_launch(h, 1, crit, obs, obw, c0, f32b);
                    if (rc) return rc;
                    if (la) {
                        const ItemList bulk{st.trail_tc.off + st.trail_tc_ncrit, st.trail_tc.cnt - st.trail_tc_ncrit};
                        rc = on_side([&]() {
                            return h->tc_split ? tc_launch_split(h, 1, bulk, ItemList{}, obs, obw, c0, f32b)
                                               : tc_launch(h, 1, bulk, obs, obw, c0, f32b);
                        });
                        if (rc) return rc;
                    }
                }
                continue;
            }
            if (!upd && st.left.cnt) {
                Timer t(h, K_LEFT);
                if (int rc = gemm_role<T, G_LEFT, LDLT>(h, st.left, st.left_tc, obs, obw, c0, fb)) return rc;
            }
            // FP64: the block's update, factor and inverse, and LEFT beside it.
            // LEFT takes no wait before it reads (see k_gemm64), so nothing
            // may come between the two, and LEFT follows no other kernel
            auto diag_and_left = [&]() -> int {
                {
                    Timer t(h, K_DIAG);
                    launch_diag(std::bool_constant<upd>{});
                    MF_CUDA(cudaGetLastError());
                }
                if (!st.panel.cnt) return 0;
                Timer t(h, K_LEFT);
                return gemm_role<T, G_LEFT, LDLT>(h, st.panel, st.panel_tc, obs, obw, c0, fb);
            };
            if (upd && st.s > 0) {
                if (int rc = diag_and_left()) return rc;
            } else if (st.diag.cnt) {
                Timer t(h, K_DIAG);
                launch_diag(std::false_type{});
                MF_CUDA(cudaGetLastError());
            }
            if (st.panel.cnt) {
                Timer t(h, K_PANEL);
                if (int rc = gemm_role<T, G_TRSM, LDLT>(h, st.panel, st.panel_tc, obs, obw, c0, fb)) return rc;
            }
            if (st.trail.cnt) {
                Timer t(h, K_UPDATE);
                if (int rc = join()) return rc;
                const bool la = la_on && st.trail_ncrit > 0 && st.trail_ncrit < st.trail.cnt;
                const int64_t n1 = la ? st.trail_ncrit : st.trail.cnt, n2 = la ? st.trail_tc_ncrit : st.trail_tc.cnt;
                if (int rc = gemm_role<T, G_TRAIL, LDLT>(h, ItemList{st.trail.off, n1}, ItemList{st.trail_tc.off, n2}, obs,
                                                         obw, c0, fb))
                    return rc;
                if (la) {
                    const int rc = on_side([&]() -> int {
                        return gemm_role<T, G_TRAIL, LDLT>(h, ItemList{st.trail.off + n1, st.trail.cnt - n1},
                                                           ItemList{st.trail_tc.off + n2, st.trail_tc.cnt - n2}, obs, obw,
                                                           c0, fb);
                    });
                    if (rc) return rc;
                }
            }
        }
        if (int rc = join()) return rc;
        if (h->tuning) MF_CUDA(cudaEventRecord(tev[1], h->stream));
        if (std::is_same<T, float>::value && h->use_tc && lv.tc_syrk) {
            if (lv.syrk_tc.cnt) {
                Timer t(h, K_SYRK);
                const FactorBufs<float>& f32b = reinterpret_cast<const FactorBufs<float>&>(fb);
                int rc = h->tc_split ? tc_launch_split(h, 2, lv.syrk_tc, lv.split_syrk, 0, 0, 0, f32b)
                                     : tc_launch(h, 2, lv.syrk_tc, 0, 0, 0, f32b);
                if (rc) return rc;
            }
        } else if (lv.syrk.cnt) {
            Timer t(h, K_SYRK);
            if (int rc = gemm_role<T, G_SYRK, LDLT>(h, lv.syrk, lv.syrk_tc, 0, 0, 0, fb)) return rc;
        }
        if (lv.ea_upd.cnt) {
            Timer t(h, K_EA);
            launch_kx(early(h, h->panel_pdl || pdl_enabled()), k_ea<T, 1>, grid_for(lv.ea_upd.cnt), 256, 0, h->stream, h->d_fronts, items + lv.ea_upd.off, items,
                                                                       h->d_reltgt, fb.P, fb.M);
            MF_CUDA(cudaGetLastError());
        }
        if (h->tuning) {
            MF_CUDA(cudaEventRecord(tev[2], h->stream));
            MF_CUDA(cudaEventSynchronize(tev[2]));
            float a = 0.f, b = 0.f;
            MF_CUDA(cudaEventElapsedTime(&a, tev[0], tev[1]));
            MF_CUDA(cudaEventElapsedTime(&b, tev[1], tev[2]));
            h->tune_steps_ms[L] += a;
            h->tune_syrk_ms[L] += b;
        }
    }
    if (h->tuning)
        for (auto& e : tev) cudaEventDestroy(e);
    if (h->inv2_items.cnt) {
        Timer t(h, K_OTHER);
        launch_k(k_inv256<T>, grid_for(h->inv2_items.cnt), 256, inv256_smem<T>(), h->stream, 
            h->d_fronts, items + h->inv2_items.off, fb.P, fb.inv, fb.inv2);
        MF_CUDA(cudaGetLastError());
    }
    return 0;
}

int run_captured(mf_handle* h, int64_t k0, int64_t k1, int64_t k2, int64_t k3, const std::function<int()>& body) {
    if (!h->use_graphs || h->profile || h->tuning || !h->stream) return body();
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    MF_CUDA(cudaStreamIsCapturing(h->stream, &cs));
    if (cs != cudaStreamCaptureStatusNone) return body();
    for (const GraphEntry& g : h->graphs)
        if (g.key[0] == k0 && g.key[1] == k1 && g.key[2] == k2 && g.key[3] == k3) {
            MF_CUDA(cudaGraphLaunch(g.exec, h->stream));
            return 0;
        }
    std::lock_guard<std::recursive_mutex> lk(device_mutex());
    MF_CUDA(cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal));
    const int rc = body();
    cudaGraph_t graph = nullptr;
    const cudaError_t e = cudaStreamEndCapture(h->stream, &graph);
    if (rc || e != cudaSuccess) {
        if (graph) cudaGraphDestroy(graph);
        cudaGetLastError();
        return rc ? rc : cuda_fail(e, "cudaStreamEndCapture");
    }
    cudaGraphExec_t exec = nullptr;
    const cudaError_t ei = cudaGraphInstantiate(&exec, graph, 0);
    cudaGraphDestroy(graph);
    if (ei != cudaSuccess) return cuda_fail(ei, "cudaGraphInstantiate");
    h->graphs.push_back(GraphEntry{{k0, k1, k2, k3}, exec});
    MF_CUDA(cudaGraphLaunch(exec, h->stream));
    return 0;
}

void release_graphs(mf_handle* h) {
    for (GraphEntry& g : h->graphs)
        if (g.exec) cudaGraphExecDestroy(g.exec);
    h->graphs.clear();
}

// graph keys: kind (1 FP64 factor, 2 FP32 factor), then what the launch
// sequence reads through pointers that can change between calls
int launch_factor(mf_handle* h) {
    if (!have_fp64(h)) {
        set_error("no FP64 factor storage: a mixed handle has it only after an FP64 factorization");
        return -1;
    }
    FactorBufs<double> fb{h->d_P, h->d_M, h->d_inv, h->d_d, h->d_inv2};
    int rc = run_captured(h, 1, (int64_t)(uintptr_t)h->d_signs, 0, 0, [&]() {
        if (h->reg.delta >= 0.0) return h->diag ? factor_impl<double, 1, true>(h, fb) : factor_impl<double, 0, true>(h, fb);
        return h->diag ? factor_impl<double, 1, false>(h, fb) : factor_impl<double, 0, false>(h, fb);
    });
    h->fp64_current = rc == 0;
    h->selinv_done = false;
    return rc;
}

int launch_factor_mixed(mf_handle* h) {
    FactorBufs<float> fb{h->f32.P, h->f32.M, h->f32.inv, h->f32.d, h->f32.inv2};
    if (h->use_tc) {
        int rc = tc_prepare(h);
        if (rc) return rc;
    }
    return run_captured(h, 2, (int64_t)(uintptr_t)h->d_signs, h->use_tc ? 1 : 0, 0, [&]() {
        return h->diag ? factor_impl<float, 1, false>(h, fb) : factor_impl<float, 0, false>(h, fb);
    });
}

}  // namespace mf

// ---------------------------------------------------------------------------
// log|det| of the factored matrix, reduced on the device
// (LinearAlgebra.logabsdet / logdet / det of a ChordalFactorization,
// src/Multifrontal.jl/src/abstract_factorization.jl:156-179).  Cholesky: the
// terms are log of the squared diagonal of L; LDLt: log|d_j| and the sign of
// d_j.  A mixed handle without an FP64 factor uses its single-precision factor
// of S A S and adds -2 log s_j.  Each block reduces a contiguous range of
// columns in a fixed tree order and writes (sum, negatives, zeros); the host
// adds the block results in block order, so the result is bitwise repeatable.
// ---------------------------------------------------------------------------
namespace mf {

constexpr int kLogdetThreads = 256;
constexpr int kLogdetBlocks = 296;  // 2 x 148 SMs

template <typename T, int UNIT>
__global__ void __launch_bounds__(kLogdetThreads)
k_logdet(const Front* __restrict__ fronts, const RefFront* __restrict__ ref, const int32_t* __restrict__ colref,
         const T* __restrict__ P, const T* __restrict__ d, const double* __restrict__ scale, int64_t n,
         double* __restrict__ out) {
    pdl_prologue();
    __shared__ double s_sum[kLogdetThreads];
    __shared__ int s_neg[kLogdetThreads], s_zero[kLogdetThreads];
    const int64_t per = (n + gridDim.x - 1) / gridDim.x;
    const int64_t c0 = blockIdx.x * per;
    const int64_t c1 = c0 + per < n ? c0 + per : n;
    double acc = 0.0;
    int neg = 0, zero = 0;
    for (int64_t c = c0 + threadIdx.x; c < c1; c += kLogdetThreads) {
        double v;
        if (UNIT) {
            v = (double)d[c];
        } else {
            const RefFront rf = ref[colref[c]];
            const Front f = fronts[rf.exec];
            const int64_t k = c - f.col0;
            const double l = (double)P[f.poff + k + k * f.ldp];
            v = l * l;
        }
        if (scale) v /= scale[c] * scale[c];
        if (v == 0.0) zero += 1;
        if (v < 0.0) neg += 1;
        acc += log(fabs(v));
    }
    s_sum[threadIdx.x] = acc;
    s_neg[threadIdx.x] = neg;
    s_zero[threadIdx.x] = zero;
    __syncthreads();
    for (int w = kLogdetThreads / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) {
            s_sum[threadIdx.x] += s_sum[threadIdx.x + w];
            s_neg[threadIdx.x] += s_neg[threadIdx.x + w];
            s_zero[threadIdx.x] += s_zero[threadIdx.x + w];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        out[3 * blockIdx.x] = s_sum[0];
        out[3 * blockIdx.x + 1] = (double)s_neg[0];
        out[3 * blockIdx.x + 2] = (double)s_zero[0];
    }
}

int launch_logdet(mf_handle* h, double* logabsdet, double* sign) {
    const bool fp64 = have_fp64(h) && (!h->mixed || h->fp64_current);
    if (!fp64 && !h->mixed) {
        set_error("mf_logdet: no factor on the device");
        return -1;
    }
    if (!h->d_logdet) {
        std::lock_guard<std::recursive_mutex> lk(device_mutex());
        MF_CUDA(cudaMalloc((void**)&h->d_logdet, sizeof(double) * 3 * kLogdetBlocks));
        h->bytes += (int64_t)sizeof(double) * 3 * kLogdetBlocks;
    }
    double* part = h->d_logdet;
    const int64_t n = h->n;
    if (n > 0) {
        if (fp64) {
            if (h->diag)
                launch_k(k_logdet<double, 1>, kLogdetBlocks, kLogdetThreads, 0, h->stream, 
                    h->d_fronts, h->d_ref, h->d_colfront, h->d_P, h->d_d, nullptr, n, part);
            else
                launch_k(k_logdet<double, 0>, kLogdetBlocks, kLogdetThreads, 0, h->stream, 
                    h->d_fronts, h->d_ref, h->d_colfront, h->d_P, h->d_d, nullptr, n, part);
        } else {
            if (h->diag)
                launch_k(k_logdet<float, 1>, kLogdetBlocks, kLogdetThreads, 0, h->stream, 
                    h->d_fronts, h->d_ref, h->d_colfront, h->f32.P, h->f32.d, h->d_scale, n, part);
            else
                launch_k(k_logdet<float, 0>, kLogdetBlocks, kLogdetThreads, 0, h->stream, 
                    h->d_fronts, h->d_ref, h->d_colfront, h->f32.P, h->f32.d, h->d_scale, n, part);
        }
        MF_CUDA(cudaGetLastError());
    }
    std::vector<double> hp(3 * kLogdetBlocks, 0.0);
    cudaError_t e = cudaSuccess;
    if (n > 0)
        e = cudaMemcpyAsync(hp.data(), part, sizeof(double) * 3 * kLogdetBlocks, cudaMemcpyDeviceToHost, h->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
    if (e != cudaSuccess) return cuda_fail(e, "mf_logdet");
    double sum = 0.0, neg = 0.0, zero = 0.0;
    for (int b = 0; b < kLogdetBlocks; ++b) {
        sum += hp[3 * b];
        neg += hp[3 * b + 1];
        zero += hp[3 * b + 2];
    }
    *logabsdet = zero > 0 ? -INFINITY : sum;
    *sign = zero > 0 ? 0.0 : (fmod(neg, 2.0) == 0.0 ? 1.0 : -1.0);
    return 0;
}

}  // namespace mf
