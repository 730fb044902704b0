// Forward and backward solves of the small fronts of a narrow tree level, one
// CTA per front (mf_solve.cu has the solves of everything else and describes
// the vectors C and R).
//
// A level of few fronts is a chain of dependent steps, not a stream: with a
// warp per front (k_s_small_*) it waits for a memory trip per four columns, per
// 64 rows of L21 and per child, and with sixteen right-hand sides one warp
// does all their products.  Here a front's whole panel is copied to shared
// memory at once -- before the kernel waits for the level below, as no solve
// writes panels -- then warps share the right-hand sides and rows, and the
// column chain runs on shared memory with the reciprocal diagonal formed ahead
// of it.  Every entry gets k_s_small_*'s operations in the same order, so the
// results are bitwise equal to them, and a front may take either path (a
// batch's wide level, the same matrix's narrow level alone).
//
// Measured, both directions of all narrow levels: 100^2 FP64, one right-hand
// side, 640 -> 260 us; 16^3 FP64, sixteen, 2.4 -> 0.45 ms; batch of 512 2D
// systems, FP32, four, three solves, 3.4 -> 1.7 ms.
#include <algorithm>
#include <type_traits>

#include "mf_internal.cuh"

namespace mf {

namespace {

constexpr int kCtaThreads = 128, kCtaWarps = kCtaThreads / 32;
constexpr int kCtaKids = 16;                         // child records fetched at once
constexpr int kCtaChunks = (kSmallMax + 31) / 32;    // rows per lane in the column chain

__device__ __forceinline__ void copy16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// leading dimension of a panel in the backward kernel's shared memory: an odd
// number of 16-byte units, so that lanes on neighbouring columns read their
// 16-byte groups of rows from different banks
template <typename T>
__host__ __device__ constexpr int pad_ld(int ldp) {
    return ((ldp * (int)sizeof(T) / 16) & 1) ? ldp : ldp + 16 / (int)sizeof(T);
}

// right-hand sides a warp takes at once in the column chain
template <int NR>
constexpr int rhs_per_warp() { return NR > kCtaWarps ? NR / kCtaWarps : 1; }

// right-hand sides a thread takes at once in the products with L21: few, so that
// the rows (columns) of a small front times the groups fill the CTA
template <int NR>
constexpr int rhs_per_thread() { return NR >= 8 ? 4 : NR >= 4 ? 2 : 1; }

// The triangular solve of one front by the CTA, vectors V[k + r * ldv] in
// shared memory, L(i, k) at L[i * ri + k * rk]: forward (BWD = 0) columns
// ascending, x_k = v_k / L_kk, then the rows after k lose L_ak x_k; backward
// columns descending on L^T.  A warp takes rhs_per_warp right-hand sides,
// lane i their rows i, i + 32, i + 64.
template <typename T, int UNIT, int NR, int BWD>
__device__ __forceinline__ void column_chain(const T* L, int ld, const T* rinv, T* V, int ldv, int nn, int nrhs, T* C,
                                             int64_t n) {
    constexpr int Q = rhs_per_warp<NR>();
    const int lane = threadIdx.x & 31, r0 = (threadIdx.x >> 5) * Q;
    if (r0 >= NR) return;
    T x[kCtaChunks][Q];
#pragma unroll
    for (int s = 0; s < kCtaChunks; ++s)
#pragma unroll
        for (int r = 0; r < Q; ++r) {
            const int a = lane + 32 * s;
            x[s][r] = a < nn ? V[a + (r0 + r) * ldv] : T(0);
        }
    auto chunk = [&](auto ks_) {
        constexpr int ks = decltype(ks_)::value;
        const int kb = 32 * ks, ke = min(nn, kb + 32);
#pragma unroll 4
        for (int q = 0; q < ke - kb; ++q) {
            const int k = BWD ? ke - 1 - q : kb + q;
            T l[kCtaChunks];
#pragma unroll
            for (int s = 0; s < kCtaChunks; ++s) {
                const int a = lane + 32 * s;
                l[s] = T(0);
                if (BWD ? (s <= ks && a < k) : (s >= ks && a > k && a < nn)) l[s] = BWD ? L[k + a * ld] : L[a + k * ld];
            }
            const T d = UNIT ? T(1) : rinv[k];
#pragma unroll
            for (int r = 0; r < Q; ++r) {
                const T xk = __shfl_sync(0xffffffffu, x[ks][r], k & 31) * d;
#pragma unroll
                for (int s = 0; s < kCtaChunks; ++s)
                    if (BWD ? s <= ks : s >= ks) x[s][r] -= l[s] * xk;
                if (lane == (k & 31)) x[ks][r] = xk;
            }
        }
    };
    if (BWD) {
        if (nn > 64) chunk(std::integral_constant<int, 2>());
        if (nn > 32) chunk(std::integral_constant<int, 1>());
        chunk(std::integral_constant<int, 0>());
    } else {
        chunk(std::integral_constant<int, 0>());
        if (nn > 32) chunk(std::integral_constant<int, 1>());
        if (nn > 64) chunk(std::integral_constant<int, 2>());
    }
#pragma unroll
    for (int s = 0; s < kCtaChunks; ++s)
#pragma unroll
        for (int r = 0; r < Q; ++r) {
            const int a = lane + 32 * s;
            if (a < nn) {
                V[a + (r0 + r) * ldv] = x[s][r];
                if (r0 + r < nrhs) C[a + (int64_t)(r0 + r) * n] = x[s][r];
            }
        }
}

// pan: shared-memory entries of the panel; ldv: rows of the vectors
template <typename T, int UNIT, int NR>
__global__ void __launch_bounds__(kCtaThreads) k_s_cta_fwd(const Front* __restrict__ fronts,
                                                           const Item* __restrict__ items, int pan, int ldv,
                                                           const int32_t* __restrict__ reltgt,
                                                           const int32_t* __restrict__ chdtgt,
                                                           const T* __restrict__ P, T* C, T* R, int64_t n, int nrhs) {
    pdl_trigger();
    extern __shared__ __align__(16) unsigned char sm_raw[];
    __shared__ int kid_na[kCtaKids], kid_sep0[kCtaKids];
    __shared__ int64_t kid_roff[kCtaKids];
    T* Ps = reinterpret_cast<T*>(sm_raw);
    T* V = Ps + pan;           // V[a + r * ldv]
    T* rinv = V + ldv * NR;    // 1 / L_kk
    const Front f = fronts[items[blockIdx.x].front];
    const int nn = f.nn, na = f.na, nj = nn + na, ld = f.ldp;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int W = 16 / (int)sizeof(T);
    for (int i = W * tid; i < ld * nn; i += W * kCtaThreads) copy16(Ps + i, P + f.poff + i);
    copy_commit();
    const int nch = f.chd1 - f.chd0;
    for (int q = tid; q < min(nch, kCtaKids); q += kCtaThreads) {
        const Front fc = fronts[chdtgt[f.chd1 - 1 - q]];
        kid_na[q] = fc.na, kid_sep0[q] = fc.sep0, kid_roff[q] = fc.roff;
    }
    grid_wait();
    T* Cj = C + f.col0;
    for (int r = warp; r < NR; r += kCtaWarps)
        for (int a = lane; a < nj; a += 32) V[a + r * ldv] = (a < nn && r < nrhs) ? __ldcg(Cj + a + (int64_t)r * n) : T(0);
    // children in reverse order (the reference pops its stack), four at a
    // time: a thread's first entry of each is loaded before the first is added
    for (int k0 = 0; k0 < nch; k0 += kCtaKids) {
        if (k0 > 0) {
            for (int q = tid; q < min(nch - k0, kCtaKids); q += kCtaThreads) {
                const Front fc = fronts[chdtgt[f.chd1 - 1 - k0 - q]];
                kid_na[q] = fc.na, kid_sep0[q] = fc.sep0, kid_roff[q] = fc.roff;
            }
        }
        __syncthreads();
        const int m = min(nch - k0, kCtaKids);
        for (int q0 = 0; q0 < m; q0 += 4) {
            int at[4];
            T mv[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                at[u] = -1;
                mv[u] = T(0);
                if (q0 + u < m) {
                    const int ma = kid_na[q0 + u];
                    if (tid < ma * nrhs) {
                        const int a = tid % ma, r = tid / ma;
                        at[u] = reltgt[kid_sep0[q0 + u] + a] + r * ldv;
                        mv[u] = __ldcg(R + kid_roff[q0 + u] * nrhs + tid);
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (q0 + u >= m) continue;  // uniform
                if (at[u] >= 0) V[at[u]] += mv[u];
                const int ma = kid_na[q0 + u];
                const int32_t* rel = reltgt + kid_sep0[q0 + u];
                const T* Mc = R + kid_roff[q0 + u] * nrhs;
#pragma unroll 4
                for (int i = tid + kCtaThreads; i < ma * nrhs; i += kCtaThreads)
                    V[rel[i % ma] + (i / ma) * ldv] += __ldcg(Mc + i);
                __syncthreads();
            }
        }
    }
    copy_wait();
    __syncthreads();
    if (!UNIT) {
        for (int k = tid; k < nn; k += kCtaThreads) rinv[k] = T(1) / Ps[k + k * ld];
        __syncthreads();
    }
    column_chain<T, UNIT, NR, 0>(Ps, ld, rinv, V, ldv, nn, nrhs, Cj, n);
    __syncthreads();
    // R_j = (child sums) - L21 x, a thread per row and group of right-hand sides
    constexpr int Q = rhs_per_thread<NR>(), G = NR / Q;
    T* Rj = R + f.roff * nrhs;
    for (int i = tid; i < na * G; i += kCtaThreads) {
        const int a = i % na, r0 = (i / na) * Q;
        const T* l = Ps + nn + a;
        T acc[Q];
#pragma unroll
        for (int r = 0; r < Q; ++r) acc[r] = T(0);
#pragma unroll 4
        for (int k = 0; k < nn; ++k) {
            const T lv = l[k * ld];
#pragma unroll
            for (int r = 0; r < Q; ++r) acc[r] += lv * V[k + (r0 + r) * ldv];
        }
#pragma unroll
        for (int r = 0; r < Q; ++r)
            if (r0 + r < nrhs) Rj[a + (int64_t)(r0 + r) * na] = V[nn + a + (r0 + r) * ldv] - acc[r];
    }
}

template <typename T, int UNIT, int NR>
__global__ void __launch_bounds__(kCtaThreads) k_s_cta_bwd(const Front* __restrict__ fronts,
                                                           const Item* __restrict__ items, int pan, int ldv,
                                                           const int32_t* __restrict__ septgt,
                                                           const T* __restrict__ P, T* C, int64_t n, int nrhs) {
    pdl_trigger();
    extern __shared__ __align__(16) unsigned char sm_raw[];
    T* Ps = reinterpret_cast<T*>(sm_raw);
    T* V = Ps + pan;           // V[a + r * ldv]: rows of the front, then x[sep]
    T* rinv = V + ldv * NR;    // 1 / L_kk
    const Front f = fronts[items[blockIdx.x].front];
    const int nn = f.nn, na = f.na, nj = nn + na, ld = pad_ld<T>(f.ldp);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int W = 16 / (int)sizeof(T);
    for (int c = warp; c < nn; c += kCtaWarps)
        for (int i = W * lane; i < f.ldp; i += W * 32) copy16(Ps + c * ld + i, P + f.poff + (int64_t)c * f.ldp + i);
    copy_commit();
    const int32_t* sep = septgt + f.sep0;
    T* Cj = C + f.col0;
    grid_wait();
    for (int r = warp; r < NR; r += kCtaWarps)
        for (int a = lane; a < nj; a += 32)
            V[a + r * ldv] = r < nrhs ? __ldcg((a < nn ? Cj + a : C + sep[a - nn]) + (int64_t)r * n) : T(0);
    copy_wait();
    __syncthreads();
    if (!UNIT)
        for (int k = tid; k < nn; k += kCtaThreads) rinv[k] = T(1) / Ps[k + k * ld];
    // C1 - L21^T x[sep]: a thread per column and group of right-hand sides,
    // rows in order, 16 bytes of the column at a time
    constexpr int Q = rhs_per_thread<NR>(), G = NR / Q;
    for (int i = tid; i < nn * G; i += kCtaThreads) {
        const int k = i % nn, r0 = (i / nn) * Q;
        const T* l = Ps + k * ld;
        const T* v = V + r0 * ldv;
        T acc[Q];
#pragma unroll
        for (int r = 0; r < Q; ++r) acc[r] = T(0);
        int a0 = nn;
        for (; (a0 & (W - 1)) && a0 < nj; ++a0)  // up to the first aligned row
#pragma unroll
            for (int r = 0; r < Q; ++r) acc[r] += l[a0] * v[a0 + r * ldv];
#pragma unroll 2
        for (; a0 + W <= nj; a0 += W) {
            T lv[W];
            *reinterpret_cast<int4*>(lv) = *reinterpret_cast<const int4*>(l + a0);
#pragma unroll
            for (int e = 0; e < W; ++e)
#pragma unroll
                for (int r = 0; r < Q; ++r) acc[r] += lv[e] * v[a0 + e + r * ldv];
        }
        for (; a0 < nj; ++a0)
#pragma unroll
            for (int r = 0; r < Q; ++r) acc[r] += l[a0] * v[a0 + r * ldv];
#pragma unroll
        for (int r = 0; r < Q; ++r) V[k + (r0 + r) * ldv] -= acc[r];
    }
    __syncthreads();
    column_chain<T, UNIT, NR, 1>(Ps, ld, rinv, V, ldv, nn, nrhs, Cj, n);
}

template <typename T, int UNIT, int NR>
int cta_go(mf_handle* h, const CtaList& l, const SolveBufs<T>& sb, int bwd, int nrhs) {
    const Item* it = h->d_items + l.items.off;
    const unsigned g = (unsigned)l.items.cnt;
    const int pan = bwd ? (sizeof(T) == 4 ? l.pad32 : l.pad64) : l.panel;
    const size_t sm = ((size_t)pan + (size_t)l.rows * NR + kSmallMax) * sizeof(T);
    if (!bwd) {
        MF_CUDA(cudaFuncSetAttribute(k_s_cta_fwd<T, UNIT, NR>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem));
        launch_kx(early(h, h->step_pdl), k_s_cta_fwd<T, UNIT, NR>, g, kCtaThreads, sm, h->stream, h->d_fronts, it, pan,
                  l.rows, h->d_reltgt, h->d_chdtgt, sb.P, sb.C, sb.R, h->n, nrhs);
    } else {
        MF_CUDA(cudaFuncSetAttribute(k_s_cta_bwd<T, UNIT, NR>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem));
        launch_kx(early(h, h->step_pdl), k_s_cta_bwd<T, UNIT, NR>, g, kCtaThreads, sm, h->stream, h->d_fronts, it, pan,
                  l.rows, h->d_septgt, sb.P, sb.C, h->n, nrhs);
    }
    MF_CUDA(cudaGetLastError());
    return 0;
}

template <typename T, int UNIT>
int cta_rhs(mf_handle* h, const CtaList& l, const SolveBufs<T>& sb, int bwd, int nrb, int nrhs) {
    Timer t(h, K_S_SMALL);
    switch (nrb) {
        case 1: return cta_go<T, UNIT, 1>(h, l, sb, bwd, nrhs);
        case 2: return cta_go<T, UNIT, 2>(h, l, sb, bwd, nrhs);
        case 4: return cta_go<T, UNIT, 4>(h, l, sb, bwd, nrhs);
        case 8: return cta_go<T, UNIT, 8>(h, l, sb, bwd, nrhs);
        default: return cta_go<T, UNIT, 16>(h, l, sb, bwd, nrhs);
    }
}

}  // namespace

int launch_solve_cta(mf_handle* h, const Level& lv, const SolveBufs<double>& sb, int bwd, int nrb, int nrhs) {
    return h->diag ? cta_rhs<double, 1>(h, lv.s_cta, sb, bwd, nrb, nrhs) : cta_rhs<double, 0>(h, lv.s_cta, sb, bwd, nrb, nrhs);
}
int launch_solve_cta(mf_handle* h, const Level& lv, const SolveBufs<float>& sb, int bwd, int nrb, int nrhs) {
    return h->diag ? cta_rhs<float, 1>(h, lv.s_cta, sb, bwd, nrb, nrhs) : cta_rhs<float, 0>(h, lv.s_cta, sb, bwd, nrb, nrhs);
}

}  // namespace mf
