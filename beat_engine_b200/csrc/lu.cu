// lu.cu -- blocked right-looking complex LU with partial pivoting, and the
// multi-right-hand-side triangular solves, on one B200.
//
// Replaces the reference's lu!(system.matrix) / factorization \ rhs
// (BeatEngineCompiledDriver.jl:902-903 -> cuSOLVER getrf/getrs through
// CUDA.jl, and OpenBLAS zgetrf on the CPU path, BeatEngineDenseSolve.jl:1104-1110).
// Pivoting is the partial pivoting LAPACK uses (first maximum of |re| + |im|
// in the column), so the factorisation is P A = L U with unit-lower L.
//
// Layout: A is row-major complex, row stride ld (complex entries).  Row
// interchanges are then contiguous copies.
//
// Per panel of nb columns:
//   1. cluster_panel_kernel (cluster_panel.cu): a thread-block cluster factors each sub-panel (32
//      FP32 or 16 FP64 columns), its rows in registers, one exchange per column
//      (panel_kernel, a cooperative kernel with one grid-wide barrier per
//      column, where the rows do not fit a cluster), then the rest of the
//      panel is solved and updated.
//   2. laswp_panel_kernel: the panel's interchanges on all other columns (and
//      on the running row permutation).
//   3. U12 = L11^-1 A12 (trsm_narrow_kernel, trsm_blocked_kernel; the FP64
//      form's trailing columns trsm_mma_kernel).
//   4. trailing update A22 -= L21 U12: FP64 tensor cores (dmma_update_kernel), or
//      tcgen05 FP16-split products in the FP32 form (tc_gemm.cu).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <utility>

#include "lu.cuh"

namespace bb {

// L2-coherent loads of values other CTAs published before a grid barrier
__device__ __forceinline__ Cx<double> ldcg(const Cx<double> *p) {
    const double2 v = __ldcg(reinterpret_cast<const double2 *>(p));
    return Cx<double>{v.x, v.y};
}
__device__ __forceinline__ Cx<float> ldcg(const Cx<float> *p) {
    const float2 v = __ldcg(reinterpret_cast<const float2 *>(p));
    return Cx<float>{v.x, v.y};
}
__device__ __forceinline__ double ldcg(const double *p) { return __ldcg(p); }
__device__ __forceinline__ float ldcg(const float *p) { return __ldcg(p); }
__device__ __forceinline__ int ldcg(const int *p) { return __ldcg(p); }

// Pivot candidate of one CTA for one column (value |re| + |im| and global row).
struct PivotRec {
    double val;
    int idx;
    int pad;
};

template <typename T> struct PanelArgs {
    Cx<T> *A;
    int64_t ld;
    int n, k, nb;
    int rpc;            // rows per CTA
    int *ipiv;
    Cx<T> *pub_rows;    // [2][G][nb]
    Cx<T> *pub_diag;    // [2][nb]
    PivotRec *recs;     // [2][G]
    unsigned *counter;  // grid-barrier arrivals of this panel launch (zeroed before it)
    int *status;
    unsigned spin_limit;
};

constexpr int PANEL_THREADS = 256;

template <typename T> __global__ void __launch_bounds__(PANEL_THREADS) panel_kernel(PanelArgs<T> a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int nb = a.nb, G = gridDim.x, cta = blockIdx.x, tid = threadIdx.x;
    Cx<T> *P = reinterpret_cast<Cx<T> *>(smem_raw);  // rpc x nb
    Cx<T> *prow = P + (size_t)a.rpc * nb;             // nb
    Cx<T> *drow = prow + nb;                          // nb
    Cx<T> *lcol = drow + nb;                          // rpc
    __shared__ T red_v[PANEL_THREADS / 32];
    __shared__ int red_i[PANEL_THREADS / 32];
    __shared__ int red_c[PANEL_THREADS / 32];
    __shared__ int s_piv;
    __shared__ T s_pv;

    const int gr0 = a.k + cta * a.rpc;
    const int nrows = max(0, min(a.rpc, a.n - gr0));
    batched_copy<PANEL_THREADS, 8, Cx<T>>(
        nrows * nb, [&](int i) { return a.A[(int64_t)(gr0 + i / nb) * a.ld + a.k + i % nb]; },
        [&](int i, Cx<T> v) { P[i] = v; });
    __syncthreads();

    for (int j = 0; j < nb && a.k + j < a.n; ++j) {
        const int jr = a.k + j, par = j & 1;
        // local candidate: first maximum of |re|+|im| among own rows >= jr
        T bv = T(-1);
        int bi = -1;
        for (int i = tid; i < nrows; i += PANEL_THREADS) {
            if (gr0 + i < jr) continue;
            const T v = cabs1(P[i * nb + j]);
            if (v > bv) {
                bv = v;
                bi = gr0 + i;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const T ov = __shfl_xor_sync(0xffffffffu, bv, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > bv || (ov == bv && oi >= 0 && (bi < 0 || oi < bi))) {
                bv = ov;
                bi = oi;
            }
        }
        if ((tid & 31) == 0) {
            red_v[tid >> 5] = bv;
            red_i[tid >> 5] = bi;
        }
        __syncthreads();
        if (tid == 0) {
            for (int w = 1; w < PANEL_THREADS / 32; ++w)
                if (red_v[w] > bv || (red_v[w] == bv && red_i[w] >= 0 && (bi < 0 || red_i[w] < bi))) {
                    bv = red_v[w];
                    bi = red_i[w];
                }
            s_piv = bi;
            s_pv = bv;
        }
        __syncthreads();
        const int mine = s_piv;
        if (mine >= 0)
            for (int c = tid; c < nb; c += PANEL_THREADS)
                a.pub_rows[((size_t)par * G + cta) * nb + c] = P[(mine - gr0) * nb + c];
        if (jr >= gr0 && jr < gr0 + nrows)
            for (int c = tid; c < nb; c += PANEL_THREADS) a.pub_diag[(size_t)par * nb + c] = P[(jr - gr0) * nb + c];
        __syncthreads();
        // candidate record, then one grid-wide barrier: each CTA adds one
        // arrival (release) and waits until all G arrivals of this column are in
        if (tid == 0) {
            PivotRec *rec = &a.recs[par * G + cta];
            rec->val = (double)s_pv;
            rec->idx = mine;
            __threadfence();
            asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(a.counter), "r"(1u) : "memory");
            const unsigned target = (unsigned)(j + 1) * (unsigned)G;
            unsigned it = 0;
            while (true) {
                unsigned v;
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(a.counter) : "memory");
                if (v >= target) break;
                if ((*(volatile int *)a.status & DEV_BARRIER_TIMEOUT) || ++it > a.spin_limit) {
                    atomicOr(a.status, (int)DEV_BARRIER_TIMEOUT);
                    break;
                }
            }
        }
        __syncthreads();
        // every CTA reads all G records at once and picks the same winner
        {
            T wv = T(-1);
            int wi = -1, wc = -1;
            if (tid < G) {
                const PivotRec *rec = &a.recs[par * G + tid];
                wi = __ldcg(&rec->idx);
                wv = wi >= 0 ? (T)__ldcg(&rec->val) : T(-1);
                wc = tid;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const T ov = __shfl_xor_sync(0xffffffffu, wv, o);
                const int oi = __shfl_xor_sync(0xffffffffu, wi, o);
                const int oc = __shfl_xor_sync(0xffffffffu, wc, o);
                if (oi >= 0 && (ov > wv || (ov == wv && (wi < 0 || oi < wi)))) {
                    wv = ov;
                    wi = oi;
                    wc = oc;
                }
            }
            if ((tid & 31) == 0) {
                red_v[tid >> 5] = wv;
                red_i[tid >> 5] = wi;
                red_c[tid >> 5] = wc;
            }
            __syncthreads();
            if (tid == 0) {
                for (int w = 1; w < PANEL_THREADS / 32; ++w)
                    if (red_i[w] >= 0 && (red_v[w] > wv || (red_v[w] == wv && (wi < 0 || red_i[w] < wi)))) {
                        wv = red_v[w];
                        wi = red_i[w];
                        wc = red_c[w];
                    }
                s_piv = wi < 0 ? jr : wi;
                s_pv = wv;
                red_i[0] = wc;
                if (wv <= T(0)) atomicOr(a.status, (int)DEV_ZERO_PIVOT);
                if (cta == 0) a.ipiv[jr] = s_piv;
            }
        }
        __syncthreads();
        const int p = s_piv, wc = red_i[0];
        for (int c = tid; c < nb; c += PANEL_THREADS) {
            prow[c] = wc >= 0 ? ldcg(&a.pub_rows[((size_t)par * G + wc) * nb + c]) : Cx<T>{T(0), T(0)};
            drow[c] = ldcg(&a.pub_diag[(size_t)par * nb + c]);
        }
        __syncthreads();
        if (p != jr) {
            if (jr >= gr0 && jr < gr0 + nrows)
                for (int c = tid; c < nb; c += PANEL_THREADS) P[(jr - gr0) * nb + c] = prow[c];
            if (p >= gr0 && p < gr0 + nrows)
                for (int c = tid; c < nb; c += PANEL_THREADS) P[(p - gr0) * nb + c] = drow[c];
        }
        __syncthreads();
        // eliminate below the pivot
        const Cx<T> pv = prow[j];
        const T den = pv.re * pv.re + pv.im * pv.im;
        const Cx<T> inv = den > T(0) ? Cx<T>{pv.re / den, -pv.im / den} : Cx<T>{T(0), T(0)};
        const int first = max(0, jr + 1 - gr0);
        for (int i = first + tid; i < nrows; i += PANEL_THREADS) lcol[i] = cmul(P[i * nb + j], inv);
        __syncthreads();
        const int w = nb - j - 1;
        if (w > 0) {
            for (int idx = tid; idx < (nrows - first) * w; idx += PANEL_THREADS) {
                const int i = first + idx / w, c = j + 1 + idx % w;
                const Cx<T> l = lcol[i], u = prow[c];
                Cx<T> &d = P[i * nb + c];
                d.re -= l.re * u.re - l.im * u.im;
                d.im -= l.re * u.im + l.im * u.re;
            }
        }
        for (int i = first + tid; i < nrows; i += PANEL_THREADS) P[i * nb + j] = lcol[i];
        __syncthreads();
    }
    for (int i = tid; i < nrows * nb; i += PANEL_THREADS) {
        const int r = i / nb, c = i % nb;
        a.A[(int64_t)(gr0 + r) * a.ld + a.k + c] = P[i];
    }
}

// Row interchanges ipiv[k .. k+nsw), nsw <= LS_MAX, on the columns [c_lo, c_hi)
// outside [x_lo, x_hi) and, with perm non-null, on the running permutation (the
// look-ahead swaps a sub-panel's rows inside its panel first and on the other
// columns once per panel), as one permutation of at most 2 nsw rows: every CTA
// derives the moves from ipiv, then loads every moved entry of its LS_COLS
// columns before it stores any, so no column walks a chain of dependent global
// loads.  With swap j exchanging
// positions k + j and p_j >= k + j, position k + j is final after swap j; its
// content then is what stood at p_j just before, and
//   X_j (the content of k + j just before swap j) = X_prevX[j], or the row k + j
//       itself when no earlier swap's far end was k + j;
//   V_j (the content of p_j just before swap j) = X_j when p_j = k + j, else
//       X_lastP[j] for the last earlier swap with the same far end, else p_j.
// Final contents: k + j <- V_j; a far end q >= k + nsw <- X_j of the last swap
// that names it.  X is a root search over prevX (pointer jumping).
constexpr int LS_MAX = 256;
template <typename T> __host__ __device__ constexpr int ls_cols() { return sizeof(T) == 4 ? 32 : 16; }
template <typename T> static size_t laswp_panel_smem(int nsw) {
    return sizeof(Cx<T>) * 2 * (size_t)nsw * ls_cols<T>();
}
template <typename T>
__global__ void __launch_bounds__(256) laswp_panel_kernel(Cx<T> *A, int64_t ld, int n, int k, int nsw, const int *ipiv,
                                                          int c_lo, int c_hi, int x_lo, int x_hi, int *perm) {
    constexpr int LC = ls_cols<T>();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Cx<T> *vals = reinterpret_cast<Cx<T> *>(smem_raw);  // [moves][LC]
    __shared__ int sp[LS_MAX], root[2][LS_MAX], xs[LS_MAX], msrc[2 * LS_MAX], mdst[2 * LS_MAX], pv[2 * LS_MAX];
    __shared__ int nmove;
    const int tid = threadIdx.x;
    const int jmax = min(min(nsw, n - k), LS_MAX);
    if (tid == 0) nmove = 0;
    for (int j = tid; j < jmax; j += 256) {
        const int p = ipiv[k + j];
        sp[j] = (p > k + j && p < n) ? p : k + j;  // out-of-range entries are no interchange
    }
    __syncthreads();
    int prev_x = -1, last_p = -1;
    bool has_next = false;
    const int j = tid;
    if (j < jmax) {
        const int pj = sp[j];
        for (int i = 0; i < jmax; ++i) {
            const int pi = sp[i];
            if (i < j) {
                if (pi == k + j) prev_x = i;
                if (pi == pj && pj != k + j) last_p = i;
            } else if (i > j && pi == pj) {
                has_next = true;
            }
        }
        root[0][j] = prev_x < 0 ? j : prev_x;
    }
    __syncthreads();
    int b = 0;
    for (int step = 1; step < LS_MAX; step *= 2) {  // log2(LS_MAX) rounds
        if (j < jmax) root[b ^ 1][j] = root[b][root[b][j]];
        b ^= 1;
        __syncthreads();
    }
    if (j < jmax) xs[j] = k + root[b][j];
    __syncthreads();
    if (j < jmax) {
        const int pj = sp[j], xj = xs[j];
        const int vj = pj == k + j ? xj : (last_p >= 0 ? xs[last_p] : pj);
        if (vj != k + j) {
            const int m = atomicAdd(&nmove, 1);
            msrc[m] = vj;
            mdst[m] = k + j;
        }
        if (pj >= k + jmax && !has_next) {
            const int m = atomicAdd(&nmove, 1);
            msrc[m] = xj;
            mdst[m] = pj;
        }
    }
    __syncthreads();
    const int nm = nmove;
    const int cbase = c_lo + (int)blockIdx.x * LC;
    for (int i = tid; i < nm * LC; i += 256) {
        const int c = cbase + i % LC;
        if (c < c_hi && (c < x_lo || c >= x_hi)) vals[i] = A[(int64_t)msrc[i / LC] * ld + c];
    }
    if (perm && blockIdx.x == 0)
        for (int m = tid; m < nm; m += 256) pv[m] = perm[msrc[m]];
    __syncthreads();
    for (int i = tid; i < nm * LC; i += 256) {
        const int c = cbase + i % LC;
        if (c < c_hi && (c < x_lo || c >= x_hi)) A[(int64_t)mdst[i / LC] * ld + c] = vals[i];
    }
    if (perm && blockIdx.x == 0)
        for (int m = tid; m < nm; m += 256) perm[mdst[m]] = pv[m];
}

__global__ void iota_kernel(int *perm, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) perm[i] = i;
}

// Inverse of a unit lower triangular kb x kb block (kb <= W <= 32), by one
// warp: lane c forward-substitutes column c of the inverse with four partial
// sums per row.  L holds the strictly lower part (row stride ldl), Y is W x
// (W + 1) scratch, D receives the W x W inverse row-major (identity past kb).
template <typename T>
__device__ __forceinline__ void warp_unit_lower_inverse(const Cx<T> *L, int ldl, int kb, int W, Cx<T> *Y, Cx<T> *D) {
    const int c = threadIdx.x & 31, ldy = W + 1;
    if (c < W) {
        for (int i = 0; i < W; ++i) {
            Cx<T> s0{T(i == c), T(0)}, s1{T(0), T(0)}, s2{T(0), T(0)}, s3{T(0), T(0)};
            if (i > c && i < kb) {
                int t = c;
                for (; t + 4 <= i; t += 4) {
                    s0 = cms(s0, L[i * ldl + t], Y[t * ldy + c]);
                    s1 = cms(s1, L[i * ldl + t + 1], Y[(t + 1) * ldy + c]);
                    s2 = cms(s2, L[i * ldl + t + 2], Y[(t + 2) * ldy + c]);
                    s3 = cms(s3, L[i * ldl + t + 3], Y[(t + 3) * ldy + c]);
                }
                for (; t < i; ++t) s0 = cms(s0, L[i * ldl + t], Y[t * ldy + c]);
            }
            Y[i * ldy + c] = Cx<T>{(s0.re + s1.re) + (s2.re + s3.re), (s0.im + s1.im) + (s2.im + s3.im)};
        }
        for (int i = 0; i < W; ++i) D[(size_t)i * W + c] = Y[i * ldy + c];
    }
}

// The same for the diagonal block A[k:k+kb, k:k+kb] (kb = min(W, n - k)) of
// a sub-panel factored by the grid-wide panel kernel.
template <typename T>
__global__ void __launch_bounds__(32) diag_block_inverse_kernel(const Cx<T> *A, int64_t ld, int n, int k, int W, Cx<T> *D) {
    __shared__ Cx<T> L[32 * 33];
    __shared__ Cx<T> Y[32 * 33];
    const int kb = min(W, n - k);
    batched_copy<32, 32, Cx<T>>(
        kb * kb, [&](int i) { return A[(int64_t)(k + i / kb) * ld + k + i % kb]; },
        [&](int i, Cx<T> v) { L[(i / kb) * 33 + i % kb] = v; });
    __syncwarp();
    warp_unit_lower_inverse(L, 33, kb, W, Y, D);
}

// Blocked U12 = L11^-1 A12 for L11 = A[k:k+kb, k:k+kb] (kb = S W) with the
// inverses D_s of its W x W diagonal blocks:  X_s = D_s (A_s - sum_{t<s}
// L_st X_t), s = 0..S-1.  32 columns per CTA, 256 threads, each thread W/8
// complex outputs of a W x 32 block per product; one barrier per block step
// instead of one per row.
constexpr int TB_COLS = 32;
// With bhi non-null (FP32, the tensor-core path) the solved block is also
// written in the trailing update's B-operand layout (the staging of
// tc_gemm.cu: rows 2j and 2j + 1 of B_s hold (Ur, -Ui) 2^s and (Ui, Ur) 2^s at
// K = 2kk for column j = c - j0 and row kk of the block, s from the column's
// largest |re| or |im|, as FP16 high parts and, when split == 3, FP16
// remainders; bscale[j] = 2^-(s + L_SHIFT)), so no separate staging pass
// rereads U12.  stage_u_block does it for a block of COLS columns in shared
// memory (X[row * COLS + column]); all 256 threads of the CTA call it.
template <int COLS>
__device__ void stage_u_block(const Cx<float> *X, int kb, int nc, int c0, int j0, __half *bhi, __half *blo,
                              float *bscale, int split) {
    __shared__ unsigned cmax[COLS];  // largest |re| or |im| of each column, as ordered bits
    const int tid = threadIdx.x;
    if (tid < COLS) cmax[tid] = 0u;
    __syncthreads();
    {
        const int c = tid % COLS;
        float mx = 0.f;
        for (int r = tid / COLS; r < kb; r += 256 / COLS) {
            const Cx<float> u = X[r * COLS + c];
            mx = fmaxf(mx, fmaxf(fabsf(u.re), fabsf(u.im)));
        }
        atomicMax(&cmax[c], __float_as_uint(mx));
    }
    __syncthreads();
    if (tid < nc) bscale[c0 + tid - j0] = pow2f(-stage_exp(__uint_as_float(cmax[tid])) - L_SHIFT);
    // consecutive threads: consecutive K (rows kk of the block) of one B_s row
    for (int i = tid; i < 2 * COLS * kb; i += 256) {
        const int row = i / kb, kk = i % kb, c = row >> 1;
        if (c >= nc) continue;
        const float sc = pow2f(stage_exp(__uint_as_float(cmax[c])));
        const Cx<float> u = X[kk * COLS + c];
        const float vx = ((row & 1) ? u.im : u.re) * sc, vy = ((row & 1) ? u.re : -u.im) * sc;
        const int64_t at = (int64_t)(2 * (c0 + c - j0) + (row & 1)) * 2 * kb + 2 * kk;
        __half hx, hy, lx, ly;
        split_f16(vx, hx, lx);
        split_f16(vy, hy, ly);
        *reinterpret_cast<__half2 *>(bhi + at) = __halves2half2(hx, hy);
        if (split == 3) *reinterpret_cast<__half2 *>(blo + at) = __halves2half2(lx, ly);
    }
}
template <typename T, int W>
__global__ void __launch_bounds__(256) trsm_blocked_kernel(Cx<T> *A, int64_t ld, int k, int S, const Cx<T> *D,
                                                            int c_begin, int c_end, __half *bhi = nullptr,
                                                            __half *blo = nullptr, float *bscale = nullptr,
                                                            int j0 = 0, int split = 3) {
    constexpr int OPT = W * TB_COLS / 256;  // outputs per thread: 4 (W = 32) or 2 (W = 16)
    constexpr int CG = TB_COLS / OPT;       // column groups
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int kb = S * W;
    Cx<T> *X = reinterpret_cast<Cx<T> *>(smem_raw);  // kb x TB_COLS
    Cx<T> *Dt = X + (size_t)kb * TB_COLS;             // W x (W + 1)
    Cx<T> *Lt = Dt + W * (W + 1);                     // W x (r0 + 1), r0 <= kb - W
    const int tid = threadIdx.x, r = tid / CG, cg = tid % CG;
    const int c0 = c_begin + blockIdx.x * TB_COLS;
    const int nc = min(TB_COLS, c_end - c0);
    batched_copy<256, 8, Cx<T>>(
        kb * TB_COLS,
        [&](int i) {
            const int c = i % TB_COLS;
            return c < nc ? A[(int64_t)(k + i / TB_COLS) * ld + c0 + c] : Cx<T>{T(0), T(0)};
        },
        [&](int i, Cx<T> v) { X[i] = v; });
    for (int s = 0; s < S; ++s) {
        const int r0 = s * W;
        batched_copy<256, 4, Cx<T>>(
            W * W, [&](int i) { return D[(size_t)s * W * W + i]; },
            [&](int i, Cx<T> v) { Dt[(i / W) * (W + 1) + i % W] = v; });
        if (s > 0)
            batched_copy<256, 8, Cx<T>>(
                W * r0, [&](int i) { return A[(int64_t)(k + r0 + i / r0) * ld + k + i % r0]; },
                [&](int i, Cx<T> v) { Lt[(i / r0) * (r0 + 1) + i % r0] = v; });
        __syncthreads();
        Cx<T> acc[OPT];
#pragma unroll
        for (int o = 0; o < OPT; ++o) acc[o] = X[(r0 + r) * TB_COLS + cg * OPT + o];
        for (int t = 0; t < r0; ++t) {  // A_s - L_s,<s X_<s
            const Cx<T> l = Lt[r * (r0 + 1) + t];
#pragma unroll
            for (int o = 0; o < OPT; ++o) {
                const Cx<T> x = X[t * TB_COLS + cg * OPT + o];
                acc[o].re -= l.re * x.re - l.im * x.im;
                acc[o].im -= l.re * x.im + l.im * x.re;
            }
        }
        __syncthreads();  // every thread has read block s of X
#pragma unroll
        for (int o = 0; o < OPT; ++o) X[(r0 + r) * TB_COLS + cg * OPT + o] = acc[o];
        __syncthreads();
        Cx<T> y[OPT];
#pragma unroll
        for (int o = 0; o < OPT; ++o) y[o] = Cx<T>{T(0), T(0)};
        for (int t = 0; t <= r; ++t) {  // D_s is lower triangular
            const Cx<T> d = Dt[r * (W + 1) + t];
#pragma unroll
            for (int o = 0; o < OPT; ++o) {
                const Cx<T> x = X[(r0 + t) * TB_COLS + cg * OPT + o];
                y[o].re += d.re * x.re - d.im * x.im;
                y[o].im += d.re * x.im + d.im * x.re;
            }
        }
        __syncthreads();
#pragma unroll
        for (int o = 0; o < OPT; ++o) X[(r0 + r) * TB_COLS + cg * OPT + o] = y[o];
        // the next block step's loads of Dt / Lt follow the next barrier
        __syncthreads();
    }
    for (int i = tid; i < kb * TB_COLS; i += 256) {
        const int rr = i / TB_COLS, c = i % TB_COLS;
        if (c < nc) A[(int64_t)(k + rr) * ld + c0 + c] = X[rr * TB_COLS + c];
    }
    if constexpr (sizeof(T) == 4) {
        if (bhi) stage_u_block<TB_COLS>(X, kb, nc, c0, j0, bhi, blo, bscale, split);
    }
}

// one complex element, global -> shared, through the asynchronous copy unit
template <typename T> __device__ __forceinline__ void cp_async_cx(Cx<T> *smem, const Cx<T> *gmem) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem);
    if constexpr (sizeof(Cx<T>) == 8)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(gmem) : "memory");
    else
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gmem) : "memory");
}

// The same solve for the launches on the factorisation's critical path (the
// next panel's columns, the rest of a panel after each sub-panel).  256 / W
// columns per CTA, one entry of a W-row block per thread, so that the columns
// spread over 4 times more CTAs; the right-hand sides, every diagonal-block
// inverse and every off-diagonal L block of the triangle are in flight
// together before the first block step, so the S dependent steps wait on no
// global load.  Two partial sums per product.  The same optional B-operand
// staging as trsm_blocked_kernel.
template <int W> __host__ __device__ constexpr int narrow_cols() { return 256 / W; }
template <typename T, int W, int NC = narrow_cols<W>()> static size_t trsm_narrow_smem(int S) {
    return sizeof(Cx<T>) * ((size_t)S * W * NC + (size_t)S * W * (W + 1) +
                            (size_t)W * ((size_t)W * S * (S - 1) / 2 + (S - 1)) + (size_t)W * NC);
}
// NC columns per CTA (a multiple of 256 / W): each thread holds OPT = NC W / 256
// entries of a W-row block, row tid / (256 / W), columns tid % (256 / W) + (256 / W) o.
template <typename T, int W, int NC = narrow_cols<W>()>
__global__ void __launch_bounds__(256) trsm_narrow_kernel(Cx<T> *A, int64_t ld, int k, int S, const Cx<T> *D,
                                                          int c_begin, int c_end, __half *bhi, __half *blo,
                                                          float *bscale, int j0, int split) {
    constexpr int CG = narrow_cols<W>(), OPT = NC / CG;
    static_assert(OPT >= 1 && NC % CG == 0, "NC: a multiple of 256 / W");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int kb = S * W;
    Cx<T> *X = reinterpret_cast<Cx<T> *>(smem_raw);  // kb x NC
    Cx<T> *Ds = X + (size_t)kb * NC;                  // S blocks of W x (W + 1)
    Cx<T> *Ls = Ds + (size_t)S * W * (W + 1);         // block row s >= 1: W x (s W + 1)
    Cx<T> *Z = Ls + (size_t)W * ((size_t)W * S * (S - 1) / 2 + (S - 1));  // W x NC
    const int tid = threadIdx.x, r = tid / CG, cg = tid % CG;
    const int c0 = c_begin + blockIdx.x * NC;
    const int nc = min(NC, c_end - c0);
    for (int i = tid; i < kb * NC; i += 256) {
        const int c = i % NC;
        if (c < nc)
            cp_async_cx(&X[i], &A[(int64_t)(k + i / NC) * ld + c0 + c]);
        else
            X[i] = Cx<T>{T(0), T(0)};
    }
    for (int i = tid; i < S * W * W; i += 256) {
        const int s = i / (W * W), e = i % (W * W);
        cp_async_cx(&Ds[(size_t)s * W * (W + 1) + (e / W) * (W + 1) + e % W], &D[i]);
    }
    for (int s = 1; s < S; ++s) {  // L rows [s W, s W + W) x columns [0, s W)
        const int r0 = s * W;
        Cx<T> *Lb = Ls + (size_t)W * ((size_t)W * s * (s - 1) / 2 + (s - 1));
        for (int i = tid; i < W * r0; i += 256)
            cp_async_cx(&Lb[(i / r0) * (r0 + 1) + i % r0], &A[(int64_t)(k + r0 + i / r0) * ld + k + i % r0]);
    }
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    for (int s = 0; s < S; ++s) {
        const int r0 = s * W;
        Cx<T> a0[OPT], a1[OPT];
#pragma unroll
        for (int o = 0; o < OPT; ++o) {
            a0[o] = X[(r0 + r) * NC + cg + CG * o];
            a1[o] = Cx<T>{T(0), T(0)};
        }
        if (s > 0) {  // A_s - L_s,<s X_<s
            const Cx<T> *Lr = Ls + (size_t)W * ((size_t)W * s * (s - 1) / 2 + (s - 1)) + (size_t)r * (r0 + 1);
            for (int t = 0; t < r0; t += 2) {  // r0 is a multiple of W, so even
                const Cx<T> l0 = Lr[t], l1 = Lr[t + 1];
#pragma unroll
                for (int o = 0; o < OPT; ++o) {
                    a0[o] = cms(a0[o], l0, X[t * NC + cg + CG * o]);
                    a1[o] = cms(a1[o], l1, X[(t + 1) * NC + cg + CG * o]);
                }
            }
        }
#pragma unroll
        for (int o = 0; o < OPT; ++o) Z[r * NC + cg + CG * o] = Cx<T>{a0[o].re + a1[o].re, a0[o].im + a1[o].im};
        __syncthreads();
        const Cx<T> *Dr = Ds + (size_t)s * W * (W + 1) + (size_t)r * (W + 1);
        Cx<T> y0[OPT], y1[OPT];
#pragma unroll
        for (int o = 0; o < OPT; ++o) y0[o] = y1[o] = Cx<T>{T(0), T(0)};
        int t = 0;
        for (; t + 1 <= r; t += 2) {  // D_s is lower triangular
            const Cx<T> d0 = Dr[t], d1 = Dr[t + 1];
#pragma unroll
            for (int o = 0; o < OPT; ++o) {
                const Cx<T> z0 = Z[t * NC + cg + CG * o], z1 = Z[(t + 1) * NC + cg + CG * o];
                y0[o] = Cx<T>{y0[o].re + (d0.re * z0.re - d0.im * z0.im), y0[o].im + (d0.re * z0.im + d0.im * z0.re)};
                y1[o] = Cx<T>{y1[o].re + (d1.re * z1.re - d1.im * z1.im), y1[o].im + (d1.re * z1.im + d1.im * z1.re)};
            }
        }
        if (t == r) {
            const Cx<T> d0 = Dr[t];
#pragma unroll
            for (int o = 0; o < OPT; ++o) {
                const Cx<T> z0 = Z[t * NC + cg + CG * o];
                y0[o] = Cx<T>{y0[o].re + (d0.re * z0.re - d0.im * z0.im), y0[o].im + (d0.re * z0.im + d0.im * z0.re)};
            }
        }
#pragma unroll
        for (int o = 0; o < OPT; ++o)
            X[(r0 + r) * NC + cg + CG * o] = Cx<T>{y0[o].re + y1[o].re, y0[o].im + y1[o].im};
        __syncthreads();  // block s of X is complete; Z is free again
    }
    for (int i = tid; i < kb * NC; i += 256) {
        const int c = i % NC;
        if (c < nc) A[(int64_t)(k + i / NC) * ld + c0 + c] = X[i];
    }
    if constexpr (sizeof(T) == 4) {
        if (bhi) stage_u_block<NC>(X, kb, nc, c0, j0, bhi, blo, bscale, split);
    }
}

// ---------------------------------------------------------------------------
// FP64 tensor-core (DMMA) complex GEMM for the FP64 form's updates:
// C[r0.., c0..] -= L U, 8 x 8 complex blocks by mma.sync.m8n8k4.f64 (4 real
// products per complex block: re += Lr Ur - Li Ui, im += Lr Ui + Li Ur, the
// sign on the L fragment).  Fragments (PTX ISA, m8n8k4 .f64): A a0 at
// (lane / 4, lane % 4); B b0 at (lane % 4, lane / 4); C c0, c1 at (lane / 4,
// 2 (lane % 4) + 0, 1).
//
// L U is summed apart and subtracted from C once, so that an entry takes one
// rounding at its own magnitude per panel instead of two per index: with C as
// the accumulators' start the solutions' error at N = 998 / 2,616 / 10,242 was
// 2.0 / 2.8 / 5.0e-15, so it is 4.4 / 4.6 / 7.9e-16 (the three kernels that
// eliminate, together; LU at N = 10,242 104.5 -> 104.7 ms, N = 2,616 7.75 ->
// 7.90).  K goes in chunks of 8 through DU_ST cp.async stages, one barrier per
// chunk.  Complex entries stay interleaved (a fragment's real and imaginary
// part are one 16-byte load); row strides of 4 mod 8 (L) and 2 mod 8 (U)
// entries keep a quarter-warp's loads on distinct banks.
//
// Tiles of 64 x 32, four warps of 32 x 16 complex (64 registers of sums), four
// CTAs per SM: what holds the pipe back is the start and the end of each tile
// (the first chunk, C's latency, the stores), and with 16 warps in four places
// the others' products cover them.  m x m updates of K = 128 at m = 10,114 /
// 5,000 / 2,500, TFLOP/s of the 37 measured with mma.sync alone: two CTAs of
// 64 x 64 (32 x 32 per warp, 4 stages) 29.7 / 28.1 / 27.0 (two warps per
// scheduler, the pipe 80 % busy); 64 x 48, 3 CTAs, 3 stages 31.2 / 29.1; these
// with 3 CTAs and 4 stages 30.3 / 27.5, with 4 and 2 32.8 / 31.8 / 29.1; 32 x 32,
// 8 CTAs 32.8 / 32.2 at twice the reads of L; 5 CTAs no more.
// C goes through L2 as evict-first (streaming loads and stores): L, U and the
// next panel's columns stay (N = 10,242: LU 106.0 -> 104.5 ms).
// ---------------------------------------------------------------------------
constexpr int DU_K = 8, DU_ST = 2, DU_M = 64, DU_N = 32, DU_THREADS = 128;

__device__ __forceinline__ void dmma884(double (&c)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(c[0]), "+d"(c[1])
        : "d"(a), "d"(b));
}
// 16 bytes, global -> shared, asynchronously; zeros when `in` is false
__device__ __forceinline__ void cp_async16_zfill(double2 *smem, const double2 *gmem, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(smem)),
                 "l"(gmem), "r"(in ? 16 : 0)
                 : "memory");
}

constexpr int DU_LDA = DU_K + 4, DU_LDB = DU_N + 2, DU_STAGE = DU_M * DU_LDA + DU_K * DU_LDB;  // complex entries
constexpr size_t DU_SMEM = sizeof(double2) * DU_ST * DU_STAGE;
__global__ void __launch_bounds__(DU_THREADS, 4)
    dmma_update_kernel(Cx<double> *A_, int64_t ld, int n, int k, int kk, int row0, int col0, int col_end) {
    constexpr int WM = 32, WN = 16, MI = WM / 8, NJ = WN / 8;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double2 *ring = reinterpret_cast<double2 *>(smem_raw);
    double2 *A = reinterpret_cast<double2 *>(A_);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int r0 = row0 + blockIdx.y * DU_M, c0 = col0 + blockIdx.x * DU_N;
    const int wr = (warp / (DU_N / WN)) * WM, wc = (warp % (DU_N / WN)) * WN;
    const int nk = (kk + DU_K - 1) / DU_K;
    auto load = [&](int kt) {  // chunk kt of L (DU_M x DU_K) and U (DU_K x DU_N)
        if (kt < nk) {
            double2 *sl = ring + (kt % DU_ST) * DU_STAGE, *su = sl + DU_M * DU_LDA;
            const int kc = kt * DU_K;
            static_assert(DU_M * DU_K % DU_THREADS == 0 && DU_N * DU_K % DU_THREADS == 0, "whole rounds of copies");
#pragma unroll
            for (int u = 0; u < DU_M * DU_K / DU_THREADS; ++u) {
                const int i = (tid + u * DU_THREADS) / DU_K, q = tid % DU_K;
                const bool in = r0 + i < n && kc + q < kk;
                cp_async16_zfill(&sl[i * DU_LDA + q], in ? &A[(int64_t)(r0 + i) * ld + k + kc + q] : A, in);
            }
#pragma unroll
            for (int u = 0; u < DU_N * DU_K / DU_THREADS; ++u) {
                const int q = (tid + u * DU_THREADS) / DU_N, j = (tid + u * DU_THREADS) % DU_N;
                const bool in = c0 + j < col_end && kc + q < kk;
                cp_async16_zfill(&su[q * DU_LDB + j], in ? &A[(int64_t)(k + kc + q) * ld + c0 + j] : A, in);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int s = 0; s < DU_ST - 1; ++s) load(s);
    double cr[MI][NJ][2] = {}, ci[MI][NJ][2] = {};  // [row block][column block][fragment]: L U
    for (int kt = 0; kt < nk; ++kt) {
        asm volatile("cp.async.wait_group %0;" ::"n"(DU_ST - 2) : "memory");
        __syncthreads();  // chunk kt is in; every warp is done with chunk kt - 1, whose place the next load takes
        load(kt + DU_ST - 1);
        const double2 *sl = ring + (kt % DU_ST) * DU_STAGE, *su = sl + DU_M * DU_LDA;
#pragma unroll
        for (int k4 = 0; k4 < DU_K; k4 += 4) {
            double2 a[MI], b[NJ];
#pragma unroll
            for (int i = 0; i < MI; ++i) a[i] = sl[(wr + 8 * i + g) * DU_LDA + k4 + t];
#pragma unroll
            for (int j = 0; j < NJ; ++j) b[j] = su[(k4 + t) * DU_LDB + wc + 8 * j + g];
#pragma unroll
            for (int i = 0; i < MI; ++i) {
                const double ni = -a[i].y;
                // (2 NJ products between the two that add to one block)
#pragma unroll
                for (int j = 0; j < NJ; ++j) {
                    dmma884(cr[i][j], a[i].x, b[j].x);
                    dmma884(ci[i][j], a[i].x, b[j].y);
                }
#pragma unroll
                for (int j = 0; j < NJ; ++j) {
                    dmma884(cr[i][j], ni, b[j].y);
                    dmma884(ci[i][j], a[i].y, b[j].x);
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < MI; ++i) {
        double2 v[NJ][2];
#pragma unroll
        for (int j = 0; j < NJ; ++j)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int r = r0 + wr + 8 * i + g, c = c0 + wc + 8 * j + 2 * t + e;
                v[j][e] = (r < n && c < col_end) ? __ldcs(&A[(int64_t)r * ld + c]) : make_double2(0.0, 0.0);
            }
#pragma unroll
        for (int j = 0; j < NJ; ++j)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int r = r0 + wr + 8 * i + g, c = c0 + wc + 8 * j + 2 * t + e;
                if (r < n && c < col_end)
                    __stcs(&A[(int64_t)r * ld + c], make_double2(v[j][e].x - cr[i][j][e], v[j][e].y - ci[i][j][e]));
            }
    }
}

// the FP64 form's trailing / in-panel update C -= L U, L = A[row0.., k..k+kk),
// U = A[k..k+kk, col0..col_end)
static void launch_update(cudaStream_t st, Cx<double> *A, int64_t ld, int n, int k, int kk, int row0, int col0,
                          int col_end) {
    const int rows = n - row0, cols = col_end - col0;
    if (rows <= 0 || cols <= 0) return;
    dmma_update_kernel<<<dim3((cols + DU_N - 1) / DU_N, (rows + DU_M - 1) / DU_M), DU_THREADS, DU_SMEM, st>>>(
        A, ld, n, k, kk, row0, col0, col_end);
    BB_CUDA(cudaGetLastError());
}
static void update_setup() {
    BB_CUDA(cudaFuncSetAttribute(dmma_update_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DU_SMEM));
}

// ---------------------------------------------------------------------------
// FP64 U12 = L11^-1 A12 on the FP64 tensor cores: one warp solves 8 columns on
// its own (no block barrier), 16 rows at a time: A12 minus L_s,<s X_<s (summed
// apart, as in the update) with L's fragments read through L1 and X from the
// warp's shared memory, then times the diagonal block's inverse D_s (its upper
// half is not read).  The next block's rows and this block's D are on their way
// meanwhile.
// X rows of 10 entries keep a quarter-warp's fragment loads on distinct banks.
// Bound: the warp's own chain, 1,152 products for 128 rows (16 cycles each on a
// sub-core, 9.5 us), two warps per sub-core at 9,000 columns.
// 128 rows x 9,120 columns: 16 columns per CTA with FP64 FMA from shared memory
// and its barriers took 168 us, this 30.  The next panel's 128 columns, on the
// critical path, stay with trsm_narrow_kernel, whose chain is shorter (24 us
// against 31 here) at the price of whole SMs.
// ---------------------------------------------------------------------------
constexpr int TS_COLS = 8, TS_LD = 10;
static size_t trsm_mma_smem(int nb, int warps) { return sizeof(double2) * (size_t)nb * TS_LD * warps; }
__global__ void __launch_bounds__(128, 2) trsm_mma_kernel(Cx<double> *A_, int64_t ld, int k, int S, const Cx<double> *D_,
                                                         int c_begin, int c_end) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double2 *A = reinterpret_cast<double2 *>(A_);
    const double2 *D = reinterpret_cast<const double2 *>(D_);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int c0 = c_begin + (blockIdx.x * (blockDim.x >> 5) + warp) * TS_COLS;
    if (c0 >= c_end) return;
    double2 *X = reinterpret_cast<double2 *>(smem_raw) + (size_t)warp * S * 16 * TS_LD;
    double2 v[2][2];
    auto fetch = [&](int s) {
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int c = c0 + 2 * t + e;
                v[i][e] = c < c_end ? A[(int64_t)(k + 16 * s + 8 * i + g) * ld + c] : make_double2(0.0, 0.0);
            }
    };
    fetch(0);
    for (int s = 0; s < S; ++s) {
        double2 b0[2][2];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int e = 0; e < 2; ++e) b0[i][e] = v[i][e];
        double cr[2][2] = {}, ci[2][2] = {};  // L_s,<s X_<s
        if (s + 1 < S) fetch(s + 1);
        double2 d[2][4];  // D_s: rows 8 i + g, columns 4 j + t, zero above the diagonal
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 2 + 2 * i; ++j)
                d[i][j] = 4 * j + t <= 8 * i + g ? __ldg(&D[(size_t)s * 256 + (8 * i + g) * 16 + 4 * j + t])
                                                 : make_double2(0.0, 0.0);
        const double2 *L0 = A + (int64_t)(k + 16 * s + g) * ld + k + t, *L1 = L0 + 8 * ld;
#pragma unroll 4
        for (int q = 0; q < 16 * s; q += 4) {
            const double2 l0 = __ldg(L0 + q), l1 = __ldg(L1 + q), b = X[(q + t) * TS_LD + g];
            dmma884(cr[0], l0.x, b.x);
            dmma884(ci[0], l0.x, b.y);
            dmma884(cr[1], l1.x, b.x);
            dmma884(ci[1], l1.x, b.y);
            dmma884(cr[0], -l0.y, b.y);
            dmma884(ci[0], l0.y, b.x);
            dmma884(cr[1], -l1.y, b.y);
            dmma884(ci[1], l1.y, b.x);
        }
        double2 *Xs = X + 16 * s * TS_LD;
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int e = 0; e < 2; ++e)
                Xs[(8 * i + g) * TS_LD + 2 * t + e] = make_double2(b0[i][e].x - cr[i][e], b0[i][e].y - ci[i][e]);
        __syncwarp();
        double yr[2][2] = {}, yi[2][2] = {};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const double2 b = Xs[(4 * j + t) * TS_LD + g];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                if (j >= 2 + 2 * i) continue;
                dmma884(yr[i], d[i][j].x, b.x);
                dmma884(yi[i], d[i][j].x, b.y);
                dmma884(yr[i], -d[i][j].y, b.y);
                dmma884(yi[i], d[i][j].y, b.x);
            }
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const double2 y = make_double2(yr[i][e], yi[i][e]);
                Xs[(8 * i + g) * TS_LD + 2 * t + e] = y;
                const int c = c0 + 2 * t + e;
                if (c < c_end) A[(int64_t)(k + 16 * s + 8 * i + g) * ld + c] = y;
            }
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// FP32 update inside a panel, after each of its sub-panels: C[row0.., col0 ..
// col_end) -= L U with L = A[r, k:k+kk], U = A[k:k+kk, c], kk <= 32.  The
// update is 32, 64 or 96 columns wide, so the tiles are 128 x 32 complex: the
// whole K is staged at once by the asynchronous copy unit while each thread
// prefetches its 4 x 4 outputs, then one barrier and kk rank-1 steps from
// shared memory.  (Square 64 x 64 tiles left half of each tile idle on the
// 32-column updates and staged K in two synchronised chunks.)  C never overlaps L or U: rows >= row0 > k + kk, columns >= col0.
// ---------------------------------------------------------------------------
constexpr int PU_ROWS = 128, PU_COLS = 32, PU_K = 32;
__global__ void __launch_bounds__(256, 2) panel_update_kernel(Cx<float> *A, int64_t ld, int n, int k, int kk, int row0,
                                                             int col0, int col_end) {
    __shared__ __align__(16) Cx<float> sL[PU_ROWS][PU_K + 1];
    __shared__ __align__(16) Cx<float> sU[PU_K][PU_COLS];
    const int tid = threadIdx.x, tx = tid % 8, ty = tid / 8;  // outputs: rows ty + 32 i, columns tx + 8 j
    const int r0 = row0 + blockIdx.y * PU_ROWS, c0 = col0 + blockIdx.x * PU_COLS;
    for (int i = tid; i < PU_ROWS * PU_K; i += 256) {
        const int rr = i / PU_K, q = i % PU_K, r = r0 + rr;
        if (r < n && q < kk)
            cp_async_cx(&sL[rr][q], &A[(int64_t)r * ld + k + q]);
        else
            sL[rr][q] = Cx<float>{0.f, 0.f};
    }
    for (int i = tid; i < PU_K * PU_COLS; i += 256) {
        const int q = i / PU_COLS, cc = i % PU_COLS, c = c0 + cc;
        if (c < col_end && q < kk)
            cp_async_cx(&sU[q][cc], &A[(int64_t)(k + q) * ld + c]);
        else
            sU[q][cc] = Cx<float>{0.f, 0.f};
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    Cx<float> cur[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int r = r0 + ty + 32 * i, c = c0 + tx + 8 * j;
            cur[i][j] = (r < n && c < col_end) ? A[(int64_t)r * ld + c] : Cx<float>{0.f, 0.f};
        }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    float acc[4][4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.f;
#pragma unroll 4
    for (int q = 0; q < PU_K; ++q) {
        Cx<float> a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = sL[ty + 32 * i][q];
#pragma unroll
        for (int j = 0; j < 4; ++j) b[j] = sU[q][tx + 8 * j];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                acc[i][j][0] += a[i].re * b[j].re - a[i].im * b[j].im;
                acc[i][j][1] += a[i].re * b[j].im + a[i].im * b[j].re;
            }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int r = r0 + ty + 32 * i, c = c0 + tx + 8 * j;
            if (r < n && c < col_end)
                A[(int64_t)r * ld + c] = Cx<float>{cur[i][j].re - acc[i][j][0], cur[i][j].im - acc[i][j][1]};
        }
}

// Launches the cluster kernel for a sub-panel of W columns; false when the rows
// do not fit the cluster's shared memory or the cluster cannot be scheduled.
template <typename T>
static bool cluster_panel(beat_b200_ctx *c, Cx<T> *A, int64_t ld, int n, int k, int *ipiv, Cx<T> *dinv, int xc0, int xc1) {
    using S = CpShape<T>;
    const int m = n - k;
    const int C = m <= CP_ONE_CTA ? 1 : CP_CTAS;
    const int rpc = (m + C - 1) / C;
    // one row per thread on four warps (one per scheduler), then two, then two
    // or three on eight warps
    const int threads = rpc <= CP_THREADS ? CP_THREADS / 2 : CP_THREADS;
    const int rpt = (rpc + threads - 1) / threads;
    constexpr size_t cap = 226 * 1024;
    if (n >= (1 << 30) || rpt > 3) return false;
    const size_t smem = S::smem(rpc, C);
    if (smem > cap) return false;
    const void *kernel = rpt == 1   ? cluster_panel_entry<T, 1>()
                         : rpt == 2 ? cluster_panel_entry<T, 2>()
                                    : cluster_panel_entry<T, 3>();
    static std::atomic<bool> attr_done[3];  // sweep lanes call this from several threads
    if (!attr_done[rpt - 1]) {
        BB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        BB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap));
        attr_done[rpt - 1] = true;
    }
    ClusterPanelArgs<T> a;
    a.A = A;
    a.ld = ld;
    a.n = n;
    a.k = k;
    a.rpc = rpc;
    a.ipiv = ipiv;
    a.status = c->status.as<int>();
    a.dinv = dinv;
    a.xc0 = xc0;
    a.xc1 = xc1;
    a.timeout_ns = 100000000ull;  // 0.1 s per column wait
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(CP_CTAS);
    cfg.blockDim = dim3(CP_THREADS);
    cfg.dynamicSmemBytes = cap;  // the largest request any sub-panel makes
    cfg.stream = c->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CP_CTAS;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (!c->cluster_checked) {  // (any variant: all may use every register of an SM and the same shared memory)
        int nclusters = 0;
        cudaError_t e = cudaOccupancyMaxActiveClusters(&nclusters, kernel, &cfg);
        c->cluster_ok = (e == cudaSuccess && nclusters >= 1);
        cudaGetLastError();
        c->cluster_checked = true;
    }
    if (!c->cluster_ok) return false;
    cfg.gridDim = dim3(C);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    attr[0].val.clusterDim.x = C;
    void *args[] = {&a};
    BB_CUDA(cudaLaunchKernelExC(&cfg, kernel, args));
    return true;
}

// FP32 form trailing update on the tensor cores (tc_gemm.cu)
void tc_stage_l(beat_b200_ctx *c, int k, int nb, int split_terms, cudaStream_t st);
void tc_stage_u_buffers(beat_b200_ctx *c, int k, int nb, __half **bhi, __half **blo, float **bscale);
void tc_update_cols(beat_b200_ctx *c, int k, int nb, int split_terms, int col_lo, int col_hi, cudaStream_t st,
                    int max_ctas);

// ---------------------------------------------------------------------------
// host driver
// ---------------------------------------------------------------------------
template <typename T> static void lu_factor_t(beat_b200_ctx *c, int nb, int split_terms) {
    Workspace &w = c->ws;
    const int n = c->V;
    const int64_t ld = w.ld;
    Cx<T> *A = w.A.as<Cx<T>>();
    int G = c->sm_count;
    // shared memory per CTA for the panel: rows x nb + 2 nb + rows
    const size_t smem_cap = 200 * 1024;
    int rpc = (n + G - 1) / G;
    size_t smem = sizeof(Cx<T>) * ((size_t)rpc * nb + 2 * nb + rpc);
    BB_REQUIRE(smem <= smem_cap, BEAT_B200_INVALID_ARG,
               "LU: system of order " + std::to_string(n) + " exceeds the shared-memory panel limit");
    // scratch: [2][G] pivot records, [2][G][nb] candidate rows, [2][nb] diagonal rows
    // and the inverses of the sub-panels' W x W diagonal blocks
    constexpr int WF = 256 / sizeof(Cx<T>), W = WF;  // a sub-panel's columns: 256-byte rows
    BB_REQUIRE(nb % 32 == 0 && nb <= LS_MAX, BEAT_B200_INVALID_ARG, "LU: panels of 32, 64, 128 or 256 columns");
    const size_t rec_bytes = sizeof(PivotRec) * 2 * (size_t)G;
    const size_t scratch = rec_bytes + sizeof(Cx<T>) * (2 * (size_t)G * nb + 2 * nb);
    const size_t dinv_off = (scratch + 255) / 256 * 256;
    const size_t dinv_bytes = sizeof(Cx<T>) * (size_t)W * W * ((n + W - 1) / W);
    w.panel_scratch.alloc(dinv_off + dinv_bytes);
    PivotRec *recs = w.panel_scratch.as<PivotRec>();
    Cx<T> *pub_rows = reinterpret_cast<Cx<T> *>(recs + 2 * G);
    Cx<T> *pub_diag = pub_rows + 2 * (size_t)G * nb;
    Cx<T> *dinv = reinterpret_cast<Cx<T> *>(w.panel_scratch.as<unsigned char>() + dinv_off);
    const size_t tb_smem = sizeof(Cx<T>) * ((size_t)nb * TB_COLS + (size_t)W * (W + 1) + (size_t)W * (nb - W + 1));
    BB_CUDA(cudaFuncSetAttribute(trsm_blocked_kernel<T, WF>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)tb_smem));
    // the critical-path solves take the narrow kernel when its whole triangle fits
    constexpr int NC = narrow_cols<WF>();
    const bool narrow = trsm_narrow_smem<T, WF>(nb / W) <= 227 * 1024;
    if (narrow)
        BB_CUDA(cudaFuncSetAttribute(trsm_narrow_kernel<T, WF>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)trsm_narrow_smem<T, WF>(nb / W)));
    // the FP32 form's solve of the remaining columns on the side stream: the same kernel with 16 columns
    // per CTA (two entries per thread), two CTAs per SM (FP64: trsm_mma_kernel)
    constexpr int NCS = NC > 16 ? NC : 16;
    const bool wide = sizeof(T) == 4 && trsm_narrow_smem<T, WF, NCS>(nb / W) <= 110 * 1024;
    if (wide)
        BB_CUDA(cudaFuncSetAttribute(trsm_narrow_kernel<T, WF, NCS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)trsm_narrow_smem<T, WF, NCS>(nb / W)));
    if (sizeof(T) == 8) {
        update_setup();
        BB_CUDA(cudaFuncSetAttribute(trsm_mma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)trsm_mma_smem(nb, 4)));
    }
    c->barrier.alloc(sizeof(unsigned) * 4096);
    BB_CUDA(cudaFuncSetAttribute(panel_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_cap));
    constexpr int LC = ls_cols<T>();
    BB_CUDA(cudaFuncSetAttribute(laswp_panel_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)laswp_panel_smem<T>(nb)));
    iota_kernel<<<(n + 255) / 256, 256, 0, c->stream>>>(w.perm.as<int>(), n);
    BB_CUDA(cudaMemsetAsync(c->status.p, 0, sizeof(int), c->stream));
    int *ipiv = w.ipiv.as<int>();
    int *perm = w.perm.as<int>();
    cudaStream_t s0 = c->stream, s1 = c->side_stream;
    constexpr bool tc = sizeof(T) == 4;  // the tensor-core update (K = 2 nb, a multiple of its 64)
    // SMs the look-ahead update leaves to the panel factorisation beside it: one
    // 16-CTA cluster, and as many again for the panel's own updates and solves
    // between its sub-panels (measured at N = 10,242: mixed LU 46.4 ms with one
    // cluster's SMs left, 44.5 with two, 44.0 with three, where the sweep slows);
    // the grid-wide panel fallback waits for its own SMs
    const int side_cap = std::max(1, G - 2 * CP_CTAS);
    // U12 = L11^-1 A12 of panel k for the columns [c_lo, c_hi), on stream st
    // with the tensor-core update the same launch stages U12 as the update's B operand
    // (crit: the next panel's columns, on the critical path)
    auto u_solve = [&](int k, int c_lo, int c_hi, cudaStream_t st, bool crit) {
        const int cols = c_hi - c_lo;
        if (cols <= 0) return;
        __half *bhi = nullptr, *blo = nullptr;
        float *bsc = nullptr;
        if (tc) tc_stage_u_buffers(c, k, nb, &bhi, &blo, &bsc);
        if constexpr (sizeof(T) == 8) {
            if (!(crit && narrow)) {
                constexpr int per = 4 * TS_COLS;
                trsm_mma_kernel<<<(cols + per - 1) / per, 128, trsm_mma_smem(nb, 4), st>>>(
                    A, ld, k, nb / W, dinv + (size_t)(k / W) * W * W, c_lo, c_hi);
                BB_CUDA(cudaGetLastError());
                return;
            }
        }
        if (crit && narrow)
            trsm_narrow_kernel<T, WF><<<(cols + NC - 1) / NC, 256, trsm_narrow_smem<T, WF>(nb / W), st>>>(
                A, ld, k, nb / W, dinv + (size_t)(k / W) * W * W, c_lo, c_hi, bhi, blo, bsc, k + nb, split_terms);
        else if (wide)
            trsm_narrow_kernel<T, WF, NCS><<<(cols + NCS - 1) / NCS, 256, trsm_narrow_smem<T, WF, NCS>(nb / W), st>>>(
                A, ld, k, nb / W, dinv + (size_t)(k / W) * W * W, c_lo, c_hi, bhi, blo, bsc, k + nb, split_terms);
        else
            trsm_blocked_kernel<T, WF><<<(cols + TB_COLS - 1) / TB_COLS, 256, tb_smem, st>>>(
                A, ld, k, nb / W, dinv + (size_t)(k / W) * W * W, c_lo, c_hi, bhi, blo, bsc, k + nb, split_terms);
        BB_CUDA(cudaGetLastError());
    };
    // A[k+nb.., c_lo..c_hi) -= L21 U12 of panel k, on stream st
    auto update = [&](int k, int c_lo, int c_hi, cudaStream_t st, int cap) {
        if (c_hi <= c_lo || k + nb >= n) return;
        if constexpr (tc)
            tc_update_cols(c, k, nb, split_terms, c_lo, c_hi, st, cap);
        else  // one CTA per tile: a grid capped as the tensor-core one is was slower (154 against 136 ms a factorisation)
            launch_update(st, A, ld, n, k, nb, k + nb, c_lo, c_hi);
    };
    // Right-looking LU with a look-ahead of one panel.  For panel k (columns
    // [k, pe)):
    //   1. factor its sub-panels on s0, swapping rows inside the panel only;
    //   2. wait for the side stream (the previous panel's update of the
    //      columns right of this panel);
    //   3. the panel's interchanges on every other column and the permutation;
    //   4. U12 and the update of the next panel's columns on s0 (they are all
    //      the next panel needs);
    //   5. U12 and the update of the remaining columns on s1, which then runs
    //      beside the next panel's factorisation (step 1 of panel k + nb).
    // The next panel touches only its own columns and rows >= pe until its
    // step 3, which follows the join: the streams never touch the same entries.
    bool side_pending = false;
    for (int k = 0; k < n; k += nb) {
        const int pe = std::min(k + nb, n);  // end of this panel
        for (int ks = k; ks < pe; ks += W) {
            const int m = n - ks;
            Cx<T> *dinv_s = dinv + (size_t)(ks / W) * W * W;
            // the cluster kernel also swaps the panel's other columns when they fit its registers
            constexpr int CHUNK = 16 / sizeof(Cx<T>);
            const int right = std::max(0, pe - ks - W), others = ks - k + right;
            const bool own_swaps = others > 0 && others <= CpShape<T>::MVC * CHUNK && right % CHUNK == 0;
            const bool on_cluster =
                cluster_panel<T>(c, A, ld, n, ks, ipiv, dinv_s, own_swaps ? k : 0, own_swaps ? pe : 0);
            if (!on_cluster) {
                // grid-wide panel kernel on the sub-panel
                int g = std::min(G, std::max(1, (m + 15) / 16));
                int rows = (m + g - 1) / g;
                PanelArgs<T> a;
                a.A = A;
                a.ld = ld;
                a.n = n;
                a.k = ks;
                a.nb = W;
                a.rpc = rows;
                a.ipiv = ipiv;
                a.pub_rows = pub_rows;
                a.pub_diag = pub_diag;
                a.recs = recs;
                a.counter = c->barrier.as<unsigned>();
                a.status = c->status.as<int>();
                a.spin_limit = 1u << 22;
                const size_t ps = sizeof(Cx<T>) * ((size_t)rows * W + 2 * W + rows);
                BB_CUDA(cudaMemsetAsync(c->barrier.p, 0, sizeof(unsigned), s0));
                void *args[] = {&a};
                BB_CUDA(cudaLaunchCooperativeKernel((void *)panel_kernel<T>, dim3(g), dim3(PANEL_THREADS), args, ps,
                                                    s0));
            }
            // this sub-panel's interchanges on the rest of the panel (unless the cluster kernel did them)
            if (others > 0 && !(on_cluster && own_swaps)) {
                laswp_panel_kernel<T><<<(pe - k + LC - 1) / LC, 256, laswp_panel_smem<T>(W), s0>>>(
                    A, ld, n, ks, W, ipiv, k, pe, ks, ks + W, nullptr);
                BB_CUDA(cudaGetLastError());
            }
            if (!on_cluster) {
                diag_block_inverse_kernel<T><<<1, 32, 0, s0>>>(A, ld, n, ks, W, dinv_s);
                BB_CUDA(cudaGetLastError());
            }
            if (ks + W < pe) {
                // rest of this panel: U row block, then the panel's own trailing update
                const int cols = pe - ks - W;
                if (narrow)
                    trsm_narrow_kernel<T, WF><<<(cols + NC - 1) / NC, 256, trsm_narrow_smem<T, WF>(1), s0>>>(
                        A, ld, ks, 1, dinv + (size_t)(ks / W) * W * W, ks + W, pe, nullptr, nullptr, nullptr, 0,
                        split_terms);
                else
                    trsm_blocked_kernel<T, WF><<<(cols + TB_COLS - 1) / TB_COLS, 256, tb_smem, s0>>>(
                        A, ld, ks, 1, dinv + (size_t)(ks / W) * W * W, ks + W, pe);
                if constexpr (sizeof(T) == 4) {
                    dim3 grid((cols + PU_COLS - 1) / PU_COLS, (n - ks - W + PU_ROWS - 1) / PU_ROWS);
                    panel_update_kernel<<<grid, 256, 0, s0>>>(A, ld, n, ks, W, ks + W, ks + W, pe);
                } else {
                    launch_update(s0, A, ld, n, ks, W, ks + W, ks + W, pe);
                }
                BB_CUDA(cudaGetLastError());
            }
        }
        if (side_pending) {
            BB_CUDA(cudaStreamWaitEvent(s0, c->la_join, 0));
            side_pending = false;
        }
        // the panel's interchanges on every column outside it, and on perm
        laswp_panel_kernel<T><<<(n + LC - 1) / LC, 256, laswp_panel_smem<T>(pe - k), s0>>>(A, ld, n, k, pe - k, ipiv, 0,
                                                                                        n, k, pe, perm);
        BB_CUDA(cudaGetLastError());
        if (pe >= n) break;
        const int ne = std::min(pe + nb, n);  // end of the next panel
        if (tc) {
            // L21's staging reads rows >= pe, the U12 solve writes rows < pe: the staging runs on
            // the side stream (idle since the join) beside the solve
            BB_CUDA(cudaEventRecord(c->la_fork, s0));
            BB_CUDA(cudaStreamWaitEvent(s1, c->la_fork, 0));
            tc_stage_l(c, k, nb, split_terms, s1);
            BB_CUDA(cudaEventRecord(c->la_join, s1));
        }
        u_solve(k, pe, ne, s0, true);
        if (tc) BB_CUDA(cudaStreamWaitEvent(s0, c->la_join, 0));
        update(k, pe, ne, s0, 0);
        if (ne < n) {
            BB_CUDA(cudaEventRecord(c->la_fork, s0));
            BB_CUDA(cudaStreamWaitEvent(s1, c->la_fork, 0));
            u_solve(k, ne, n, s1, false);
            update(k, ne, n, s1, side_cap);
            BB_CUDA(cudaEventRecord(c->la_join, s1));
            side_pending = true;
        }
    }
    if (side_pending) BB_CUDA(cudaStreamWaitEvent(s0, c->la_join, 0));
}

// ---------------------------------------------------------------------------
// triangular solves with R right-hand sides (X column-major N x R, FP64)
// ---------------------------------------------------------------------------
__global__ void permute_rows_kernel(const double2 *in, double2 *out, const int *perm, int n, int R) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int src = perm[i];
    for (int r = 0; r < R; ++r) out[(size_t)r * n + i] = in[(size_t)r * n + src];
}

constexpr int SB = 64, SRC = 16, SBP = SB + 1;

template <typename T> __device__ __forceinline__ Cx<double> to_d(Cx<T> v) {
    return Cx<double>{(double)v.re, (double)v.im};
}

// Inverse of every 64 x 64 diagonal block of L (unit lower, blockIdx.y = 0)
// and U (upper, blockIdx.y = 1), FP64, one CTA per block: the 8 x 8 diagonal
// blocks by substitution, a column per thread in registers, then doubling
// (8 -> 64): with the s x s diagonal blocks inverted, the off-diagonal block of
// a pair of them is -Y22 (L21 Y11) for L, -Y11 (U12 Y22) for U.  A block is a
// dependent chain, not bandwidth: substitution over all 64 rows by one thread
// per column took 79 us for N up to 4,700 (one wave), this 17 us.
constexpr int DI_THREADS = 256;
template <typename T>
__global__ void __launch_bounds__(DI_THREADS) diag_inverse_kernel(const Cx<T> *A, int64_t ld, int n, Cx<double> *Dinv) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Cx<double>(*D)[SBP] = reinterpret_cast<Cx<double>(*)[SBP]>(smem_raw);
    Cx<double>(*X)[SBP] = reinterpret_cast<Cx<double>(*)[SBP]>(smem_raw + sizeof(Cx<double>) * SB * SBP);
    const int b = blockIdx.x, upper = blockIdx.y;
    const int rb = b * SB, rows = min(SB, n - rb), tid = threadIdx.x;
    batched_copy<DI_THREADS, 8, Cx<double>>(
        SB * SB,
        [&](int e) {
            const int i = e / SB, c = e % SB;
            return (i < rows && c < rows) ? to_d(A[(int64_t)(rb + i) * ld + rb + c])
                                          : Cx<double>{i == c ? 1.0 : 0.0, 0.0};
        },
        [&](int e, Cx<double> v) {
            D[e / SB][e % SB] = v;
            X[e / SB][e % SB] = Cx<double>{0.0, 0.0};
        });
    __syncthreads();
    if (tid < SB) {
        const int d = tid & ~7, c = tid & 7;
        Cx<double> v[8];
        if (!upper) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                v[i] = Cx<double>{i == c ? 1.0 : 0.0, 0.0};
#pragma unroll
                for (int q = 0; q < i; ++q) v[i] = cms(v[i], D[d + i][d + q], v[q]);
                X[d + i][tid] = v[i];
            }
        } else {
#pragma unroll
            for (int i = 7; i >= 0; --i) {
                v[i] = Cx<double>{i == c ? 1.0 : 0.0, 0.0};
#pragma unroll
                for (int q = i + 1; q < 8; ++q) v[i] = cms(v[i], D[d + i][d + q], v[q]);
                const Cx<double> u = D[d + i][d + i];
                const double den = u.re * u.re + u.im * u.im;
                const double rd = den > 0 ? 1.0 / den : 0.0;
                v[i] = Cx<double>{(v[i].re * u.re + v[i].im * u.im) * rd, (v[i].im * u.re - v[i].re * u.im) * rd};
                X[d + i][tid] = v[i];
            }
        }
    }
    __syncthreads();
    // D's own triangle is read, its other triangle holds the inner products
#pragma unroll 1
    for (int h = 8; h < SB; h *= 2)
#pragma unroll 1
        for (int pass = 0; pass < 2; ++pass) {
            for (int e = tid; e < SB / 2 * h; e += DI_THREADS) {
                const int d = e / (h * h) * 2 * h, i = e / h % h, c = e % h;
                // lower: D[h.., 0..] X[0.., 0..], then X[h.., h..] times it; upper: the halves swapped
                const int lo = upper ? d : d + h, hi = upper ? d + h : d;
                const Cx<double> *left = pass ? &X[lo + i][lo] : &D[lo + i][hi];
                const Cx<double> *right = pass ? &D[hi][lo + c] : &X[hi][hi + c];
                Cx<double> s0{0, 0}, s1{0, 0};
#pragma unroll 4
                for (int t = 0; t < h; t += 2) {
                    s0 = cms(s0, left[t], right[t * SBP]);
                    s1 = cms(s1, left[t + 1], right[(t + 1) * SBP]);
                }
                const Cx<double> v{s0.re + s1.re, s0.im + s1.im};  // -(left right)
                if (pass == 0)
                    D[hi + i][lo + c] = Cx<double>{-v.re, -v.im};
                else
                    X[lo + i][hi + c] = v;
            }
            __syncthreads();
        }
    Cx<double> *out = Dinv + ((size_t)upper * gridDim.x + b) * SB * SB;
    for (int e = tid; e < SB * SB; e += DI_THREADS) out[e] = X[e / SB][e % SB];
}

// H_b^(d) = D_b^-1 M_b for the two blocks nearest the diagonal on the solve's
// critical path: M_b = L[b, b-d] (lower) or U[b, b+d] (upper), d = 1, 2
// (blockIdx.y = 2 (d - 1) + upper; stored in slot 2 + blockIdx.y).  With them,
// X_b = Z_b - H^(2)_b X_{b-+2} - H^(1)_b X_{b-+1}, where Z_b holds everything
// else and is formed while the two neighbouring blocks are solved.
// ADJ: the same for the solves with U^H (lower) and L^H (upper), from D: the
// blocks' inverses of the factors themselves, into Dadj: slots 0, 1 the
// conjugate transposes of D_U, D_L (blockIdx.y = 4, 5), and
// H = (M D_b)^H with M = U[b-d, b] (lower) or L[b+d, b] (upper).
// Each thread forms 4 x 4 outputs (rows ty + 16 i, columns tx + 16 j): FP64
// issue instead of two shared-memory loads per multiply-add (32 -> 17 us, N = 1,390).
template <typename T, bool ADJ>
__global__ void __launch_bounds__(256) offdiag_product_kernel(const Cx<T> *A, int64_t ld, int n,
                                                              const Cx<double> *Dinv, Cx<double> *Dout) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Cx<double> *Lt = reinterpret_cast<Cx<double> *>(smem_raw);  // SB x SBP: the left factor
    Cx<double> *Rt = Lt + SB * SBP;                               // SB x SBP: the right factor
    const int nblk = gridDim.x, b = blockIdx.x, upper = blockIdx.y & 1, dist = 1 + (blockIdx.y >> 1);
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    // the factor whose diagonal block is inverted: ADJ's lower solve is with U^H
    const Cx<double> *D = Dinv + ((size_t)(ADJ ? 1 - upper : upper) * nblk + b) * SB * SB;
    if (ADJ && blockIdx.y >= 4) {
        Cx<double> *out = Dout + ((size_t)upper * nblk + b) * SB * SB;
        for (int i = threadIdx.x; i < SB * SB; i += 256) {
            const Cx<double> v = D[(i % SB) * SB + i / SB];
            out[i] = Cx<double>{v.re, -v.im};
        }
        return;
    }
    const int nb2 = upper ? b + dist : b - dist;
    Cx<double> *H = Dout + ((size_t)(2 + blockIdx.y) * nblk + b) * SB * SB;
    if (nb2 < 0 || nb2 >= nblk) {
        for (int i = threadIdx.x; i < SB * SB; i += 256) H[i] = Cx<double>{0.0, 0.0};
        return;
    }
    const int br = ADJ ? nb2 : b, bc = ADJ ? b : nb2;  // the off-diagonal block's block row and column
    const int rb = br * SB, rows = min(SB, n - rb), cb = bc * SB, cols = min(SB, n - cb);
    Cx<double> *Dt = ADJ ? Rt : Lt, *Mt = ADJ ? Lt : Rt;
    batched_copy<256, 8, Cx<double>>(SB * SB, [&](int i) { return D[i]; },
                                     [&](int i, Cx<double> v) { Dt[(i / SB) * SBP + i % SB] = v; });
    batched_copy<256, 8, Cx<double>>(
        SB * SB,
        [&](int i) {
            const int a = i / SB, q = i % SB;
            return (a < rows && q < cols) ? to_d(A[(int64_t)(rb + a) * ld + cb + q]) : Cx<double>{0.0, 0.0};
        },
        [&](int i, Cx<double> v) { Mt[(i / SB) * SBP + i % SB] = v; });
    __syncthreads();
    Cx<double> acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = Cx<double>{0.0, 0.0};
#pragma unroll 2
    for (int q = 0; q < SB; ++q) {
        Cx<double> l[4], r[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            l[i] = Lt[(ty + 16 * i) * SBP + q];
            r[i] = Rt[q * SBP + tx + 16 * i];
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                acc[i][j].re = fma(l[i].re, r[j].re, fma(-l[i].im, r[j].im, acc[i][j].re));
                acc[i][j].im = fma(l[i].re, r[j].im, fma(l[i].im, r[j].re, acc[i][j].im));
            }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int r = ty + 16 * i, c = tx + 16 * j;
            if (ADJ)
                H[c * SB + r] = Cx<double>{acc[i][j].re, -acc[i][j].im};
            else
                H[r * SB + c] = acc[i][j];
        }
}

// Block substitution in one kernel.  The solution is cut into 64-row blocks;
// each CTA claims the next block from a counter (so it only ever waits on
// blocks already claimed by running CTAs).  For block b it folds in
// L_bj X_j (or U_bj X_j) for every finished block j at distance 3 or more,
// forms Z_b = D_b^-1 (B_b - that sum), subtracts H^(2)_b X_{b-+2} once that
// block is done, and then X_b = Z_b - H^(1)_b X_{b-+1}: the chain from one
// block to the next is a single 64 x 64 x R product, run by the whole CTA.
// Waits are bounded: on expiry the kernel sets a status bit and continues, so
// it always terminates.
//
// Arithmetic is in the factors' type: FP64 for the FP64 form, FP32 for the
// mixed form's factors (there the substitution is the preconditioner of the
// FP64 refinement).  The folded-in products are shared by NG warp groups of
// 128 threads (4 for FP32, 2 for FP64), group g taking steps g, g + NG, ...
// with its own factor tile (cp.async, zero-filled past the matrix edge) and
// X block, synchronised by its own named barrier, so that one SM always has
// several independent tile products in flight; each thread keeps a 2-row x
// RC/4-column block of the 64 x RC product in registers, RC = 4, 8 or 16 the
// columns of a pass (the fewest that hold the right-hand sides left: a pass of
// 16 for one column spends 16 times the arithmetic; one column: FP32 N = 1,390
// 98 -> 79 us a triangle, FP64 N = 2,616 430 -> 220 us).  The groups'
// partial sums meet in shared memory for the tail.
//
// ADJ: the solves with U^H (LOWER) and L^H (upper), FP64 arithmetic in both
// forms: a tile is the conjugate transpose of the factor's tile on the other
// side of the diagonal, and Dinv holds the adjoint blocks.
template <typename T, int RC> struct SubstTile {
    // padded row length: rows start on 16-byte boundaries (cp.async) and a
    // warp's 8 rows fall on distinct banks
    static constexpr int LP = SB + (sizeof(Cx<T>) == 16 ? 1 : 2);
    // the X block column-major with a padded column: the loads (consecutive
    // rows) and the product's reads (four columns at one row) spread over banks
    static constexpr int XP = SB + 1;
    static constexpr int NG = sizeof(Cx<T>) == 16 ? 2 : 4;
    static constexpr int THREADS = 128 * NG;
    static constexpr int GROUP = SB * LP + RC * XP;  // complex entries per group
    static constexpr size_t smem() { return sizeof(Cx<T>) * (size_t)NG * GROUP; }
};

__device__ __forceinline__ bool wait_flag(const int *flag, int epoch, int *status, unsigned spin_limit) {
    unsigned it = 0;
    while (true) {
        int v;
        asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
        if (v == epoch) return true;
        if ((*(volatile int *)status & DEV_BARRIER_TIMEOUT) || ++it > spin_limit) {
            atomicOr(status, (int)DEV_BARRIER_TIMEOUT);
            return false;
        }
    }
}

__device__ __forceinline__ void cp_async16(void *dst, const void *src, int src_bytes) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }
// barrier of one 128-thread warp group (ids 1.. ; 0 is __syncthreads)
__device__ __forceinline__ void group_bar(int grp) {
    asm volatile("bar.sync %0, 128;" ::"r"(grp + 1) : "memory");
}

// acc[2][CT] += M[rows rp, rp + 32][:] V[:][CT cg .. CT cg + CT - 1], V
// column-major with column stride XP
template <typename C, int LP, int XP, int CT>
__device__ __forceinline__ void subst_product(const Cx<C> *M, const Cx<C> *V, int rp, int cg, C (&ar)[2][CT],
                                              C (&ai)[2][CT]) {
#pragma unroll 8
    for (int q = 0; q < SB; ++q) {
        const Cx<C> m0 = M[rp * LP + q], m1 = M[(rp + 32) * LP + q];
#pragma unroll
        for (int e = 0; e < CT; ++e) {
            const Cx<C> v = V[(CT * cg + e) * XP + q];
            ar[0][e] += m0.re * v.re - m0.im * v.im;
            ai[0][e] += m0.re * v.im + m0.im * v.re;
            ar[1][e] += m1.re * v.re - m1.im * v.im;
            ai[1][e] += m1.re * v.im + m1.im * v.re;
        }
    }
}

template <typename T, bool ADJ> using SubstType = std::conditional_t<ADJ, double, T>;
template <typename T, bool LOWER, bool ADJ, int RC>
__global__ void __launch_bounds__(SubstTile<SubstType<T, ADJ>, RC>::THREADS, 1)
    block_subst_kernel(const Cx<T> *A, int64_t ld, int n, const Cx<double> *Dinv, double2 *X, int R, int r0,
                       int *counter, int *flags, int epoch, int *status, unsigned spin_limit) {
    using C = SubstType<T, ADJ>;
    using ST = SubstTile<C, RC>;
    constexpr int LP = ST::LP, XP = ST::XP, NG = ST::NG, CT = RC / 4;
    constexpr int CH = 16 / sizeof(Cx<T>);  // complex entries per 16-byte chunk
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Cx<C> *base = reinterpret_cast<Cx<C> *>(smem_raw);
    __shared__ int s_blk;
    const int nblk = (n + SB - 1) / SB;
    // persistent: a CTA claims the next block when it has released its last one
    for (;;) {
    if (threadIdx.x == 0) s_blk = atomicAdd(counter, 1);
    __syncthreads();
    const int claim = s_blk;
    if (claim >= nblk) return;
    const int tid = threadIdx.x, grp = tid >> 7, gt = tid & 127;
    Cx<C> *Lg = base + (size_t)grp * ST::GROUP;  // this group's factor tile [SB][LP]
    Cx<C> *Xg = Lg + SB * LP;                    // this group's X block [SRC][XP]
    const int b = LOWER ? claim : nblk - 1 - claim;
    const int rb = b * SB, rows = min(SB, n - rb);
    const int rc = min(RC, R - r0);
    const int rp = gt >> 2, cg = gt & 3;  // rows rp, rp + 32; columns CT cg .. CT cg + CT - 1
    // the factor tile of block row b, block column j, into dst: by cp.async,
    // or (ADJ) block row j, block column b transposed and conjugated
    auto issue_tile = [&](int j, Cx<C> *dst) {
        const int cj = j * SB, cols = min(SB, n - cj);
        if constexpr (ADJ) {
            constexpr int BATCH = 16;
            for (int base = 0; base < SB * SB; base += 128 * BATCH) {
                Cx<T> v[BATCH];
#pragma unroll
                for (int u = 0; u < BATCH; ++u) {
                    const int i = base + u * 128 + gt, q = i / SB, a = i % SB;
                    v[u] = (a < rows && q < cols) ? A[(int64_t)(cj + q) * ld + rb + a] : Cx<T>{T(0), T(0)};
                }
#pragma unroll
                for (int u = 0; u < BATCH; ++u) {
                    const int i = base + u * 128 + gt;
                    dst[(i % SB) * LP + i / SB] = Cx<C>{(C)v[u].re, -(C)v[u].im};
                }
            }
        } else {
            for (int i = gt; i < SB * (SB / CH); i += 128) {
                const int a = i / (SB / CH), q = (i % (SB / CH)) * CH;
                const int valid = (a < rows) ? max(0, min(CH, cols - q)) : 0;
                const Cx<T> *src = valid > 0 ? A + (int64_t)(rb + a) * ld + cj + q : A;
                cp_async16(dst + a * LP + q, src, valid * (int)sizeof(Cx<T>));
            }
            cp_async_commit();
        }
    };
    // X_j (FP64, columns r0 .. r0 + rc) into dst in the compute type
    auto load_x = [&](int j, Cx<C> *dst) {
        const int cj = j * SB, cols = min(SB, n - cj);
        for (int i = gt; i < SB * RC; i += 128) {
            const int q = i / SB, a = i % SB;  // consecutive threads: consecutive rows of one column
            const double2 v = (a < cols && q < rc) ? __ldcg(&X[(size_t)(r0 + q) * n + cj + a]) : make_double2(0, 0);
            dst[q * XP + a] = Cx<C>{(C)v.x, (C)v.y};
        }
    };
    C ar[2][CT], ai[2][CT];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int e = 0; e < CT; ++e) ar[h][e] = ai[h][e] = C(0);
    // every finished block at distance >= 3, shared round-robin by the groups
    const int nsteps = claim > 2 ? claim - 2 : 0;
    for (int step = grp; step < nsteps; step += NG) {
        const int j = LOWER ? step : nblk - 1 - step;
        issue_tile(j, Lg);
        if (gt == 0) wait_flag(flags + j, epoch, status, spin_limit);
        group_bar(grp);
        load_x(j, Xg);
        cp_async_wait_all();
        group_bar(grp);
        subst_product<C, LP, XP, CT>(Lg, Xg, rp, cg, ar, ai);
        group_bar(grp);
    }
    // the groups' partial sums meet in shared memory (each in its own X block)
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int e = 0; e < CT; ++e) Xg[(CT * cg + e) * XP + rp + 32 * h] = Cx<C>{ar[h][e], ai[h][e]};
    __syncthreads();

    // tail, the whole CTA.  Thread tid owns rows tr, tr + 32 and columns tc ..
    // tc + TC - 1 of the 64 x RC block; the 64-term sums are split between QS
    // neighbouring lanes (terms qh, qh + QS, ..., so that their loads fall on
    // distinct banks) and combined by shuffles.
    constexpr int THREADS = ST::THREADS, TC = RC == 16 ? 2 : 1, TPR = RC / TC, QS = THREADS / (32 * TPR);
    const int tile = tid / QS, qh = tid % QS;
    const int tr = tile / TPR, tc = (tile % TPR) * TC;
    Cx<C> *T0 = base, *T1 = base + ST::GROUP;  // groups 0 and 1's tiles
    // H^(1)_b: group 2's tile when there is one (loaded with D and H^(2)),
    // else group 0's after the D product
    Cx<C> *TH1 = NG >= 3 ? base + 2 * ST::GROUP : T0;
    Cx<C> *X0 = base + SB * LP;                // group 0's X block
    // an FP64 64 x 64 block (D_b^-1 or H_b) into dst in the compute type
    auto load_block_all = [&](const Cx<double> *src, Cx<C> *dst) {
        for (int i = tid; i < SB * SB; i += THREADS) {
            const Cx<double> v = src[i];
            dst[(i / SB) * LP + i % SB] = Cx<C>{(C)v.re, (C)v.im};
        }
    };
    auto load_x_all = [&](int j) {
        const int cj = j * SB, cols = min(SB, n - cj);
        for (int i = tid; i < SB * RC; i += THREADS) {
            const int q = i / SB, a = i % SB;
            const double2 v = (a < cols && q < rc) ? __ldcg(&X[(size_t)(r0 + q) * n + cj + a]) : make_double2(0, 0);
            X0[q * XP + a] = Cx<C>{(C)v.x, (C)v.y};
        }
    };
    // o[h][e] = M[tr + 32 h, :] X0[:, tc + e]
    auto tail_product = [&](const Cx<C> *M, C (&orr)[2][TC], C (&oi)[2][TC]) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int e = 0; e < TC; ++e) orr[h][e] = oi[h][e] = C(0);
#pragma unroll 8
        for (int i = 0; i < SB / QS; ++i) {
            const int q = QS * i + qh;
            const Cx<C> m0 = M[tr * LP + q], m1 = M[(tr + 32) * LP + q];
#pragma unroll
            for (int e = 0; e < TC; ++e) {
                const Cx<C> v = X0[(tc + e) * XP + q];
                orr[0][e] += m0.re * v.re - m0.im * v.im;
                oi[0][e] += m0.re * v.im + m0.im * v.re;
                orr[1][e] += m1.re * v.re - m1.im * v.im;
                oi[1][e] += m1.re * v.im + m1.im * v.re;
            }
        }
#pragma unroll
        for (int o = 1; o < QS; o *= 2)
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int e = 0; e < TC; ++e) {
                    orr[h][e] += __shfl_xor_sync(0xffffffffu, orr[h][e], o);
                    oi[h][e] += __shfl_xor_sync(0xffffffffu, oi[h][e], o);
                }
    };
    const Cx<double> *Di = Dinv + ((size_t)(LOWER ? 0 : 1) * nblk + b) * SB * SB;
    const Cx<double> *H1 = Dinv + ((size_t)(LOWER ? 2 : 3) * nblk + b) * SB * SB;
    const Cx<double> *H2 = Dinv + ((size_t)(LOWER ? 4 : 5) * nblk + b) * SB * SB;
    // B_b - sum of the partials
    C vr[2][TC], vi[2][TC];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int e = 0; e < TC; ++e) {
            const int r = tr + 32 * h, cc = tc + e;
            C sr = C(0), si = C(0);
#pragma unroll
            for (int g = 0; g < NG; ++g) {
                const Cx<C> v = base[(size_t)g * ST::GROUP + SB * LP + cc * XP + r];
                sr += v.re;
                si += v.im;
            }
            double2 v = make_double2(0, 0);
            if (r < rows && cc < rc) v = X[(size_t)(r0 + cc) * n + rb + r];
            vr[h][e] = (C)v.x - sr;
            vi[h][e] = (C)v.y - si;
        }
    __syncthreads();  // partials read: the groups' buffers are free
    if (qh == 0)
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int e = 0; e < TC; ++e) X0[(tc + e) * XP + tr + 32 * h] = Cx<C>{vr[h][e], vi[h][e]};
    load_block_all(Di, T0);
    if (claim >= 2) load_block_all(H2, T1);
    if (NG >= 3 && claim >= 1) load_block_all(H1, TH1);
    __syncthreads();
    // Z_b = D_b^-1 (B_b - sum)
    C zr[2][TC], zi[2][TC], hr[2][TC], hi[2][TC];
    tail_product(T0, zr, zi);
    __syncthreads();  // T0 and X0 free
    if (NG < 3 && claim >= 1) load_block_all(H1, TH1);  // overlaps the waits below
    auto subtract = [&]() {
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int e = 0; e < TC; ++e) {
                zr[h][e] -= hr[h][e];
                zi[h][e] -= hi[h][e];
            }
    };
    if (claim >= 2) {
        // Z_b -= H^(2)_b X_{b-+2}
        if (tid == 0) wait_flag(flags + (LOWER ? b - 2 : b + 2), epoch, status, spin_limit);
        __syncthreads();
        load_x_all(LOWER ? b - 2 : b + 2);
        __syncthreads();
        tail_product(T1, hr, hi);
        subtract();
        __syncthreads();  // X0 free
    }
    if (claim >= 1) {
        // X_b = Z_b - H^(1)_b X_{b-+1}
        if (tid == 0) wait_flag(flags + (LOWER ? b - 1 : b + 1), epoch, status, spin_limit);
        __syncthreads();
        load_x_all(LOWER ? b - 1 : b + 1);
        __syncthreads();
        tail_product(TH1, hr, hi);
        subtract();
    }
    {  // lane qh < 2 of a tile stores row tr + 32 qh (with one lane per tile, both rows)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (QS >= 2 && h != qh) continue;
            const int r = tr + 32 * h;
#pragma unroll
            for (int e = 0; e < TC; ++e)
                if (r < rows && tc + e < rc)
                    X[(size_t)(r0 + tc + e) * n + rb + r] = make_double2(zr[h][e], zi[h][e]);
        }
    }
    // the CTA barrier orders every thread's stores before thread 0's release
    // (release is cumulative), and consumers acquire the flag before a barrier
    // and their loads
    __syncthreads();
    if (tid == 0) asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(flags + b), "r"(epoch) : "memory");
    }
}

// Persistent CTAs of a block substitution: half the SMs.  A CTA holds about 58 K
// registers, so each one keeps its SM from every other kernel while the chain
// of blocks waits on its flags; at N = 10,242 one triangle takes the same time
// on 74 CTAs as on 148 (2.00 against 2.02 ms for the solve's two), 2.26 ms on 48,
// and the six-lane sweep's best of 8 runs read 18.7-19.1 freq-solves/s with 74
// against 18.3 with 148.
#define SUBST_CTAS_CAP(c) (std::max(1, (c)->sm_count / 2))
// CTAs of a substitution launch: every block's folded-in sum must be under
// way well before the chain reaches it, but a CTA spinning on a flag holds its
// SM, which the other lanes of a sweep could use
static int subst_grid(const beat_b200_ctx *c, int nblk) { return std::min(nblk, SUBST_CTAS_CAP(c)); }

// loads the substitution kernels of every pass width and allows their shared
// memory: at the factorisation, so that a later solve (the allocation-free one
// among them) only launches
template <typename T, bool ADJ> static void subst_setup() {
    auto allow = [](auto *f, size_t smem) {
        BB_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    };
    auto both = [&](auto rc) {
        constexpr int RC = decltype(rc)::value;
        const size_t smem = SubstTile<SubstType<T, ADJ>, RC>::smem();
        allow(block_subst_kernel<T, true, ADJ, RC>, smem);
        allow(block_subst_kernel<T, false, ADJ, RC>, smem);
    };
    both(std::integral_constant<int, 4>{});
    both(std::integral_constant<int, 8>{});
    both(std::integral_constant<int, SRC>{});
}
template <typename T> static void diag_inverses(beat_b200_ctx *c) {
    subst_setup<T, false>();
    Workspace &w = c->ws;
    const int n = c->V, nblk = (n + SB - 1) / SB;
    w.dinv.alloc(sizeof(Cx<double>) * 6 * (size_t)nblk * SB * SB);  // D (L, U), H^(1) (L, U), H^(2) (L, U)
    const size_t smem = 2 * sizeof(Cx<double>) * SB * SBP;
    BB_CUDA(cudaFuncSetAttribute(diag_inverse_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    Cx<double> *d = w.dinv.as<Cx<double>>();
    diag_inverse_kernel<T><<<dim3(nblk, 2), DI_THREADS, smem, c->stream>>>(w.A.as<Cx<T>>(), w.ld, n, d);
    BB_CUDA(cudaFuncSetAttribute(offdiag_product_kernel<T, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem));
    offdiag_product_kernel<T, false><<<dim3(nblk, 4), 256, smem, c->stream>>>(w.A.as<Cx<T>>(), w.ld, n, d, d);
    BB_CUDA(cudaGetLastError());
}

// Both triangles' substitutions on X (N x R, in place) in passes of up to 16
// columns; flags[nblk] must not hold a value of epoch + 1 .. on entry.
template <typename T, bool ADJ, int RC>
static void launch_subst(beat_b200_ctx *c, bool lower, const Cx<double> *Dinv, double2 *X, int R, int r0, int *counter,
                         int *flags, int epoch) {
    using ST = SubstTile<SubstType<T, ADJ>, RC>;
    Workspace &w = c->ws;
    const int n = c->V, nblk = (n + SB - 1) / SB;
    auto *kernel = lower ? block_subst_kernel<T, true, ADJ, RC> : block_subst_kernel<T, false, ADJ, RC>;
    BB_CUDA(cudaMemsetAsync(counter, 0, sizeof(int), c->stream));
    kernel<<<subst_grid(c, nblk), ST::THREADS, ST::smem(), c->stream>>>(w.A.as<Cx<T>>(), w.ld, n, Dinv, X, R, r0,
                                                                        counter, flags, epoch, c->status.as<int>(),
                                                                        1u << 22);
    BB_CUDA(cudaGetLastError());
}
template <typename T, bool ADJ>
static void substitute(beat_b200_ctx *c, const Cx<double> *Dinv, double2 *X, int R, int *counter, int *flags,
                       int &epoch) {
    for (int r0 = 0; r0 < R; r0 += SRC)
        for (int pass = 0; pass < 2; ++pass) {
            const int left = R - r0;
            ++epoch;
            if (left <= 4)
                launch_subst<T, ADJ, 4>(c, pass == 0, Dinv, X, R, r0, counter, flags, epoch);
            else if (left <= 8)
                launch_subst<T, ADJ, 8>(c, pass == 0, Dinv, X, R, r0, counter, flags, epoch);
            else
                launch_subst<T, ADJ, SRC>(c, pass == 0, Dinv, X, R, r0, counter, flags, epoch);
        }
}

// the claim counter and the per-block flags of the context's substitutions
static std::pair<int *, int *> subst_flags(beat_b200_ctx *c) {
    Workspace &w = c->ws;
    const int nblk = (c->V + SB - 1) / SB;
    w.small_solve.alloc(sizeof(int) * (size_t)(nblk + 64));  // [0] claim counter, then nblk flags
    int *counter = w.small_solve.as<int>(), *flags = counter + 32;
    if (w.solve_epoch == 0) BB_CUDA(cudaMemsetAsync(flags, 0, sizeof(int) * nblk, c->stream));
    return {counter, flags};
}

template <typename T> static void lu_solve_t(beat_b200_ctx *c, int R, const double *in, double *out) {
    Workspace &w = c->ws;
    const int n = c->V;
    double2 *X = reinterpret_cast<double2 *>(out);
    const auto [counter, flags] = subst_flags(c);
    permute_rows_kernel<<<(n + 255) / 256, 256, 0, c->stream>>>(reinterpret_cast<const double2 *>(in), X,
                                                                w.perm.as<int>(), n, R);
    BB_CUDA(cudaGetLastError());
    substitute<T, false>(c, w.dinv.as<Cx<double>>(), X, R, counter, flags, w.solve_epoch);
}

// out[perm[i]] = in[i]
__global__ void unpermute_rows_kernel(const double2 *in, double2 *out, const int *perm, int n, int R) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int dst = perm[i];
    for (int r = 0; r < R; ++r) out[(size_t)r * n + dst] = in[(size_t)r * n + i];
}

// A^-H with the stored factors (P A = L U, unit L): A^H = U^H L^H P, so
// z = P^T L^-H U^-H y by the same block substitutions on the conjugate
// transposes of the factors (N = 2,616, FP64, one column: 0.5 ms, against 17 ms
// of alternating column-block products and one-CTA diagonal solves, a launch
// pair per 64 rows).  lu_adjoint_prepare forms their diagonal blocks'
// inverses and the products next to the diagonal from those of the factors,
// once per factorisation and adjoint.
template <typename T> static void adjoint_prepare_t(beat_b200_ctx *c) {
    subst_setup<T, true>();
    Workspace &w = c->ws;
    const int n = c->V, nblk = (n + SB - 1) / SB;
    w.dinv_adj.alloc(sizeof(Cx<double>) * 6 * (size_t)nblk * SB * SB);
    const size_t smem = 2 * sizeof(Cx<double>) * SB * SBP;
    BB_CUDA(cudaFuncSetAttribute(offdiag_product_kernel<T, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem));
    offdiag_product_kernel<T, true><<<dim3(nblk, 6), 256, smem, c->stream>>>(
        w.A.as<Cx<T>>(), w.ld, n, w.dinv.as<Cx<double>>(), w.dinv_adj.as<Cx<double>>());
    BB_CUDA(cudaGetLastError());
}
void lu_adjoint_prepare(beat_b200_ctx *c) {
    if (c->ws.precision == BEAT_B200_FP64)
        adjoint_prepare_t<double>(c);
    else
        adjoint_prepare_t<float>(c);
}
template <typename T> static void lu_solve_adjoint_t(beat_b200_ctx *c, int R, const double *in, double *out) {
    Workspace &w = c->ws;
    const int n = c->V;
    w.x.alloc(sizeof(double2) * (size_t)n * R);
    double2 *Z = w.x.as<double2>();
    BB_CUDA(cudaMemcpyAsync(Z, in, sizeof(double2) * (size_t)n * R, cudaMemcpyDeviceToDevice, c->stream));
    const auto [counter, flags] = subst_flags(c);
    substitute<T, true>(c, w.dinv_adj.as<Cx<double>>(), Z, R, counter, flags, w.solve_epoch);
    unpermute_rows_kernel<<<(n + 255) / 256, 256, 0, c->stream>>>(Z, reinterpret_cast<double2 *>(out),
                                                                  w.perm.as<int>(), n, R);
    BB_CUDA(cudaGetLastError());
}
void lu_solve_adjoint(beat_b200_ctx *c, int R, const double *in, double *out) {
    if (c->ws.precision == BEAT_B200_FP64)
        lu_solve_adjoint_t<double>(c, R, in, out);
    else
        lu_solve_adjoint_t<float>(c, R, in, out);
}

static void lu_factor_eager(beat_b200_ctx *c, int precision, int nb, int split_terms) {
    if (precision == BEAT_B200_FP64) {
        lu_factor_t<double>(c, nb, split_terms);
        diag_inverses<double>(c);
    } else {
        lu_factor_t<float>(c, nb, split_terms);
        diag_inverses<float>(c);
    }
}

void lu_graph_release(beat_b200_ctx *c) {
    if (c->lu_graph) cudaGraphExecDestroy(c->lu_graph);
    c->lu_graph = nullptr;
    c->lu_graph_state = 0;
}

// The factorisation is about 1,300 launches on two streams whose arguments
// depend only on the sizes, the options and the workspace's buffers.  The
// first factorisation with a given key runs eagerly (allocating what it
// needs) and is then captured, without running, into a CUDA graph that later
// factorisations with the same key replay.  The graph keeps each kernel's
// stream priority (the look-ahead's side stream stays below the panels').  A
// capture that fails leaves the eager path in place for that key.
static void lu_key(const beat_b200_ctx *c, int precision, int nb, int split_terms, uint64_t (&key)[12]) {
    const Workspace &w = c->ws;
    const uint64_t k[12] = {(uint64_t)precision, (uint64_t)nb, (uint64_t)split_terms, (uint64_t)c->V,
                            (uint64_t)w.ld, (uint64_t)(uintptr_t)w.A.p, (uint64_t)(uintptr_t)w.ipiv.p,
                            (uint64_t)(uintptr_t)w.perm.p, (uint64_t)(uintptr_t)w.panel_scratch.p,
                            (uint64_t)(uintptr_t)w.stage.p, (uint64_t)(uintptr_t)w.dinv.p,
                            (uint64_t)(uintptr_t)c->status.p};
    std::memcpy(key, k, sizeof(k));
}

void lu_factor(beat_b200_ctx *c, int precision, int nb, int split_terms) {
    uint64_t key[12];
    lu_key(c, precision, nb, split_terms, key);
    const bool same = std::memcmp(key, c->lu_graph_key, sizeof(key)) == 0;
    if (same && c->lu_graph_state == 2) {
        BB_CUDA(cudaGraphLaunch(c->lu_graph, c->stream));
        return;
    }
    if (same && c->lu_graph_state == 3) {
        lu_factor_eager(c, precision, nb, split_terms);
        return;
    }
    lu_graph_release(c);
    lu_factor_eager(c, precision, nb, split_terms);
    // the buffers exist now: capture the same sequence for the next time
    lu_key(c, precision, nb, split_terms, key);
    std::memcpy(c->lu_graph_key, key, sizeof(key));
    c->lu_graph_state = 3;
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return;
    }
    try {
        lu_factor_eager(c, precision, nb, split_terms);
    } catch (...) {
        cudaStreamEndCapture(c->stream, &g);
        if (g) cudaGraphDestroy(g);
        cudaGetLastError();
        return;  // the eager factorisation above stands; this key stays eager
    }
    e = cudaStreamEndCapture(c->stream, &g);
    if (e == cudaSuccess && g) e = cudaGraphInstantiateWithFlags(&c->lu_graph, g, cudaGraphInstantiateFlagUseNodePriority);
    if (g) cudaGraphDestroy(g);
    // upload now, so that the first replay does not pay for it
    if (e == cudaSuccess && c->lu_graph) e = cudaGraphUpload(c->lu_graph, c->stream);
    if (e == cudaSuccess && c->lu_graph) {
        c->lu_graph_state = 2;
    } else {
        if (c->lu_graph) cudaGraphExecDestroy(c->lu_graph);
        c->lu_graph = nullptr;
        cudaGetLastError();
    }
}

void lu_solve_fp64(beat_b200_ctx *c, int R, double *x_dev) {
    // x_dev holds b on entry (N x R), solution on exit; uses ws.x as scratch
    BB_CUDA(cudaMemcpyAsync(c->ws.x.p, x_dev, (size_t)c->V * R * 16, cudaMemcpyDeviceToDevice, c->stream));
    lu_solve_t<double>(c, R, c->ws.x.as<double>(), x_dev);
}

void lu_precond_fp32(beat_b200_ctx *c, int R, const double *in, double *out) {
    lu_solve_t<float>(c, R, in, out);
}

// The same permutation and block substitutions as lu_solve_t, with the claim
// counter and per-block flags in caller-provided device memory (`scratch`,
// at least nblk + 32 ints): x = (L U)^-1 P b with the context's factors.
template <typename T>
static void lu_resolve_into_t(beat_b200_ctx *c, int R, const double *b, double *x, int *scratch) {
    Workspace &w = c->ws;
    const int n = c->V, nblk = (n + SB - 1) / SB;
    double2 *X = reinterpret_cast<double2 *>(x);
    BB_CUDA(cudaMemsetAsync(scratch, 0, sizeof(int) * (size_t)(nblk + 32), c->stream));
    permute_rows_kernel<<<(n + 255) / 256, 256, 0, c->stream>>>(reinterpret_cast<const double2 *>(b), X,
                                                                w.perm.as<int>(), n, R);
    BB_CUDA(cudaGetLastError());
    int epoch = 0;
    substitute<T, false>(c, w.dinv.as<Cx<double>>(), X, R, scratch, scratch + 32, epoch);
}

void lu_resolve_into(beat_b200_ctx *c, int R, const double *b, double *x, int *scratch) {
    if (c->ws.precision == BEAT_B200_FP64)
        lu_resolve_into_t<double>(c, R, b, x, scratch);
    else
        lu_resolve_into_t<float>(c, R, b, x, scratch);
}

}  // namespace bb
