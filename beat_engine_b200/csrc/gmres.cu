// gmres.cu -- FP64 GMRES iterative refinement of the mixed-precision solve.
//
// Right-preconditioned restarted GMRES (flexible form: the preconditioned
// directions Z are kept) on the assembled operator A, one independent Krylov
// space per right-hand side, all columns advanced in lock-step:
//   operator      y = A x with A stored in FP32, arithmetic and vectors FP64
//   preconditioner z = (L U)^-1 P v with the FP32 factors (lu.cu)
//   orthogonalisation classical Gram-Schmidt with one re-orthogonalisation
//   convergence  ||b - A x|| / ||b|| <= rtol for every column
// The reference's nearest counterparts are beat_gmres! (FP64 Krylov space,
// src/BeatEngineDenseSolve.jl:521-665) and beat_refine_cpu_lu (FP64 residual
// of a ComplexF32 LU, src/BeatEngineCpuRefinement.jl:5-78).  Like the latter
// this refines the operator as assembled: FP32 regular-pair arithmetic stays
// in the answer (about 1e-7 relative on these systems).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <complex>
#include <cstring>
#include <vector>

#include "internal.cuh"

namespace bb {

// ---------------------------------------------------------------------------
// Tall-skinny complex products Y += alpha M X and Y += alpha M^H X (M row-major
// in the workspace precision; X, Y FP64 column-major with R columns), on the
// FP64 tensor cores: m8n8k4 blocks, four real products per complex block, an
// FP32 M widened exactly as it is read.  Fragments (PTX ISA, m8n8k4 .f64): A
// (lane / 4, lane % 4), B (lane % 4, lane / 4), C (lane / 4, 2 (lane % 4) + 0, 1).
//
// A warp owns TM_MB blocks of 8 outputs and 8 NB right-hand sides; M's
// fragments go from memory straight to registers (four lanes read four
// neighbours of a row, or eight lanes eight of them in the M^H case: whole
// 32-byte sectors either way; 8- and 16-byte loads, so any ld will do), the next
// 16 reduction indices while the present ones are multiplied.  X goes through
// two cp.async stages; rows of 2 mod 8 entries keep a quarter-warp's loads on
// distinct banks.  The reduction is cut into slices that fill whole waves of
// resident CTAs; they add into Y with FP64 atomics.
//
// An FP64 M's sums of TM_G indices are added to totals (a thread's own places in
// shared memory) and begin again at zero: n terms with random signs in one chain
// round like sqrt(n + K / 2n), and a whole slice as one chain gave B q an error
// of 3.7 / 4.6 / 16e-16 at F = 636 / 1,184 / 9,064, this 2.3 / 2.4 / 3.5e-16 (one
// column of registers per thread in shorter slices: 2.8 / 3.5 / 11e-16), for 5 %
// of the product's time.  An FP32 M's own rounding hides the sum's.
// Bound: M's bytes with up to 8 columns, the FP64 tensor cores with 16.
// FP32 M, R = 16, one N x F and three N x N products with N = 10,242, F = 20,480:
// 3.63 ms with one row and 16 columns of FP64 FMA per thread, 2.80 ms (24
// TFLOP/s of the 37 measured) with this; N = 1,390, R = 4, N x N: 17.8 -> 7.5 us
// (16 columns were computed whatever R was).
// ---------------------------------------------------------------------------
constexpr int TM_WARPS = 8, TM_MB = 2, TM_ROWS = TM_WARPS * TM_MB * 8, TM_KC = 32, TM_G = 16;

__device__ __forceinline__ void tm_mma(double (&c)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(c[0]), "+d"(c[1])
        : "d"(a), "d"(b));
}

template <typename T, int NB> struct TallShape {
    static constexpr bool APART = sizeof(T) == 8;  // groups of TM_G indices summed apart
    static constexpr int XS = 8 * NB + 2;
    static constexpr size_t STAGES = sizeof(double2) * 2 * TM_KC * XS;
    static constexpr size_t SMEM = STAGES + (APART ? sizeof(double2) * 2 * TM_MB * NB * TM_WARPS * 32 : 0);
};

// no outputs, reduction length K: M is no x K (row-major, H = false) or K x no (H = true)
template <typename T, bool H, int NB>
__global__ void __launch_bounds__(TM_WARPS * 32, 2) tall_mma_kernel(const Cx<T> *M, int64_t ld, int no, int K,
                                                                    const double2 *X, double2 *Y, int R, int r0,
                                                                    double alpha, int kslice) {
    using TS = TallShape<T, NB>;
    constexpr int COLS = 8 * NB, XS = TS::XS, STEPS = TM_G / 4, THREADS = TM_WARPS * 32;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    auto sX = reinterpret_cast<double2(*)[TM_KC * XS]>(smem_raw);
    // (FP64) this thread's totals: block (m, n)'s real parts at [2 (m NB + n) THREADS], the imaginary after them
    double2 *tot = reinterpret_cast<double2 *>(smem_raw + TS::STAGES) + threadIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, row = lane >> 2, q = lane & 3;
    const int kb = blockIdx.y * kslice, ke = min(K, kb + kslice);
    const int rc = min(COLS, R - r0);
    const int o0 = blockIdx.x * TM_ROWS + warp * TM_MB * 8 + row;
    const Cx<T> *base[TM_MB];  // outputs past the end read the last one's entries and are not stored
#pragma unroll
    for (int m = 0; m < TM_MB; ++m) {
        const int o = min(o0 + 8 * m, no - 1);
        base[m] = H ? M + o : M + (int64_t)o * ld;
    }
    Cx<T> cur[STEPS][TM_MB], nxt[STEPS][TM_MB];
    auto load = [&](Cx<T> (&a)[STEPS][TM_MB], int k0) {
#pragma unroll
        for (int s = 0; s < STEPS; ++s) {
            const int k = k0 + 4 * s + q;
#pragma unroll
            for (int m = 0; m < TM_MB; ++m)
                a[s][m] = k < ke ? base[m][H ? (int64_t)k * ld : (int64_t)k] : Cx<T>{T(0), T(0)};
        }
    };
    auto stage = [&](int buf, int k0) {
        for (int i = threadIdx.x; i < TM_KC * COLS; i += TM_WARPS * 32) {
            const int c = i / TM_KC, k = i % TM_KC;
            const bool in = c < rc && k0 + k < ke;
            const double2 *src = in ? &X[(size_t)(r0 + c) * K + k0 + k] : X;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                             (unsigned)__cvta_generic_to_shared(&sX[buf][k * XS + c])),
                         "l"(src), "r"(in ? 16 : 0)
                         : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    double re[TM_MB][NB][2] = {}, im[TM_MB][NB][2] = {};
    if constexpr (TS::APART) {
#pragma unroll
        for (int i = 0; i < 2 * TM_MB * NB; ++i) tot[i * THREADS] = make_double2(0.0, 0.0);
    }
    auto add = [&](double2 &t, double (&v)[2]) {
        t = make_double2(t.x + v[0], t.y + v[1]);
        v[0] = v[1] = 0.0;
    };
    stage(0, kb);
    load(cur, kb);
    int buf = 0;
    for (int k0 = kb; k0 < ke; k0 += TM_KC, buf ^= 1) {
        stage(buf ^ 1, k0 + TM_KC);  // past the slice: zeros
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
#pragma unroll
        for (int g = 0; g < TM_KC; g += TM_G) {
            load(nxt, k0 + g + TM_G);
#pragma unroll
            for (int s = 0; s < STEPS; ++s) {
                const double2 *x = &sX[buf][(g + 4 * s + q) * XS + row];
                double2 b[NB];
#pragma unroll
                for (int n = 0; n < NB; ++n) b[n] = x[8 * n];
#pragma unroll
                for (int m = 0; m < TM_MB; ++m) {
                    const double ar = (double)cur[s][m].re;
                    const double ai = H ? -(double)cur[s][m].im : (double)cur[s][m].im, ni = -ai;
#pragma unroll
                    for (int n = 0; n < NB; ++n) {
                        tm_mma(re[m][n], ar, b[n].x);
                        tm_mma(im[m][n], ar, b[n].y);
                    }
#pragma unroll
                    for (int n = 0; n < NB; ++n) {
                        tm_mma(re[m][n], ni, b[n].y);
                        tm_mma(im[m][n], ai, b[n].x);
                    }
                }
            }
            if constexpr (TS::APART) {
#pragma unroll
                for (int m = 0; m < TM_MB; ++m)
#pragma unroll
                    for (int n = 0; n < NB; ++n) {
                        add(tot[2 * (m * NB + n) * THREADS], re[m][n]);
                        add(tot[(2 * (m * NB + n) + 1) * THREADS], im[m][n]);
                    }
            }
#pragma unroll
            for (int s = 0; s < STEPS; ++s)
#pragma unroll
                for (int m = 0; m < TM_MB; ++m) cur[s][m] = nxt[s][m];
        }
        __syncthreads();
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
    for (int m = 0; m < TM_MB; ++m) {
        const int o = o0 + 8 * m;
        if (o >= no) continue;
#pragma unroll
        for (int n = 0; n < NB; ++n) {
            if constexpr (TS::APART) {
                const double2 a = tot[2 * (m * NB + n) * THREADS], b = tot[(2 * (m * NB + n) + 1) * THREADS];
                re[m][n][0] = a.x, re[m][n][1] = a.y;
                im[m][n][0] = b.x, im[m][n][1] = b.y;
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int c = 8 * n + 2 * q + h;
                if (c >= rc) continue;
                double2 *y = &Y[(size_t)(r0 + c) * no + o];
                atomicAdd(&y->x, alpha * re[m][n][h]);
                atomicAdd(&y->y, alpha * im[m][n][h]);
            }
        }
    }
}

template <typename T, bool H>
static void tall_product(cudaStream_t st, int sm_count, const Cx<T> *M, int64_t ld, int no, int K, const double *X,
                         double *Y, int R, double alpha) {
    const int tiles = (no + TM_ROWS - 1) / TM_ROWS, chunks = (K + TM_KC - 1) / TM_KC;
    for (int r0 = 0; r0 < R; r0 += 16) {
        // 8 columns when no more are left: half the products, the same bytes of M
        const auto kernel = R - r0 <= 8 ? tall_mma_kernel<T, H, 1> : tall_mma_kernel<T, H, 2>;
        const size_t smem = R - r0 <= 8 ? TallShape<T, 1>::SMEM : TallShape<T, 2>::SMEM;
        if (smem > 48 * 1024)
            BB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        int per_sm = 1;
        BB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, TM_WARPS * 32, smem));
        const int per = chunks_per_slice(tiles, chunks, std::max(1, per_sm) * sm_count, 2);
        const int kslice = per * TM_KC;
        kernel<<<dim3(tiles, (K + kslice - 1) / kslice), TM_WARPS * 32, smem, st>>>(
            M, ld, no, K, reinterpret_cast<const double2 *>(X), reinterpret_cast<double2 *>(Y), R, r0, alpha, kslice);
        BB_CUDA(cudaGetLastError());
    }
}

// Y += alpha * M X for all R columns (Y must hold its starting value)
template <typename T>
void tall_gemm(cudaStream_t st, int sm_count, const Cx<T> *M, int64_t ld, int rows, int K, const double *X, double *Y,
               int R, double alpha) {
    tall_product<T, false>(st, sm_count, M, ld, rows, K, X, Y, R, alpha);
}
template void tall_gemm<float>(cudaStream_t, int, const Cx<float> *, int64_t, int, int, const double *, double *, int,
                               double);
template void tall_gemm<double>(cudaStream_t, int, const Cx<double> *, int64_t, int, int, const double *, double *,
                                int, double);

// Y += alpha * M^H X (the adjoint: B^H, and A^H inside its refinement)
template <typename T>
void tall_gemm_h(cudaStream_t st, int sm_count, const Cx<T> *M, int64_t ld, int rows, int cols, const double *X,
                 double *Y, int R, double alpha) {
    tall_product<T, true>(st, sm_count, M, ld, cols, rows, X, Y, R, alpha);
}
template void tall_gemm_h<float>(cudaStream_t, int, const Cx<float> *, int64_t, int, int, const double *, double *,
                                 int, double);
template void tall_gemm_h<double>(cudaStream_t, int, const Cx<double> *, int64_t, int, int, const double *,
                                  double *, int, double);

// Y = alpha * A X + beta * Y with beta in {0, 1}
// (with ADJ: Y = alpha * A^H X + beta * Y)
template <typename T, bool ADJ = false>
static void matvec(beat_b200_ctx *c, const Cx<T> *A, const double *X, double *Y, int R, double alpha, double beta) {
    const int n = c->V;
    if (beta == 0.0) BB_CUDA(cudaMemsetAsync(Y, 0, sizeof(double2) * (size_t)n * R, c->stream));
    if (ADJ)
        tall_gemm_h<T>(c->stream, c->sm_count, A, c->ws.ld, n, n, X, Y, R, alpha);
    else
        tall_gemm<T>(c->stream, c->sm_count, A, c->ws.ld, n, n, X, Y, R, alpha);
}

// H[i*R + r] = sum_n conj(V_i[n, r]) W[n, r] for i < nv   (one CTA per (i, r))
__global__ void block_dot_kernel(const double2 *V, size_t vstride, int nv, const double2 *W, int n, int R,
                                 double2 *H) {
    const int i = blockIdx.x / R, r = blockIdx.x % R;
    if (i >= nv) return;
    const double2 *v = V + i * vstride + (size_t)r * n, *w = W + (size_t)r * n;
    double sr = 0, si = 0;
    for (int t = threadIdx.x; t < n; t += blockDim.x) {
        const double2 a = v[t], b = w[t];
        sr += a.x * b.x + a.y * b.y;
        si += a.x * b.y - a.y * b.x;
    }
    __shared__ double rr[32], ri[32];
    for (int o = 16; o > 0; o >>= 1) {
        sr += __shfl_xor_sync(0xffffffffu, sr, o);
        si += __shfl_xor_sync(0xffffffffu, si, o);
    }
    if ((threadIdx.x & 31) == 0) {
        rr[threadIdx.x >> 5] = sr;
        ri[threadIdx.x >> 5] = si;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0, b = 0;
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) {
            a += rr[k];
            b += ri[k];
        }
        H[(size_t)i * R + r] = make_double2(a, b);
    }
}

// W[:, r] -= sum_i V_i[:, r] H[i, r]; optionally accumulates H into Hacc
__global__ void block_axpy_kernel(const double2 *V, size_t vstride, int nv, double2 *W, int n, int R,
                                  const double2 *H, double2 *Hacc) {
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx < (size_t)nv * R && Hacc) {
        Hacc[idx].x += H[idx].x;
        Hacc[idx].y += H[idx].y;
    }
    if (idx >= (size_t)n * R) return;
    const int r = (int)(idx / n);
    double sr = 0, si = 0;
    for (int i = 0; i < nv; ++i) {
        const double2 v = V[i * vstride + idx], h = H[(size_t)i * R + r];
        sr += v.x * h.x - v.y * h.y;
        si += v.x * h.y + v.y * h.x;
    }
    W[idx].x -= sr;
    W[idx].y -= si;
}

// column norms: out[r] = ||W[:, r]||^2 (real, stored in .x)
__global__ void col_norm2_kernel(const double2 *W, int n, int R, double2 *out) {
    const int r = blockIdx.x;
    double s = 0;
    for (int t = threadIdx.x; t < n; t += blockDim.x) {
        const double2 a = W[(size_t)r * n + t];
        s += a.x * a.x + a.y * a.y;
    }
    __shared__ double red[32];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0;
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) a += red[k];
        out[r] = make_double2(a, 0.0);
    }
}

// dst[:, r] = src[:, r] * scale[r] (real scale)
__global__ void col_scale_kernel(const double2 *src, double2 *dst, int n, int R, const double *scale) {
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (size_t)n * R) return;
    const double s = scale[idx / n];
    dst[idx] = make_double2(src[idx].x * s, src[idx].y * s);
}

// x[:, r] += sum_i Z_i[:, r] y[i, r]
__global__ void update_x_kernel(const double2 *Z, size_t zstride, int nz, double2 *X, int n, int R,
                                const double2 *y) {
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (size_t)n * R) return;
    const int r = (int)(idx / n);
    double sr = 0, si = 0;
    for (int i = 0; i < nz; ++i) {
        const double2 z = Z[i * zstride + idx], h = y[(size_t)i * R + r];
        sr += z.x * h.x - z.y * h.y;
        si += z.x * h.y + z.y * h.x;
    }
    X[idx].x += sr;
    X[idx].y += si;
}

using cd = std::complex<double>;

// FGMRES on A (ADJ: on A^H) with the FP32 LU (ADJ: its conjugate transpose)
// as right preconditioner
template <typename T, bool ADJ>
static IrResult gmres_t(beat_b200_ctx *c, int R, double *x_dev, const double *b_dev, int m, int max_iters,
                        double rtol) {
    Workspace &w = c->ws;
    const int n = c->V;
    const size_t vs = (size_t)n * R;  // stride between basis vectors (complex entries)
    const Cx<T> *A = (sizeof(T) == 8) ? w.A.as<Cx<T>>() : w.Aop.as<Cx<T>>();
    w.krylov.alloc(sizeof(double2) * vs * (2 * (size_t)m + 3));
    double2 *V = w.krylov.as<double2>();          // m + 1 vectors
    double2 *Z = V + vs * (m + 1);                // m vectors
    double2 *W = Z + vs * m;                      // work vector
    w.small.alloc(sizeof(double2) * ((size_t)(m + 2) * R * 3 + 4 * R));
    double2 *dH = w.small.as<double2>();          // (m+1) x R
    double2 *dH2 = dH + (size_t)(m + 2) * R;
    double2 *dY = dH2 + (size_t)(m + 2) * R;
    double *dscale = reinterpret_cast<double *>(dY + (size_t)(m + 2) * R);
    const int th = 256;
    const unsigned blocks_nr = (unsigned)((vs + th - 1) / th);

    std::vector<double> bnorm(R), res(R, 1.0);
    std::vector<double2> hbuf((size_t)(m + 2) * R);
    // norms of b and of the first residual, and the status word after the
    // factorisation queued before this refinement: one wait
    col_norm2_kernel<<<R, 256, 0, c->stream>>>(reinterpret_cast<const double2 *>(b_dev), n, R, dH + R);
    if (!ADJ) BB_CUDA(cudaMemcpyAsync(dH + 2 * R, status_kept(c), sizeof(int), cudaMemcpyDeviceToDevice, c->stream));

    int iters = 0;
    bool converged = false;
    std::vector<std::vector<cd>> H(R, std::vector<cd>((size_t)(m + 1) * m));
    std::vector<std::vector<cd>> g(R, std::vector<cd>(m + 1)), cs(R, std::vector<cd>(m)), sn(R, std::vector<cd>(m));
    std::vector<double> cs_r;
    while (iters < max_iters) {
        // r = b - A x
        BB_CUDA(cudaMemcpyAsync(W, b_dev, sizeof(double2) * vs, cudaMemcpyDeviceToDevice, c->stream));
        matvec<T, ADJ>(c, A, x_dev, reinterpret_cast<double *>(W), R, -1.0, 1.0);
        col_norm2_kernel<<<R, 256, 0, c->stream>>>(W, n, R, dH);
        const bool first = iters == 0;
        BB_CUDA(cudaMemcpyAsync(hbuf.data(), dH, sizeof(double2) * (first ? 2 * R + (ADJ ? 0 : 1) : R),
                                cudaMemcpyDeviceToHost, c->stream));
        BB_CUDA(cudaStreamSynchronize(c->stream));
        if (first) {
            if (!ADJ) {
                std::memcpy(&c->h_status[1], &hbuf[2 * R], sizeof(int));
                check_factor_status(c);
            }
            for (int r = 0; r < R; ++r) bnorm[r] = std::sqrt(hbuf[R + r].x);
        }
        std::vector<double> beta(R), sc(R);
        converged = true;
        for (int r = 0; r < R; ++r) {
            beta[r] = std::sqrt(hbuf[r].x);
            res[r] = bnorm[r] > 0 ? beta[r] / bnorm[r] : (beta[r] == 0 ? 0.0 : INFINITY);
            if (!(res[r] <= rtol)) converged = false;
            sc[r] = beta[r] > 0 ? 1.0 / beta[r] : 0.0;
            std::fill(g[r].begin(), g[r].end(), cd(0));
            g[r][0] = beta[r];
        }
        if (converged) break;
        BB_CUDA(cudaMemcpyAsync(dscale, sc.data(), sizeof(double) * R, cudaMemcpyHostToDevice, c->stream));
        col_scale_kernel<<<blocks_nr, th, 0, c->stream>>>(W, V, n, R, dscale);
        int j = 0;
        for (; j < m && iters < max_iters; ++j, ++iters) {
            if (ADJ)
                lu_solve_adjoint(c, R, reinterpret_cast<const double *>(V + vs * j),
                                 reinterpret_cast<double *>(Z + vs * j));
            else
                lu_precond_fp32(c, R, reinterpret_cast<const double *>(V + vs * j),
                                reinterpret_cast<double *>(Z + vs * j));
            matvec<T, ADJ>(c, A, reinterpret_cast<const double *>(Z + vs * j), reinterpret_cast<double *>(W), R, 1.0,
                           0.0);
            // CGS2
            BB_CUDA(cudaMemsetAsync(dH2, 0, sizeof(double2) * (size_t)(j + 1) * R, c->stream));
            for (int pass = 0; pass < 2; ++pass) {
                block_dot_kernel<<<(j + 1) * R, 256, 0, c->stream>>>(V, vs, j + 1, W, n, R, dH);
                block_axpy_kernel<<<blocks_nr, th, 0, c->stream>>>(V, vs, j + 1, W, n, R, dH, dH2);
            }
            col_norm2_kernel<<<R, 256, 0, c->stream>>>(W, n, R, dH2 + (size_t)(j + 1) * R);
            BB_CUDA(cudaMemcpyAsync(hbuf.data(), dH2, sizeof(double2) * (size_t)(j + 2) * R, cudaMemcpyDeviceToHost,
                                    c->stream));
            BB_CUDA(cudaStreamSynchronize(c->stream));
            bool all_ok = true;
            for (int r = 0; r < R; ++r) {
                std::vector<cd> &h = H[r];
                for (int i = 0; i <= j; ++i) h[(size_t)i * m + j] = cd(hbuf[(size_t)i * R + r].x, hbuf[(size_t)i * R + r].y);
                const double hn = std::sqrt(hbuf[(size_t)(j + 1) * R + r].x);
                sc[r] = hn > 0 ? 1.0 / hn : 0.0;
                // apply previous rotations
                for (int i = 0; i < j; ++i) {
                    const cd a = h[(size_t)i * m + j], b = h[(size_t)(i + 1) * m + j];
                    h[(size_t)i * m + j] = std::conj(cs[r][i]) * a + std::conj(sn[r][i]) * b;
                    h[(size_t)(i + 1) * m + j] = -sn[r][i] * a + cs[r][i] * b;
                }
                const cd a = h[(size_t)j * m + j];
                const double den = std::sqrt(std::norm(a) + hn * hn);
                if (den > 0) {
                    cs[r][j] = a / den;
                    sn[r][j] = cd(hn / den, 0.0);
                } else {
                    cs[r][j] = 1.0;
                    sn[r][j] = 0.0;
                }
                h[(size_t)j * m + j] = std::conj(cs[r][j]) * a + std::conj(sn[r][j]) * hn;
                const cd gj = g[r][j];
                g[r][j] = std::conj(cs[r][j]) * gj;
                g[r][j + 1] = -sn[r][j] * gj;
                const double est = bnorm[r] > 0 ? std::abs(g[r][j + 1]) / bnorm[r] : 0.0;
                if (!(est <= rtol)) all_ok = false;
            }
            if (all_ok) {
                ++j;
                ++iters;
                break;
            }
            BB_CUDA(cudaMemcpyAsync(dscale, sc.data(), sizeof(double) * R, cudaMemcpyHostToDevice, c->stream));
            col_scale_kernel<<<blocks_nr, th, 0, c->stream>>>(W, V + vs * (j + 1), n, R, dscale);
        }
        // back substitution per column, x += Z y
        std::vector<double2> yv((size_t)j * R);
        for (int r = 0; r < R; ++r) {
            std::vector<cd> y(j);
            for (int i = j - 1; i >= 0; --i) {
                cd s = g[r][i];
                for (int l = i + 1; l < j; ++l) s -= H[r][(size_t)i * m + l] * y[l];
                const cd d = H[r][(size_t)i * m + i];
                y[i] = std::abs(d) > 0 ? s / d : cd(0);
            }
            for (int i = 0; i < j; ++i) yv[(size_t)i * R + r] = make_double2(y[i].real(), y[i].imag());
        }
        BB_CUDA(cudaMemcpyAsync(dY, yv.data(), sizeof(double2) * yv.size(), cudaMemcpyHostToDevice, c->stream));
        update_x_kernel<<<blocks_nr, th, 0, c->stream>>>(Z, vs, j, reinterpret_cast<double2 *>(x_dev), n, R, dY);
        BB_CUDA(cudaGetLastError());
    }
    if (!converged) {
        // final true residual
        BB_CUDA(cudaMemcpyAsync(W, b_dev, sizeof(double2) * vs, cudaMemcpyDeviceToDevice, c->stream));
        matvec<T, ADJ>(c, A, x_dev, reinterpret_cast<double *>(W), R, -1.0, 1.0);
        col_norm2_kernel<<<R, 256, 0, c->stream>>>(W, n, R, dH);
        BB_CUDA(cudaMemcpyAsync(hbuf.data(), dH, sizeof(double2) * R, cudaMemcpyDeviceToHost, c->stream));
        BB_CUDA(cudaStreamSynchronize(c->stream));
        converged = true;
        for (int r = 0; r < R; ++r) {
            res[r] = bnorm[r] > 0 ? std::sqrt(hbuf[r].x) / bnorm[r] : 0.0;
            if (!(res[r] <= rtol)) converged = false;
        }
    }
    double worst = 0;
    for (int r = 0; r < R; ++r) worst = std::max(worst, res[r]);
    return IrResult{iters, converged ? 1 : 0, worst};
}

IrResult gmres_refine(beat_b200_ctx *c, int R, double *x_dev, const double *b_dev, int restart, int max_iters,
                      double rtol) {
    BB_REQUIRE(restart >= 1 && restart <= 200, BEAT_B200_INVALID_ARG, "GMRES restart must be in 1..200");
    BB_REQUIRE(rtol > 0 && std::isfinite(rtol), BEAT_B200_INVALID_ARG, "GMRES tolerance must be positive");
    return gmres_t<float, false>(c, R, x_dev, b_dev, restart, max_iters, rtol);
}

IrResult gmres_refine_adjoint(beat_b200_ctx *c, int R, double *x_dev, const double *b_dev, int restart, int max_iters,
                              double rtol) {
    BB_REQUIRE(restart >= 1 && restart <= 200, BEAT_B200_INVALID_ARG, "GMRES restart must be in 1..200");
    BB_REQUIRE(rtol > 0 && std::isfinite(rtol), BEAT_B200_INVALID_ARG, "GMRES tolerance must be positive");
    return gmres_t<float, true>(c, R, x_dev, b_dev, restart, max_iters, rtol);
}

}  // namespace bb
