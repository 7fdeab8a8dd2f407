// assembly.cu -- fused Burton-Miller system assembly on sm_100a.
//
//   A = 0.5 M_p1p1 - D + eta H            (N x N, row = test vertex)
//   B = -S - eta (K' + 0.5 M_p1dp0)       (N x F, column = trial face)
//   b = B q                               (N x R, FP64)
//
// Reference (paths relative to src/beat_engine/julia_local/src/):
//   per point pair combination   BeatEngineCpuBurtonMiller.jl:53-112 (regular),
//                                :116-167 (Duffy), green BeatEngineCpuAssembly.jl:1-6
//   CUDA element-pair kernel      BeatEngineCudaRegular.jl:18-383
//   Duffy block kernel + scatter  BeatEngineCudaSingular.jl:359-588,
//                                 BeatEngineCudaBurtonMiller.jl:97-162,273-329
//   identity kernel               BeatEngineCudaBurtonMiller.jl:21-69
//   cached RHS operator  b = B Q  BeatEngineCudaBurtonMiller.jl:774-830
//
// Design (no reference counterpart): elements are sorted along a Morton curve
// and cut into tiles of consecutive elements with few distinct vertices.  One
// CTA integrates a (test tile x trial tile) block of element pairs; each
// pair's 3x3 block and 3-vector land in shared-memory accumulators indexed by
// tile-local vertex numbers, and the CTA flushes them to HBM once with
// red.global.add.  The Duffy kernel runs one warp per touching pair, lanes
// over the Duffy points, in FP64 in both precision forms.
#include <cuda_runtime.h>

#include "internal.cuh"
#include "phase.cuh"

namespace bb {

// rule tables: index 0 -> 1-point, 1 -> 3-point, 2 -> 6-point (order 4)
__constant__ double c_rw64[3][6];
__constant__ double c_rb64[3][6][3];
__constant__ float c_rw32[3][6];
__constant__ float c_rb32[3][6][3];
__constant__ float2 c_rb32x2[3][6][3];  // (b, b): the packed-pair operand of the same basis value

template <typename T> struct RuleRef;
template <> struct RuleRef<double> {
    static __device__ __forceinline__ double w(int r, int q) { return c_rw64[r][q]; }
    static __device__ __forceinline__ double b(int r, int q, int a) { return c_rb64[r][q][a]; }
};
template <> struct RuleRef<float> {
    static __device__ __forceinline__ float w(int r, int q) { return c_rw32[r][q]; }
    static __device__ __forceinline__ float b(int r, int q, int a) { return c_rb32[r][q][a]; }
};

void upload_rule_tables(const std::vector<double> &pts, const std::vector<double> &w, int Q) {
    double w64[3][6] = {}, b64[3][6][3] = {};
    float w32[3][6] = {}, b32[3][6][3] = {};
    BB_CUDA(cudaMemcpyFromSymbol(w64, c_rw64, sizeof(w64)));
    BB_CUDA(cudaMemcpyFromSymbol(b64, c_rb64, sizeof(b64)));
    const int r = Q == 1 ? 0 : Q == 3 ? 1 : 2;
    for (int q = 0; q < Q; ++q) {
        w64[r][q] = w[q];
        b64[r][q][0] = 1.0 - pts[2 * q] - pts[2 * q + 1];
        b64[r][q][1] = pts[2 * q];
        b64[r][q][2] = pts[2 * q + 1];
    }
    for (int i = 0; i < 3; ++i)
        for (int q = 0; q < 6; ++q) {
            w32[i][q] = (float)w64[i][q];
            for (int a = 0; a < 3; ++a) b32[i][q][a] = (float)b64[i][q][a];
        }
    BB_CUDA(cudaMemcpyToSymbol(c_rw64, w64, sizeof(w64)));
    BB_CUDA(cudaMemcpyToSymbol(c_rb64, b64, sizeof(b64)));
    BB_CUDA(cudaMemcpyToSymbol(c_rw32, w32, sizeof(w32)));
    BB_CUDA(cudaMemcpyToSymbol(c_rb32, b32, sizeof(b32)));
    float2 b32x2[3][6][3];
    for (int i = 0; i < 3; ++i)
        for (int q = 0; q < 6; ++q)
            for (int a = 0; a < 3; ++a) b32x2[i][q][a] = make_float2(b32[i][q][a], b32[i][q][a]);
    BB_CUDA(cudaMemcpyToSymbol(c_rb32x2, b32x2, sizeof(b32x2)));
}

// FP32 phase given in revolutions, t = x / (2 pi): t - rint(t) is exact,
// so the reduction to [-1/2, 1/2] is one rounding and one subtraction.  The
// multiply back to radians adds at most about 2^-22 absolute on [-pi, pi],
// below the hardware approximation's own error there (about 2^-21.4); for
// large phases the rounding of t itself (relative 2^-24) dominates.
__device__ __forceinline__ void sincos_rev(float t, float *s, float *c) {
    __sincosf((t - rintf(t)) * 6.2831854820251465f, s, c);
}
__device__ __forceinline__ double rsqrt_t(double x) { return rsqrt_series(x); }
__device__ __forceinline__ float rsqrt_t(float x) { return rsqrtf(x); }

__device__ __forceinline__ void red_add(double *p, double v) { atomicAdd(p, v); }
__device__ __forceinline__ void red_add(float *p, float v) { atomicAdd(p, v); }
// Packed FP32 pairs (sm_100 f32x2 arithmetic): two lanes of one instruction,
// (re, im) of a complex value or one value twice.
using F2 = unsigned long long;
__device__ __forceinline__ F2 pk2(float lo, float hi) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void up2(F2 v, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
    F2 d;
    asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
    F2 d;
    asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
    F2 d;
    asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ F2 rule_b2(int r, int q, int a) {
    return *reinterpret_cast<const F2 *>(&c_rb32x2[r][q][a]);
}

// Adds v[i] to base[off[i]] for every i, atomically.  Shared-memory float
// adds are compare-and-swap loops, each a dependent load -> add -> swap
// chain; here the loads, then the swaps, of all N adds are in flight
// together, and only a swap that lost to another warp's add is redone as an
// ordinary atomic add.  (ABA is harmless: the swap writes old + v over old.)
template <int N>
__device__ __forceinline__ void batch_add(float *base, const int (&off)[N], const float (&v)[N]) {
    static_assert(N <= 32, "one failure bit per add");
    unsigned old[N];
#pragma unroll
    for (int i = 0; i < N; ++i) old[i] = *reinterpret_cast<volatile unsigned *>(base + off[i]);
    unsigned fail = 0;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const unsigned got =
            atomicCAS(reinterpret_cast<unsigned *>(base + off[i]), old[i], __float_as_uint(__uint_as_float(old[i]) + v[i]));
        fail |= (got != old[i] ? 1u : 0u) << i;
    }
    if (fail) {
#pragma unroll
        for (int i = 0; i < N; ++i)
            if (fail >> i & 1u) atomicAdd(base + off[i], v[i]);
    }
}
// the same for double words (64-bit compare-and-swap)
template <int N>
__device__ __forceinline__ void batch_add(double *base, const int (&off)[N], const double (&v)[N]) {
    static_assert(N <= 32, "one failure bit per add");
    using U = unsigned long long;
    U old[N];
#pragma unroll
    for (int i = 0; i < N; ++i) old[i] = *reinterpret_cast<volatile U *>(base + off[i]);
    unsigned fail = 0;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const double sum = __longlong_as_double((long long)old[i]) + v[i];
        const U got = atomicCAS(reinterpret_cast<U *>(base + off[i]), old[i], (U)__double_as_longlong(sum));
        fail |= (got != old[i] ? 1u : 0u) << i;
    }
    if (fail) {
#pragma unroll
        for (int i = 0; i < N; ++i)
            if (fail >> i & 1u) atomicAdd(base + off[i], v[i]);
    }
}
// 4-byte global -> shared copy through the asynchronous copy unit: a CTA's
// tile arrays are all in flight at once and waited for together
__device__ __forceinline__ void cp_async4(void *smem, const void *gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem)
                 : "memory");
}
// the same for one 4- or 8-byte element
template <typename E> __device__ __forceinline__ void cp_async_el(E *smem, const E *gmem) {
    static_assert(sizeof(E) == 4 || sizeof(E) == 8, "cp.async element of 4 or 8 bytes");
    if constexpr (sizeof(E) == 4)
        cp_async4(smem, gmem);
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(smem)),
                     "l"(gmem)
                     : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

__device__ __forceinline__ void red_add_cx(Cx<double> *p, double re, double im) {
    atomicAdd(&p->re, re);
    atomicAdd(&p->im, im);
}
__device__ __forceinline__ void red_add_cx(Cx<float> *p, float re, float im) {
    atomicAdd(reinterpret_cast<float2 *>(p), make_float2(re, im));
}

// Where the right-hand-side operator goes.  Cached (B set): the N x F
// mapping B, b = B q formed afterwards by one tall product.  Matrix-free (B
// null): b = B q directly for the R columns of q, so no N x F array exists
// (exterior_rhs_policy.jl restated, one pass for every column where the
// reference's matrix_free path integrates once per column).
template <typename T> struct RhsOut {
    Cx<T> *B = nullptr;             // N x F, row-major
    const Cx<double> *q = nullptr;  // F x R, column-major (matrix-free)
    Cx<double> *b = nullptr;        // N x R, column-major (matrix-free)
    int F = 0, N = 0, R = 0;
};

template <typename T>
__device__ __forceinline__ void rhs_add(const RhsOut<T> &o, int row, int face, T re, T im) {
    if (o.B) {
        red_add_cx(&o.B[(int64_t)row * o.F + face], re, im);
        return;
    }
    for (int r = 0; r < o.R; ++r) {
        const Cx<double> qq = o.q[(size_t)r * o.F + face];
        red_add_cx(&o.b[(size_t)r * o.N + row], (double)re * qq.re - (double)im * qq.im,
                   (double)re * qq.im + (double)im * qq.re);
    }
}

// columns of q per staged chunk in the matrix-free tile epilogues
constexpr int MF_RC = 8;

template <typename T> struct RegArgs {
    const T *qpts;      // by position: F x Q x 3
    const T *normal;    // F x 3
    const T *curl;      // F x 9
    const T *area;      // F
    const T *plane = nullptr;  // F: plane offset . normal (FP32; the FP64 kernel forms its own)
    const int *gvert;   // F x 3
    const int *face_id; // F
    const int *t_fstart, *t_vstart, *t_verts, *t_local;
    const int *t_inc = nullptr;  // per-tile vertex incidences (Tiling::incidence)
    Cx<T> *A;
    Cx<T> *B;
    int64_t ld;         // row stride of A (complex entries)
    int F;
    T k, eta, k2;
    // image pass: trial elements reflected by these signs (curls also by det),
    // touching pairs kept (their Duffy delta comes from image_delta_kernel)
    int image = 0;
    T xs[3] = {T(1), T(1), T(1)};
    T xdet = T(1);
    // matrix-free right-hand sides (B null): b (N x R) += B-tile x q (F x R)
    const Cx<double> *q = nullptr;
    Cx<double> *b = nullptr;
    int N = 0, R = 0;
};

// ---------------------------------------------------------------------------
// Symmetric element-pair kernel.  G(x, y) = G(y, x), so the two ordered pairs
// (tau, sigma) and (sigma, tau) of two elements share r, the phase, e^{ikr}/r
// and dG/dr at every point pair; only the normal derivatives swap roles: with
// r = y - x,
//   order 1 (test tau at x, trial sigma at y): dn_s =  r.n_sigma / r = a,
//                                               dn_t = -r.n_tau / r   = c,
//   order 2 (test sigma at y, trial tau at x): dn_s = c, dn_t = a.
// One CTA integrates an unordered pair of square tiles (I <= J; pairs of
// elements tau < sigma inside a diagonal tile) for both orders; each order
// has its own shared-memory accumulators, flushed once.
//
// Tiles: FP32 32 faces, two CTAs of 256 threads per SM (108 KB each).  FP64 16
// faces and two CTAs of 128 threads: the accumulators are twice as wide and a
// thread holds about 200 registers of sums, and one CTA of 32-face tiles (212
// KB) would leave the FP64 units idle while it zeroes, loads and flushes.
// Bound: issue (FP32), the FP64 units (FP64: about 85 FP64 instructions per
// unordered point pair, 34 ms at F = 20,480; one ordered pair at a time took
// 104.7 ms there, this 53.8).
// ---------------------------------------------------------------------------
// Accumulators.  A warp takes one tau and 32 sigma (FP64: two taus eight apart
// and 16 sigma), so the entries a lane adds to are keyed by sigma's vertex
// *slot* (s = b * F + sigma, the slot-face index) rather than by sigma's
// vertex: two lanes whose faces share a vertex would otherwise add to the same
// word in the same instruction, and shared-memory float atomics retry once per
// colliding lane.  The slot-face entries are folded onto tile J's vertices at
// the flush.
//   C1 [vI][s]      order 1, test vertex of tau x trial slot of sigma
//   C2 [s][vI]      order 2, test slot of sigma x trial vertex of tau
//   B1 [vI][sigma]  order 1 right-hand side (test vertex of tau x face sigma)
//   D2 [s][tau]     order 2 right-hand side (test slot of sigma x face tau)
// Re / im planes; a warp's lanes step 1 or an odd stride through each, so
// they spread over all banks.
template <typename T> struct SymTile {  // shapes as in context.cu
    static constexpr int F = sizeof(T) == 4 ? 32 : 16;        // faces
    static constexpr int V = sizeof(T) == 4 ? 40 : 32;        // distinct vertices
    static constexpr int THREADS = sizeof(T) == 4 ? 256 : 128;
    static constexpr int S = 3 * F;                            // slot-face indices
    static constexpr int C2S = V + 1, BS = F + 1;
    static constexpr int C1 = 0, C2 = C1 + V * S, B1 = C2 + S * C2S, D2 = B1 + V * BS;
    static constexpr int ACC = D2 + S * BS;                    // entries per plane
    static constexpr int INC = V + 1 + S;                      // Tiling::inc_stride()
    template <int Q> static size_t smem() {
        return sizeof(T) * (2 * ACC + 2 * F * (Q * 3 + 3 + 9 + 2)) + sizeof(int) * (3 * 3 * F + INC);
    }
};

// (re, im) sums: packed in FP32, two doubles in FP64
template <typename T> struct CxSum;
template <> struct CxSum<float> {
    F2 v = 0;
    __device__ __forceinline__ static F2 make(float re, float im) { return pk2(re, im); }
    __device__ __forceinline__ static F2 scaled(float a, F2 x) { return mul2(pk2(a, a), x); }
    __device__ __forceinline__ void add(int ri, int q, int b, F2 x) { v = fma2(rule_b2(ri, q, b), x, v); }
    __device__ __forceinline__ void get(float &re, float &im) const { up2(v, re, im); }
};
template <> struct CxSum<double> {
    Cx<double> v{0.0, 0.0};
    __device__ __forceinline__ static Cx<double> make(double re, double im) { return Cx<double>{re, im}; }
    __device__ __forceinline__ static Cx<double> scaled(double a, Cx<double> x) {
        return Cx<double>{a * x.re, a * x.im};
    }
    __device__ __forceinline__ void add(int ri, int q, int b, Cx<double> x) {
        v.re = fma(c_rb64[ri][q][b], x.re, v.re);
        v.im = fma(c_rb64[ri][q][b], x.im, v.im);
    }
    __device__ __forceinline__ void get(double &re, double &im) const {
        re = v.re;
        im = v.im;
    }
};
// sine and cosine of k r; kr = phase_scale(k) r is in revolutions (FP32) or radians (FP64)
__device__ __forceinline__ float phase_scale(float k) { return k * 0.15915494309189535f; }
__device__ __forceinline__ double phase_scale(double k) { return k; }
__device__ __forceinline__ void sincos_kr(float kr, float *s, float *c) { sincos_rev(kr, s, c); }
__device__ __forceinline__ void sincos_kr(double kr, double *s, double *c) { sincos_cw(kr, s, c); }

template <typename T, int Q>
__global__ void __launch_bounds__(SymTile<T>::THREADS, 2) sym_pairs_kernel(RegArgs<T> g) {
    using ST = SymTile<T>;
    constexpr int SYM_F = ST::F, SYM_S = ST::S, SYM_C2S = ST::C2S, SYM_BS = ST::BS, SYM_ACC = ST::ACC,
                  SYM_C1 = ST::C1, SYM_C2 = ST::C2, SYM_B1 = ST::B1, SYM_D2 = ST::D2, SYM_INC = ST::INC,
                  SYM_V = ST::V, THREADS = ST::THREADS;
    constexpr int RI = Q == 1 ? 0 : Q == 3 ? 1 : 2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *acc_re = reinterpret_cast<T *>(smem_raw), *acc_im = acc_re + SYM_ACC;
    T *xq = acc_im + SYM_ACC;                  // tile I: [tau][Q][3]
    T *xn = xq + SYM_F * Q * 3;                // [tau][3]
    T *xc = xn + SYM_F * 3;                    // [tau][9]
    T *xa = xc + SYM_F * 9;                    // [tau]
    T *xp = xa + SYM_F;                        // [tau]: plane offset x . n_tau
    T *yq = xp + SYM_F;                        // tile J, transposed: [Q * 3][sigma]
    T *yn = yq + SYM_F * Q * 3;                // [3][sigma]
    T *yc = yn + 3 * SYM_F;                    // [9][sigma]
    T *ya = yc + 9 * SYM_F;                    // [sigma]
    T *yp = ya + SYM_F;                        // [sigma]: plane offset y . n_sigma (a reflection keeps it)
    int *xgv = reinterpret_cast<int *>(yp + SYM_F);  // [tau][3] global vertex ids
    int *xlv = xgv + 3 * SYM_F;                      // [tau][3] tile-local vertex ids
    int *ygv = xlv + 3 * SYM_F;                      // [3][sigma]
    int *inc_start = ygv + 3 * SYM_F;                // [vJ + 1]: slot-face indices of tile J's vertex vJ
    int *inc_list = inc_start + SYM_V + 1;           //   are inc_list[inc_start[vJ] .. inc_start[vJ + 1])

    // unordered tile pair (I, J), I <= J, from the linear block index
    const int64_t bi = blockIdx.x;
    int J = (int)((sqrt(8.0 * (double)bi + 1.0) - 1.0) * 0.5);
    while ((int64_t)J * (J + 1) / 2 > bi) --J;
    while ((int64_t)(J + 1) * (J + 2) / 2 <= bi) ++J;
    const int I = (int)(bi - (int64_t)J * (J + 1) / 2);
    const bool diag = I == J;

    const int tid = threadIdx.x;
    const int t0 = g.t_fstart[I], nI = g.t_fstart[I + 1] - t0;
    const int s0 = g.t_fstart[J], nJ = g.t_fstart[J + 1] - s0;
    const int tv0 = g.t_vstart[I], nvI = g.t_vstart[I + 1] - tv0;
    const int sv0 = g.t_vstart[J], nvJ = g.t_vstart[J + 1] - sv0;

    static_assert(2 * SYM_ACC * sizeof(T) % 16 == 0, "accumulators are zeroed as float4");
    for (int i = tid; i < (int)(2 * SYM_ACC * sizeof(T) / 16); i += THREADS)
        reinterpret_cast<float4 *>(acc_re)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    // the tile arrays: every copy in flight at once, one wait
    for (int i = tid; i < nI * Q * 3; i += THREADS) cp_async_el(&xq[i], &g.qpts[(size_t)t0 * Q * 3 + i]);
    for (int i = tid; i < nI * 3; i += THREADS) {
        cp_async_el(&xn[i], &g.normal[(size_t)t0 * 3 + i]);
        cp_async_el(&xgv[i], &g.gvert[(size_t)t0 * 3 + i]);
        cp_async_el(&xlv[i], &g.t_local[(size_t)t0 * 3 + i]);
    }
    for (int i = tid; i < nI * 9; i += THREADS) cp_async_el(&xc[i], &g.curl[(size_t)t0 * 9 + i]);
    for (int i = tid; i < nI; i += THREADS) {
        cp_async_el(&xa[i], &g.area[t0 + i]);
        if (sizeof(T) == 4) cp_async_el(&xp[i], &g.plane[t0 + i]);
    }
    for (int i = tid; i < nJ * Q * 3; i += THREADS) {
        const int s = i / (Q * 3), j = i % (Q * 3);
        cp_async_el(&yq[j * SYM_F + s], &g.qpts[(size_t)s0 * Q * 3 + i]);
    }
    for (int i = tid; i < nJ * 3; i += THREADS) {
        const int s = i / 3, j = i % 3;
        cp_async_el(&yn[j * SYM_F + s], &g.normal[(size_t)s0 * 3 + i]);
        cp_async_el(&ygv[j * SYM_F + s], &g.gvert[(size_t)s0 * 3 + i]);
    }
    for (int i = tid; i < nJ * 9; i += THREADS) {
        const int s = i / 9, j = i % 9;
        cp_async_el(&yc[j * SYM_F + s], &g.curl[(size_t)s0 * 9 + i]);
    }
    for (int i = tid; i < nJ; i += THREADS) {
        cp_async_el(&ya[i], &g.area[s0 + i]);
        if (sizeof(T) == 4) cp_async_el(&yp[i], &g.plane[s0 + i]);
    }
    for (int i = tid; i < SYM_INC; i += THREADS) cp_async_el(&inc_start[i], &g.t_inc[(size_t)J * SYM_INC + i]);
    cp_async_wait_all();
    __syncthreads();
    if (sizeof(T) == 8) {  // every point y of a flat face has the same y . n
        for (int i = tid; i < nI + nJ; i += THREADS) {
            if (i < nI)
                xp[i] = xq[i * Q * 3] * xn[3 * i] + xq[i * Q * 3 + 1] * xn[3 * i + 1] + xq[i * Q * 3 + 2] * xn[3 * i + 2];
            else
                yp[i - nI] = yq[i - nI] * yn[i - nI] + yq[SYM_F + i - nI] * yn[SYM_F + i - nI] +
                             yq[2 * SYM_F + i - nI] * yn[2 * SYM_F + i - nI];
        }
        __syncthreads();
    }
    if (g.image) {
        // an image pass reflects tile J: pairs (tau, S sigma) and (sigma, S tau)
        // have the same distances, |x - Sy| = |Sx - y|, and swap dn_s / dn_t
        for (int i = tid; i < nJ * Q * 3; i += THREADS) {
            const int s = i / (Q * 3), j = i % (Q * 3);
            yq[j * SYM_F + s] *= g.xs[j % 3];
        }
        for (int i = tid; i < nJ * 3; i += THREADS) {
            const int s = i / 3, j = i % 3;
            yn[j * SYM_F + s] *= g.xs[j];
        }
        for (int i = tid; i < nJ * 9; i += THREADS) {
            const int s = i / 9, j = i % 9;
            yc[j * SYM_F + s] *= g.xdet * g.xs[j % 3];
        }
        __syncthreads();
    }

    const T k = g.k, eta = g.eta;
    const T kr = phase_scale(k);
    const T inv4pi = T(0.07957747154594767);  // 1 / (4 pi)
    for (int p = tid; p < SYM_F * SYM_F; p += THREADS) {
        // a warp: one tau (two, half a tile apart), every sigma
        const int ti = SYM_F == 32 ? p / 32 : p / 32 + (p >> 4 & 1) * 8, sj = p % SYM_F;
        // (an image pass keeps tau == sigma: the element and its own image,
        // whose two orders coincide and are taken at half weight)
        if (ti >= nI || sj >= nJ || (diag && (g.image ? sj < ti : sj <= ti))) continue;
        const int ga = xgv[3 * ti], gb = xgv[3 * ti + 1], gc = xgv[3 * ti + 2];
        const int ha = ygv[sj], hb = ygv[SYM_F + sj], hc = ygv[2 * SYM_F + sj];
        if (!g.image && (ga == ha || ga == hb || ga == hc || gb == ha || gb == hb || gb == hc || gc == ha ||
                         gc == hb || gc == hc))
            continue;  // touching pair: the Duffy kernel integrates both orders
        const T ntx = xn[3 * ti], nty = xn[3 * ti + 1], ntz = xn[3 * ti + 2];
        const T nsx = yn[sj], nsy = yn[SYM_F + sj], nsz = yn[2 * SYM_F + sj];
        const T k2n = eta * g.k2 * (ntx * nsx + nty * nsy + ntz * nsz);
        const T dtau = xp[ti], dsig = yp[sj];
        // r . n_tau = y . n_tau - x . n_tau is the same for every test point x
        // on the flat face tau: one value per trial point
        T ync[Q];
#pragma unroll
        for (int qs = 0; qs < Q; ++qs)
            ync[qs] = yq[(qs * 3) * SYM_F + sj] * ntx + yq[(qs * 3 + 1) * SYM_F + sj] * nty +
                      yq[(qs * 3 + 2) * SYM_F + sj] * ntz - dtau;
        // L1 / L2: the two orders' 3 x 3 blocks; R1: order 1's right-hand-side
        // 3-vector; TC_b: sum over both faces' points of w phi_b(y) G, which
        // gives the Green sum of the curl term and order 2's right-hand side
        T L1[9][2], L2[9][2], R1[3][2], TC[3][2];
#pragma unroll
        for (int i = 0; i < 9; ++i) L1[i][0] = L1[i][1] = L2[i][0] = L2[i][1] = T(0);
#pragma unroll
        for (int i = 0; i < 3; ++i) R1[i][0] = R1[i][1] = TC[i][0] = TC[i][1] = T(0);
#pragma unroll 1
        for (int qt = 0; qt < Q; ++qt) {
            const T x0 = xq[(ti * Q + qt) * 3], x1 = xq[(ti * Q + qt) * 3 + 1], x2 = xq[(ti * Q + qt) * 3 + 2];
            const T wt = RuleRef<T>::w(RI, qt) * inv4pi;
            const T xns = dsig - (x0 * nsx + x1 * nsy + x2 * nsz);  // r . n_sigma for every y on sigma
            // Per trial point (the test point's weight wt applied below):
            //   g = w_s exp(ikr) / r,  h = g (ik - 1/r) / r  (dG/dr / r),
            //   C_b += phi_b(y) g,  H_b += phi_b(y) h,  P_b += phi_b(y) (r . n_tau) h.
            // Order 1's kernel value -g' (r . n_sigma) / r - i k2n g sums to
            // -xns H_b - i k2n C_b, order 2's (r . n_tau) g' / r - i k2n g to
            // P_b - i k2n C_b; each sum a packed (re, im) pair.
            CxSum<T> Cs[3], Hs[3], Ps[3];
#pragma unroll
            for (int qs = 0; qs < Q; ++qs) {
                const T rx = yq[(qs * 3) * SYM_F + sj] - x0, ry = yq[(qs * 3 + 1) * SYM_F + sj] - x1,
                        rz = yq[(qs * 3 + 2) * SYM_F + sj] - x2;
                const T r2 = rx * rx + ry * ry + rz * rz;
                const T ir = rsqrt_t(r2);
                T sn_, cs_;
                sincos_kr(kr * (r2 * ir), &sn_, &cs_);
                const T scl = ir * RuleRef<T>::w(RI, qs);
                const T gr = cs_ * scl, gi = sn_ * scl;
                const T hr = (-gr * ir - gi * k) * ir;
                const T hi = (gr * k - gi * ir) * ir;
                const auto g2 = CxSum<T>::make(gr, gi), h2 = CxSum<T>::make(hr, hi);
#pragma unroll
                for (int b = 0; b < 3; ++b) Cs[b].add(RI, qs, b, g2);
#pragma unroll
                for (int b = 0; b < 3; ++b) Hs[b].add(RI, qs, b, h2);
                const auto p2 = CxSum<T>::scaled(ync[qs], h2);
#pragma unroll
                for (int b = 0; b < 3; ++b) Ps[b].add(RI, qs, b, p2);
            }
            T Cr[3], Ci[3], Hr[3], Hi[3], Pr[3], Pi[3];
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                Cs[b].get(Cr[b], Ci[b]);
                Hs[b].get(Hr[b], Hi[b]);
                Ps[b].get(Pr[b], Pi[b]);
            }
            // order 1's right-hand-side value -G + i eta W, W = sum (r . n_tau) g' / r
            const T Gr = Cr[0] + Cr[1] + Cr[2], Gi = Ci[0] + Ci[1] + Ci[2];
            const T Wr = Pr[0] + Pr[1] + Pr[2], Wi = Pi[0] + Pi[1] + Pi[2];
            const T Ur = -Gr - eta * Wi, Ui = -Gi + eta * Wr;
            T Sr[3], Si[3];
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                Sr[b] = -xns * Hr[b] + k2n * Ci[b];
                Si[b] = -xns * Hi[b] - k2n * Cr[b];
                Pr[b] += k2n * Ci[b];
                Pi[b] -= k2n * Cr[b];
                TC[b][0] += wt * Cr[b];
                TC[b][1] += wt * Ci[b];
            }
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const T ba = RuleRef<T>::b(RI, qt, a) * wt;
#pragma unroll
                for (int b = 0; b < 3; ++b) {
                    L1[3 * a + b][0] += ba * Sr[b];
                    L1[3 * a + b][1] += ba * Si[b];
                    // order 2: row = test vertex of sigma (b), column = trial vertex of tau (a)
                    L2[3 * b + a][0] += ba * Pr[b];
                    L2[3 * b + a][1] += ba * Pi[b];
                }
                R1[a][0] += ba * Ur;
                R1[a][1] += ba * Ui;
            }
        }
        // Order 2's right-hand-side value at (x, y) is -(1 + eta k2n) g + i eta
        // times order 1's kernel value, so its sum against phi_b(y) is
        // -(1 + eta k2n) TC_b + i eta sum_a L1[a][b] (the test basis sums to 1).
        const T cr = TC[0][0] + TC[1][0] + TC[2][0], ci = TC[0][1] + TC[1][1] + TC[2][1];
        const T ce = -(T(1) + eta * k2n);
        T R2[3][2];
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            const T lr = L1[b][0] + L1[3 + b][0] + L1[6 + b][0], li = L1[b][1] + L1[3 + b][1] + L1[6 + b][1];
            R2[b][0] = ce * TC[b][0] - eta * li;
            R2[b][1] = ce * TC[b][1] + eta * lr;
        }
        // hypersingular curl term: eta * sum(g w) * curl_test . curl_trial (same sum for both orders)
        const T ccr = -eta * ci, cci = eta * cr;
        const T jac = T(4) * xa[ti] * ya[sj] * ((g.image && diag && sj == ti) ? T(0.5) : T(1));
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const int ra = xlv[3 * ti + a];  // vertex a of tau, tile I local
            int off[14];  // this vertex's 14 adds (re and im planes)
            T val[14];
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                const T d = xc[9 * ti + 3 * a] * yc[(3 * b) * SYM_F + sj] +
                            xc[9 * ti + 3 * a + 1] * yc[(3 * b + 1) * SYM_F + sj] +
                            xc[9 * ti + 3 * a + 2] * yc[(3 * b + 2) * SYM_F + sj];  // curl_tau[a] . curl_sigma[b]
                const int o1 = SYM_C1 + ra * SYM_S + b * SYM_F + sj;
                off[4 * b] = o1;
                val[4 * b] = (L1[3 * a + b][0] + d * ccr) * jac;
                off[4 * b + 1] = o1 + SYM_ACC;
                val[4 * b + 1] = (L1[3 * a + b][1] + d * cci) * jac;
                // order 2 entry (sigma vertex b, tau vertex a) uses curl_sigma[b] . curl_tau[a] = d
                const int o2 = SYM_C2 + (b * SYM_F + sj) * SYM_C2S + ra;
                off[4 * b + 2] = o2;
                val[4 * b + 2] = (L2[3 * b + a][0] + d * ccr) * jac;
                off[4 * b + 3] = o2 + SYM_ACC;
                val[4 * b + 3] = (L2[3 * b + a][1] + d * cci) * jac;
            }
            off[12] = SYM_B1 + ra * SYM_BS + sj;
            val[12] = R1[a][0] * jac;
            off[13] = off[12] + SYM_ACC;
            val[13] = R1[a][1] * jac;
            // tau's other elements in flight on other warps may share vertex a
            batch_add<14>(acc_re, off, val);
            // (sigma slot a, face tau) belongs to this element pair alone: a plain store
            const int e2 = SYM_D2 + (a * SYM_F + sj) * SYM_BS + ti;
            acc_re[e2] = R2[a][0] * jac;
            acc_im[e2] = R2[a][1] * jac;
        }
    }
    __syncthreads();
    // fold the slot-face entries onto tile J's vertices and flush
    for (int i = tid; i < nvI * nvJ; i += THREADS) {
        const int li = i / nvJ, lj = i % nvJ;
        Cx<T> v{T(0), T(0)}, u{T(0), T(0)};
        for (int e = inc_start[lj]; e < inc_start[lj + 1]; ++e) {
            const int s = inc_list[e];
            v.re += acc_re[SYM_C1 + li * SYM_S + s];
            v.im += acc_im[SYM_C1 + li * SYM_S + s];
            u.re += acc_re[SYM_C2 + s * SYM_C2S + li];
            u.im += acc_im[SYM_C2 + s * SYM_C2S + li];
        }
        const int gi_ = g.t_verts[tv0 + li], gj_ = g.t_verts[sv0 + lj];
        if (v.re != T(0) || v.im != T(0)) red_add_cx(&g.A[(int64_t)gi_ * g.ld + gj_], v.re, v.im);
        if (u.re != T(0) || u.im != T(0)) red_add_cx(&g.A[(int64_t)gj_ * g.ld + gi_], u.re, u.im);
    }
    if (g.B) {
        for (int i = tid; i < nvI * nJ; i += THREADS) {
            const int li = i / nJ, sj = i % nJ;
            const Cx<T> v{acc_re[SYM_B1 + li * SYM_BS + sj], acc_im[SYM_B1 + li * SYM_BS + sj]};
            if (v.re != T(0) || v.im != T(0))
                red_add_cx(&g.B[(int64_t)g.t_verts[tv0 + li] * g.F + g.face_id[s0 + sj]], v.re, v.im);
        }
        for (int i = tid; i < nvJ * nI; i += THREADS) {
            const int lj = i / nI, ti = i % nI;
            Cx<T> v{T(0), T(0)};
            for (int e = inc_start[lj]; e < inc_start[lj + 1]; ++e) {
                const int s = inc_list[e];
                v.re += acc_re[SYM_D2 + s * SYM_BS + ti];
                v.im += acc_im[SYM_D2 + s * SYM_BS + ti];
            }
            if (v.re != T(0) || v.im != T(0))
                red_add_cx(&g.B[(int64_t)g.t_verts[sv0 + lj] * g.F + g.face_id[t0 + ti]], v.re, v.im);
        }
        return;
    }
    // matrix-free: rows of b += B1 q (tile I vertices x tile J faces) and
    // B2 q (tile J vertices x tile I faces); q of both tiles' faces staged
    // MF_RC columns at a time over the (now unused) geometry region
    Cx<T> *qs = reinterpret_cast<Cx<T> *>(xq);  // [2][SYM_F][MF_RC]: tile I faces, then tile J faces
    // order 2 rows folded onto tile J's vertices, over the (read) C1 block
    constexpr int B2V = SYM_C1;  // [vJ][tau]
    __syncthreads();
    for (int i = tid; i < nvJ * nI; i += THREADS) {
        const int lj = i / nI, ti = i % nI;
        T vr = T(0), vi = T(0);
        for (int e = inc_start[lj]; e < inc_start[lj + 1]; ++e) {
            vr += acc_re[SYM_D2 + inc_list[e] * SYM_BS + ti];
            vi += acc_im[SYM_D2 + inc_list[e] * SYM_BS + ti];
        }
        acc_re[B2V + lj * SYM_BS + ti] = vr;
        acc_im[B2V + lj * SYM_BS + ti] = vi;
    }
    for (int r0 = 0; r0 < g.R; r0 += MF_RC) {
        const int rc = min(MF_RC, g.R - r0);
        __syncthreads();
        for (int i = tid; i < 2 * SYM_F * MF_RC; i += THREADS) {
            const int h = i / (SYM_F * MF_RC), f = (i / MF_RC) % SYM_F, r = i % MF_RC;
            Cx<T> v{T(0), T(0)};
            if (f < (h ? nJ : nI) && r < rc) {
                const Cx<double> qq = g.q[(size_t)(r0 + r) * g.F + g.face_id[(h ? s0 : t0) + f]];
                v = Cx<T>{(T)qq.re, (T)qq.im};
            }
            qs[i] = v;
        }
        __syncthreads();
        for (int i = tid; i < (nvI + nvJ) * rc; i += THREADS) {
            const int row = i / rc, r = i % rc;
            const bool first = row < nvI;
            const int base = first ? SYM_B1 + row * SYM_BS : B2V + (row - nvI) * SYM_BS;
            const int nf = first ? nJ : nI;
            const Cx<T> *qh = qs + (first ? SYM_F * MF_RC : 0);
            T sr = T(0), si = T(0);
            for (int f = 0; f < nf; ++f) {
                const T br = acc_re[base + f], bi = acc_im[base + f];
                const Cx<T> qv = qh[f * MF_RC + r];
                sr += br * qv.re - bi * qv.im;
                si += br * qv.im + bi * qv.re;
            }
            const int gv = first ? g.t_verts[tv0 + row] : g.t_verts[sv0 + row - nvI];
            if (sr != T(0) || si != T(0)) red_add_cx(&g.b[(size_t)(r0 + r) * g.N + gv], (double)sr, (double)si);
        }
    }
}

// ---------------------------------------------------------------------------
// Touching pairs: one warp per pair, FP64, Duffy points over the lanes.
//
// With x = x0 + xi e1 + eta e2 on the test face and y = y0 + xi' f1 + eta' f2 on
// the trial face, every basis product is a combination of 1, xi, eta times 1,
// xi', eta'; so a point adds the kernel value times those nine monomials, and
// the nine basis products follow once per pair.  r = y - x is formed from the
// two points' own offsets, so that exchanging them in a face's pair with itself
// only changes its sign, and r . n from r: a rounding error common to all points
// (of n . e1, say, where r . n should vanish) would be weighted by 1 / r^3
// (right-hand sides at F = 320: 5.0e-15 with r . n from such constants, 3.8e-16).
// The rule's points are stored coordinate by coordinate (coalesced), and the 26
// sums are reduced over the lanes by halving: each exchange step also halves
// the number of sums a lane carries.
// Bound: the FP64 units, about 105 instructions per point (1.2 ms at F =
// 20,480, 2.22 measured; 2.23 with nine products and 26 butterfly sums a point).
// ---------------------------------------------------------------------------
template <typename T> struct SingArgs {
    const int *test, *trial, *rule;
    const double *jac, *nn;
    const int *rule_start;
    const double *rule_data;  // five arrays of npoints: xi, eta, xi', eta', weight
    int64_t npoints;
    const double *verts;      // V x 3
    const int *faces;         // F x 3
    const double *normals;    // F x 3
    const double *curls;      // F x 9
    Cx<T> *A;
    RhsOut<T> rhs;
    int64_t ld;
    int64_t npairs;
    double k, eta;
};

// Sums of v[0..31] over the lanes: lane l returns the total of v[l].  Step o
// hands half of the remaining sums to the lane o away and keeps the others.
__device__ __forceinline__ double warp_sum32(double (&v)[32]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < o; ++i) {
            const double send = up ? v[i] : v[i + o], keep = up ? v[i + o] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    return v[0];
}

// the same kernel value's sums against 1, xi', eta', xi, ... in acc[2 (3 i + j)]
// (i: test monomial 1, xi, eta; j: trial), acc[18 + 2 i]: right-hand-side value
// against the test monomials, acc[24]: Green sum
__device__ __forceinline__ void singular_point(double xi, double et, double yi, double ye, const double (&d0)[3],
                                               const double (&e1)[3], const double (&e2)[3], const double (&f1)[3],
                                               const double (&f2)[3], const double (&ns)[3], const double (&nt)[3],
                                               double w, double k, double eta, double k2n, double (&acc)[32]) {
    double r[3];
#pragma unroll
    for (int c = 0; c < 3; ++c)
        r[c] = fma(yi, f1[c], fma(ye, f2[c], d0[c])) - fma(xi, e1[c], et * e2[c]);
    const double r2 = r[0] * r[0] + r[1] * r[1] + r[2] * r[2];
    if (r2 == 0.0) return;
    const double ir = rsqrt_series(r2);
    double sn_, cs_;
    sincos_cw(k * (r2 * ir), &sn_, &cs_);
    const double scl = ir * w;
    const double gr = cs_ * scl, gi = sn_ * scl;
    const double hr = (-gr * ir - gi * k) * ir, hi = (gr * k - gi * ir) * ir;  // dG/dr / r
    const double rns = fma(r[0], ns[0], fma(r[1], ns[1], r[2] * ns[2]));
    const double rnt = fma(r[0], nt[0], fma(r[1], nt[1], r[2] * nt[2]));
    const double lr = k2n * gi - hr * rns, li = -(hi * rns + k2n * gr);
    const double pt = eta * rnt;
    const double rr = -gr - hi * pt, ri = hr * pt - gi;
    const double m[4] = {xi * yi, xi * ye, et * yi, et * ye};
    acc[0] += lr;
    acc[1] += li;
    acc[2] = fma(yi, lr, acc[2]);
    acc[3] = fma(yi, li, acc[3]);
    acc[4] = fma(ye, lr, acc[4]);
    acc[5] = fma(ye, li, acc[5]);
    acc[6] = fma(xi, lr, acc[6]);
    acc[7] = fma(xi, li, acc[7]);
    acc[8] = fma(m[0], lr, acc[8]);
    acc[9] = fma(m[0], li, acc[9]);
    acc[10] = fma(m[1], lr, acc[10]);
    acc[11] = fma(m[1], li, acc[11]);
    acc[12] = fma(et, lr, acc[12]);
    acc[13] = fma(et, li, acc[13]);
    acc[14] = fma(m[2], lr, acc[14]);
    acc[15] = fma(m[2], li, acc[15]);
    acc[16] = fma(m[3], lr, acc[16]);
    acc[17] = fma(m[3], li, acc[17]);
    acc[18] += rr;
    acc[19] += ri;
    acc[20] = fma(xi, rr, acc[20]);
    acc[21] = fma(xi, ri, acc[21]);
    acc[22] = fma(et, rr, acc[22]);
    acc[23] = fma(et, ri, acc[23]);
    acc[24] += gr;
    acc[25] += gi;
}

template <typename T>
__global__ void __launch_bounds__(256, 2) singular_pairs_kernel(SingArgs<T> g) {
    const int lane = threadIdx.x & 31;
    const int64_t pair = (int64_t)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
    if (pair >= g.npairs) return;
    const int t = g.test[pair], s = g.trial[pair], r = g.rule[pair];
    const int *ft = g.faces + 3 * t, *fs = g.faces + 3 * s;
    double d0[3], e1[3], e2[3], f1[3], f2[3], ns[3], nt[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const double x0 = g.verts[3 * ft[0] + c], y0 = g.verts[3 * fs[0] + c];
        e1[c] = g.verts[3 * ft[1] + c] - x0;
        e2[c] = g.verts[3 * ft[2] + c] - x0;
        f1[c] = g.verts[3 * fs[1] + c] - y0;
        f2[c] = g.verts[3 * fs[2] + c] - y0;
        d0[c] = y0 - x0;
        ns[c] = g.normals[3 * s + c];
        nt[c] = g.normals[3 * t + c];
    }
    const double k = g.k, eta = g.eta;
    const double k2n = eta * (k * k * g.nn[pair]);
    double acc[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) acc[i] = 0.0;
    const int q1 = g.rule_start[r + 1];
    const double *rd = g.rule_data;
    const int64_t np = g.npoints;
    for (int q = g.rule_start[r] + lane; q < q1; q += 32)
        singular_point(rd[q], rd[np + q], rd[2 * np + q], rd[3 * np + q], d0, e1, e2, f1, f2, ns, nt,
                       0.07957747154594767 * rd[4 * np + q], k, eta, k2n, acc);
    const double mine = warp_sum32(acc);  // lane i: sum i
    // the basis products: phi_0 = 1 - phi_1 - phi_2 on either face
    const double jac = g.jac[pair];
    auto sum = [&](int i) { return __shfl_sync(0xffffffffu, mine, i); };
    const double cr = sum(24), ci = sum(25);
    const int a = lane / 3, b = lane % 3;  // lanes 0..8: entry (a, b); lanes 9..11: right-hand side a = lane - 9
    // monomial sums M[i][j]: entry = sum_i,j ca(a, i) cb(b, j) M[i][j], c(0, .) = (1, -1, -1), c(1, .) = (0, 1, 0), ...
    double vr = 0.0, vi = 0.0;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const int row = lane < 9 ? a : lane - 9;
        const double ca = row == 0 ? (i == 0 ? 1.0 : -1.0) : (row == i ? 1.0 : 0.0);
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const double cb = b == 0 ? (j == 0 ? 1.0 : -1.0) : (b == j ? 1.0 : 0.0);
            const double mr = sum(2 * (3 * i + j)), mi = sum(2 * (3 * i + j) + 1);
            if (lane < 9) {
                vr = fma(ca * cb, mr, vr);
                vi = fma(ca * cb, mi, vi);
            }
        }
        const double qr = sum(18 + 2 * i), qi = sum(18 + 2 * i + 1);
        if (lane >= 9) {
            vr = fma(ca, qr, vr);
            vi = fma(ca, qi, vi);
        }
    }
    if (lane < 9) {
        const double ccr = -eta * ci, cci = eta * cr;
        const double *cta = g.curls + 9 * t + 3 * a, *csb = g.curls + 9 * s + 3 * b;
        const double d = cta[0] * csb[0] + cta[1] * csb[1] + cta[2] * csb[2];
        red_add_cx(&g.A[(int64_t)ft[a] * g.ld + fs[b]], (T)((vr + d * ccr) * jac), (T)((vi + d * cci) * jac));
    } else if (lane < 12) {
        rhs_add(g.rhs, ft[lane - 9], s, (T)(vr * jac), (T)(vi * jac));
    }
}

// ---------------------------------------------------------------------------
// touching image pairs (test t, trial s reflected by image x): the remapped
// Duffy integral minus the regular-rule integral the image pass added
// (_cuda_image_singular_delta_blocks_kernel!, BeatEngineCudaSingular.jl:590-897).
// One warp per pair, FP64, lanes over the Duffy points, then over the Q x Q
// regular points.
// ---------------------------------------------------------------------------
struct ImgXf {
    double s[3][3];  // per image: signs
    double det[3];
};

template <typename T> struct ImgArgs {
    const int *test, *trial, *rule, *img;
    const double *jac, *nn;
    const int *rule_start;
    const double *rule_data;  // five arrays of npoints
    int64_t npoints;
    const double *verts;
    const int *faces;
    const double *normals, *curls;
    int Q, RI;
    Cx<T> *A;
    RhsOut<T> rhs;
    int64_t ld;
    int64_t npairs;
    double k, eta;
    ImgXf xf;
};

__device__ __forceinline__ void bm_point_d(const double *x, const double *y, const double *bt, const double *bs,
                                           double w, const double *nt, const double *ns, double k, double eta,
                                           double k2n, double sign, double *acc) {
    const double rx = y[0] - x[0], ry = y[1] - x[1], rz = y[2] - x[2];
    const double r2 = rx * rx + ry * ry + rz * rz;
    if (r2 == 0.0) return;
    const double ir = rsqrt(r2), rad = r2 * ir;
    double sn_, cs_;
    sincos_cw(k * rad, &sn_, &cs_);
    const double scl = sign * ir * (0.07957747154594767 * w);
    const double gr = cs_ * scl, gi = sn_ * scl;
    const double gsr = -gr * ir - gi * k, gsi = gr * k - gi * ir;
    const double dns = (rx * ns[0] + ry * ns[1] + rz * ns[2]) * ir;
    const double dnt = -(rx * nt[0] + ry * nt[1] + rz * nt[2]) * ir;
    const double lr = -gsr * dns + k2n * gi, li = -gsi * dns - k2n * gr;
    const double rr = -gr + eta * (gsi * dnt), ri = -gi - eta * (gsr * dnt);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            const double bp = bt[a] * bs[b];
            acc[2 * (3 * a + b)] += bp * lr;
            acc[2 * (3 * a + b) + 1] += bp * li;
        }
        acc[18 + 2 * a] += bt[a] * rr;
        acc[18 + 2 * a + 1] += bt[a] * ri;
    }
    acc[24] += gr;
    acc[25] += gi;
}

template <typename T>
__global__ void __launch_bounds__(256, 2) image_delta_kernel(ImgArgs<T> g) {
    const int lane = threadIdx.x & 31;
    const int64_t pair = (int64_t)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
    if (pair >= g.npairs) return;
    const int t = g.test[pair], s = g.trial[pair], r = g.rule[pair], ix = g.img[pair];
    const double *sg = g.xf.s[ix];
    const int *ft = g.faces + 3 * t, *fs = g.faces + 3 * s;
    double tv[3][3], sv[3][3], nt[3], ns[3];
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            tv[a][c] = g.verts[3 * ft[a] + c];
            sv[a][c] = sg[c] * g.verts[3 * fs[a] + c];
        }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        nt[c] = g.normals[3 * t + c];
        ns[c] = sg[c] * g.normals[3 * s + c];
    }
    const double k = g.k, eta = g.eta;
    const double k2n = eta * (k * k * g.nn[pair]);
    double acc[26];
#pragma unroll
    for (int i = 0; i < 26; ++i) acc[i] = 0.0;
    // + Duffy
    for (int q = g.rule_start[r] + lane; q < g.rule_start[r + 1]; q += 32) {
        double d[5];
#pragma unroll
        for (int c = 0; c < 5; ++c) d[c] = g.rule_data[c * g.npoints + q];
        const double bt[3] = {1.0 - d[0] - d[1], d[0], d[1]}, bs[3] = {1.0 - d[2] - d[3], d[2], d[3]};
        double x[3], y[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            x[c] = bt[0] * tv[0][c] + bt[1] * tv[1][c] + bt[2] * tv[2][c];
            y[c] = bs[0] * sv[0][c] + bs[1] * sv[1][c] + bs[2] * sv[2][c];
        }
        bm_point_d(x, y, bt, bs, d[4], nt, ns, k, eta, k2n, 1.0, acc);
    }
    // - regular rule
    for (int pq = lane; pq < g.Q * g.Q; pq += 32) {
        const int qt = pq / g.Q, qs = pq % g.Q;
        const double bt[3] = {c_rb64[g.RI][qt][0], c_rb64[g.RI][qt][1], c_rb64[g.RI][qt][2]};
        const double bs[3] = {c_rb64[g.RI][qs][0], c_rb64[g.RI][qs][1], c_rb64[g.RI][qs][2]};
        double x[3], y[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            x[c] = bt[0] * tv[0][c] + bt[1] * tv[1][c] + bt[2] * tv[2][c];
            y[c] = bs[0] * sv[0][c] + bs[1] * sv[1][c] + bs[2] * sv[2][c];
        }
        bm_point_d(x, y, bt, bs, c_rw64[g.RI][qt] * c_rw64[g.RI][qs], nt, ns, k, eta, k2n, -1.0, acc);
    }
#pragma unroll
    for (int i = 0; i < 26; ++i) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], o);
    }
    const double jac = g.jac[pair];
    const double ccr = -eta * acc[25], cci = eta * acc[24];
    const double cdet = g.xf.det[ix];
    if (lane < 9) {
        const int a = lane / 3, b = lane % 3;
        const double *cta = g.curls + 9 * t + 3 * a, *csb = g.curls + 9 * s + 3 * b;
        const double d = cdet * (cta[0] * sg[0] * csb[0] + cta[1] * sg[1] * csb[1] + cta[2] * sg[2] * csb[2]);
        double vr = 0, vi = 0;
#pragma unroll
        for (int i = 0; i < 9; ++i)
            if (i == lane) {
                vr = acc[2 * i];
                vi = acc[2 * i + 1];
            }
        red_add_cx(&g.A[(int64_t)ft[a] * g.ld + fs[b]], (T)((vr + d * ccr) * jac), (T)((vi + d * cci) * jac));
    } else if (lane < 12) {
        const int a = lane - 9;
        double vr = 0, vi = 0;
#pragma unroll
        for (int i = 0; i < 3; ++i)
            if (i == a) {
                vr = acc[18 + 2 * i];
                vi = acc[18 + 2 * i + 1];
            }
        rhs_add(g.rhs, ft[a], s, (T)(vr * jac), (T)(vi * jac));
    }
}

// orbit row weights (p1_symmetry_orbit_weights, BeatEngineCore.jl:563-582):
// the rows of A and B of vertices on a symmetry plane, times 2 per plane
// (the rows of b instead of B in the matrix-free mode: b = B q is linear in B)
template <typename T>
__global__ void row_weight_kernel(const int *verts, const double *weights, int nw, Cx<T> *A, int64_t ld, int n,
                                  RhsOut<T> rhs) {
    const int v = blockIdx.y;
    if (v >= nw) return;
    const int row = verts[v];
    const double w = weights[v];
    const int cols = rhs.B ? rhs.F : rhs.R;
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n + cols; j += gridDim.x * blockDim.x) {
        if (j < n || rhs.B) {
            Cx<T> &e = j < n ? A[(int64_t)row * ld + j] : rhs.B[(int64_t)row * rhs.F + (j - n)];
            e.re *= (T)w;
            e.im *= (T)w;
        } else {
            Cx<double> &e = rhs.b[(size_t)(j - n) * rhs.N + row];
            e.re *= w;
            e.im *= w;
        }
    }
}

// ---------------------------------------------------------------------------
// identity terms: A += 0.5 M_p1p1, B += -0.5 eta M_p1dp0
// ---------------------------------------------------------------------------
template <typename T>
__global__ void identity_kernel(const int *faces, const double *areas, int F, int Q, double eta, Cx<T> *A,
                                int64_t ld, RhsOut<T> rhs) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= F) return;
    const int ri = Q == 1 ? 0 : Q == 3 ? 1 : 2;
    const double jac = 2.0 * areas[f];
    double blk[9] = {0}, col[3] = {0};
    for (int q = 0; q < Q; ++q) {
        const double w = c_rw64[ri][q];
        for (int a = 0; a < 3; ++a) {
            const double pa = c_rb64[ri][q][a];
            col[a] += pa * w * jac;
            for (int b = 0; b < 3; ++b) blk[3 * a + b] += pa * c_rb64[ri][q][b] * w * jac;
        }
    }
    const int *fc = faces + 3 * f;
    for (int a = 0; a < 3; ++a) {
        for (int b = 0; b < 3; ++b) red_add(&A[(int64_t)fc[a] * ld + fc[b]].re, (T)(0.5 * blk[3 * a + b]));
        rhs_add(rhs, fc[a], f, T(0), (T)(-0.5 * eta * col[a]));
    }
}

// ---------------------------------------------------------------------------
// host driver
// ---------------------------------------------------------------------------
template <typename T> static RhsOut<T> rhs_out(beat_b200_ctx *c, int R, const Cx<double> *q) {
    RhsOut<T> o;
    o.B = c->ws.rhs_cached ? c->ws.B.as<Cx<T>>() : nullptr;
    o.q = q;
    o.b = c->ws.b.as<Cx<double>>();
    o.F = c->F;
    o.N = c->V;
    o.R = R;
    return o;
}

// the symmetric kernel over unordered pairs of square tiles
template <typename T, int Q>
static void launch_sym(beat_b200_ctx *c, double k, double eta, int img, int R, const Cx<double> *q) {
    constexpr bool d = sizeof(T) == 8;
    const Tiling &tiles = d ? c->trial_tiles : c->sym_tiles;
    RegArgs<T> g;
    g.qpts = (const T *)(d ? c->pos_qpts64.p : c->pos_qpts32.p);
    g.normal = (const T *)(d ? c->pos_normal64.p : c->pos_normal32.p);
    g.curl = (const T *)(d ? c->pos_curl64.p : c->pos_curl32.p);
    g.area = (const T *)(d ? c->pos_area64.p : c->pos_area32.p);
    g.plane = d ? nullptr : (const T *)c->pos_plane32.p;
    g.gvert = c->pos_gvert.as<int>();
    g.face_id = c->pos_face.as<int>();
    g.t_fstart = tiles.face_start.as<int>();
    g.t_vstart = tiles.vert_start.as<int>();
    g.t_verts = tiles.verts.as<int>();
    g.t_local = tiles.local_vert.as<int>();
    g.t_inc = tiles.incidence.as<int>();
    BB_REQUIRE(tiles.inc_stride() == SymTile<T>::INC, BEAT_B200_STATE, "assembly: square tile shape mismatch");
    g.A = c->ws.A.as<Cx<T>>();
    g.B = c->ws.rhs_cached ? c->ws.B.as<Cx<T>>() : nullptr;
    g.q = q;
    g.b = c->ws.b.as<Cx<double>>();
    g.N = c->V;
    g.R = R;
    g.ld = c->ws.ld;
    g.F = c->F;
    g.k = (T)k;
    g.eta = (T)eta;
    g.k2 = (T)(k * k);
    if (img >= 0) {
        g.image = 1;
        for (int i = 0; i < 3; ++i) g.xs[i] = c->img_sign[img][i];
        g.xdet = c->img_det[img];
    }
    const size_t smem = SymTile<T>::template smem<Q>();
    BB_CUDA(cudaFuncSetAttribute(sym_pairs_kernel<T, Q>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    BB_CUDA(cudaFuncSetAttribute(sym_pairs_kernel<T, Q>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 cudaSharedmemCarveoutMaxShared));  // two CTAs per SM
    const int64_t nt = tiles.ntiles;
    const int64_t blocks = nt * (nt + 1) / 2;
    BB_REQUIRE(blocks < (1ll << 31), BEAT_B200_INVALID_ARG, "assembly: mesh too large for the tile-pair grid");
    sym_pairs_kernel<T, Q><<<(unsigned)blocks, SymTile<T>::THREADS, smem, c->stream>>>(g);
    BB_CUDA(cudaGetLastError());
}

template <typename T> static void assemble_t(beat_b200_ctx *c, double k, double eta, int R, const Cx<double> *q) {
    Workspace &w = c->ws;
    const int N = c->V, F = c->F;
    BB_CUDA(cudaEventRecord(c->ev[0], c->stream));
    BB_CUDA(cudaMemsetAsync(w.A.p, 0, (size_t)N * w.ld * sizeof(Cx<T>), c->stream));
    if (w.rhs_cached)
        BB_CUDA(cudaMemsetAsync(w.B.p, 0, (size_t)N * F * sizeof(Cx<T>), c->stream));
    else  // matrix-free: the kernels add into b directly
        BB_CUDA(cudaMemsetAsync(w.b.p, 0, sizeof(Cx<double>) * (size_t)N * R, c->stream));
    BB_CUDA(cudaEventRecord(c->ev[8], c->stream));
    for (int img = -1; img < c->nimg; ++img) {  // the mesh itself, then one pass per symmetry image
        switch (c->Q) {
            case 1: launch_sym<T, 1>(c, k, eta, img, R, q); break;
            case 3: launch_sym<T, 3>(c, k, eta, img, R, q); break;
            default: launch_sym<T, 6>(c, k, eta, img, R, q); break;
        }
    }
    BB_CUDA(cudaEventRecord(c->ev[1], c->stream));
    if (c->npairs > 0) {
        SingArgs<T> s;
        s.test = c->sp_test.as<int>();
        s.trial = c->sp_trial.as<int>();
        s.rule = c->sp_rule.as<int>();
        s.jac = c->sp_jac.as<double>();
        s.nn = c->sp_nn.as<double>();
        s.rule_start = c->rule_start.as<int>();
        s.rule_data = c->rule_data.as<double>();
        s.npoints = c->npoints;
        s.verts = c->d_verts.as<double>();
        s.faces = c->d_faces.as<int>();
        s.normals = c->d_normals.as<double>();
        s.curls = c->d_curls.as<double>();
        s.A = w.A.as<Cx<T>>();
        s.rhs = rhs_out<T>(c, R, q);
        s.ld = w.ld;
        s.npairs = c->npairs;
        s.k = k;
        s.eta = eta;
        const int wpb = 8;
        singular_pairs_kernel<T><<<(unsigned)((c->npairs + wpb - 1) / wpb), 32 * wpb, 0, c->stream>>>(s);
        BB_CUDA(cudaGetLastError());
    }
    if (c->nimg_pairs > 0) {
        ImgArgs<T> d;
        d.test = c->ip_test.as<int>();
        d.trial = c->ip_trial.as<int>();
        d.rule = c->ip_rule.as<int>();
        d.img = c->ip_img.as<int>();
        d.jac = c->ip_jac.as<double>();
        d.nn = c->ip_nn.as<double>();
        d.rule_start = c->rule_start.as<int>();
        d.rule_data = c->rule_data.as<double>();
        d.npoints = c->npoints;
        d.verts = c->d_verts.as<double>();
        d.faces = c->d_faces.as<int>();
        d.normals = c->d_normals.as<double>();
        d.curls = c->d_curls.as<double>();
        d.Q = c->Q;
        d.RI = c->Q == 1 ? 0 : c->Q == 3 ? 1 : 2;
        d.A = w.A.as<Cx<T>>();
        d.rhs = rhs_out<T>(c, R, q);
        d.ld = w.ld;
        d.npairs = c->nimg_pairs;
        d.k = k;
        d.eta = eta;
        for (int i = 0; i < 3; ++i) {
            for (int j = 0; j < 3; ++j) d.xf.s[i][j] = c->img_sign[i][j];
            d.xf.det[i] = c->img_det[i];
        }
        image_delta_kernel<T><<<(unsigned)((c->nimg_pairs + 7) / 8), 256, 0, c->stream>>>(d);
        BB_CUDA(cudaGetLastError());
    }
    BB_CUDA(cudaEventRecord(c->ev[2], c->stream));
    identity_kernel<T><<<(F + 255) / 256, 256, 0, c->stream>>>(c->d_faces.as<int>(), c->d_areas.as<double>(), F,
                                                               c->Q, eta, w.A.as<Cx<T>>(), w.ld, rhs_out<T>(c, R, q));
    BB_CUDA(cudaGetLastError());
    if (c->nweighted > 0) {
        row_weight_kernel<T><<<dim3(32, c->nweighted), 256, 0, c->stream>>>(
            c->rw_vert.as<int>(), c->rw_weight.as<double>(), c->nweighted, w.A.as<Cx<T>>(), w.ld, N,
            rhs_out<T>(c, R, q));
        BB_CUDA(cudaGetLastError());
    }
    if (w.rhs_cached && R > 0) {
        BB_CUDA(cudaMemsetAsync(w.b.p, 0, sizeof(Cx<double>) * (size_t)N * R, c->stream));
        tall_gemm<T>(c->stream, c->sm_count, w.B.as<Cx<T>>(), F, N, F, reinterpret_cast<const double *>(q),
                     w.b.as<double>(), R, 1.0);
    }
    BB_CUDA(cudaEventRecord(c->ev[3], c->stream));
}

void assembly_times(beat_b200_ctx *c, float *total, float *singular, float *regular) {
    BB_CUDA(cudaEventElapsedTime(total, c->ev[0], c->ev[3]));
    BB_CUDA(cudaEventElapsedTime(singular, c->ev[1], c->ev[2]));
    BB_CUDA(cudaEventElapsedTime(regular, c->ev[8], c->ev[1]));
}

void assemble(beat_b200_ctx *c, double k, double eta, int precision, int R, const void *q_dev) {
    BB_REQUIRE(c->F > 0, BEAT_B200_STATE, "no mesh: call beat_b200_set_mesh first");
    BB_REQUIRE(std::isfinite(k) && k != 0.0 && std::isfinite(eta), BEAT_B200_INVALID_ARG,
               "assemble: wavenumber must be finite and nonzero");
    if (precision == BEAT_B200_FP64)
        assemble_t<double>(c, k, eta, R, (const Cx<double> *)q_dev);
    else
        assemble_t<float>(c, k, eta, R, (const Cx<double> *)q_dev);
}

}  // namespace bb
