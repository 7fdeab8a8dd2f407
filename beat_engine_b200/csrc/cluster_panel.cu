// cluster_panel.cu -- the LU's sub-panel factorisation on one thread-block
// cluster.  Compiled once per precision (BB_T) and number of rows per thread
// (BB_ROWS), see build.py: a kernel's first use in a process loads its whole
// module, and each of these is two dozen unrolled column steps.  All six beside
// the other LU kernels made a module of 9.0 MB that took 4.1 ms of the first
// solve; now that one takes 2.2 ms and a variant, when it is first used, 0.5
// (first request at F = 2,776: 11.6 -> 9.8 ms; later ones 3.6).
#include <cuda_runtime.h>

#include <type_traits>

#include "lu.cuh"

namespace bb {

// ---------------------------------------------------------------------------
// Sub-panel factorisation on one thread-block cluster of C CTAs (16, or 1 for
// few rows).  A thread keeps RPT whole 256-byte rows (32 c64 or 16 c128
// columns, 64 registers each), as pairs of columns with the real and the
// imaginary parts packed (one FP32 instruction then updates both columns), so
// eliminating a column touches shared memory only for the broadcast pivot row.
// Rows never move: each carries its logical position, and an interchange only
// swaps two positions.
//
// The loop over columns advances two at a time: the even column is the first
// half of the thread's first pair, the odd one the second half, and the odd
// step shifts the pairs down by one as it updates them, so the register
// indices are compile-time constants in a loop body of fixed length.  Four
// phases of W / 4 columns drop the finished pairs from the body.  Per column j:
//   1. C > 1: wait on this CTA's mbarrier until every CTA's candidate for
//      column j (key: magnitude, position, reciprocal of the pivot; and the
//      whole candidate row) has landed; every warp picks the same winner
//      (redux.sync on the magnitude bits, then the smallest position);
//   2. the multiplier and column j + 1 of each row; each warp's best row's key
//      to shared memory; a CTA barrier; every warp picks the CTA's best;
//   3. the best row's thread writes the row as it stands before this step to
//      the staging buffer; its warp's lanes finish it, 16 bytes each, and push
//      it with its key to every CTA (st.async, complete_tx on the receiver's
//      mbarrier).  With C = 1 they leave it in the staging buffer, which every
//      thread reads next after a second CTA barrier: no exchange;
//   4. every thread eliminates the rest of step j, the other warps at once, the
//      pushing warp afterwards.
// Multipliers and retired pivot rows go to a shared-memory copy of the
// sub-panel, which the bulk-copy engine loaded and stores at the end; rank 0
// keeps the pivot rows' multipliers (L11) and inverts them during that store.
//
// Slots and mbarriers rotate over three columns: a CTA's slowest warps read
// the slot of column j after the CTA pushed its candidate for j + 1, and finish
// before it pushes j + 2; a peer pushes j + 3, which reuses the slot, only once
// it holds every candidate for j + 2.  Staging buffers and warp keys alternate
// with the column parity, separated by the column's CTA barriers.  Every wait
// is bounded.
//
// Bound: the dependent chain of one pivot per column (the exchange between
// CTAs, two argmax reductions, two barriers), at about five cycles an
// instruction: one warp per scheduler while the rows allow it, and no more
// on the chain than the candidate's own row.  Measured on a B200, the whole
// factorisation, against rows kept in shared memory by 512 threads of 16 CTAs
// whatever their number: FP32 N = 162 0.60 -> 0.41 ms, N = 1,390 4.17 -> 2.65,
// N = 10,242 38.1 -> 31.0 (72 us a sub-panel, 45 at 1,390 rows); FP64 N = 998 3.04 -> 2.83.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t cl_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t sm_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t cl_map(uint32_t a, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void cl_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cl_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void cl_sync() {
    cl_arrive();
    cl_wait();
}
__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ void mb_init(uint64_t *b, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(sm_addr(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mb_init_fence() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mb_arrive_expect(uint64_t *b, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(sm_addr(b)), "r"(bytes) : "memory");
}
// true once the phase of the given parity completed (the thread may be
// suspended inside until the phase completes or a time limit of the system
// passes; with a suspend-time hint of 1 us the panels measured 3 % slower)
__device__ __forceinline__ bool mb_try(uint64_t *b, unsigned parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(sm_addr(b)), "r"(parity)
        : "memory");
    return ok != 0;
}
// one row of 16-byte-aligned bytes between global and shared memory by the
// bulk-copy engine (no multicast); the load completes on an mbarrier
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void bulk_s2g(void *dst, uint32_t src, uint32_t bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_commit_wait_all() {
    asm volatile("cp.async.bulk.commit_group;\n\tcp.async.bulk.wait_group 0;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void st_async16(uint32_t addr, uint4 v, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(
                     addr),
                 "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(bar)
                 : "memory");
}

// ordered bits of a non-negative magnitude (0 also stands for "none")
__device__ __forceinline__ uint32_t mag_bits(float v) { return __float_as_uint(v); }
__device__ __forceinline__ uint64_t mag_bits(double v) { return (uint64_t)__double_as_longlong(v); }
__device__ __forceinline__ float mag_value(uint32_t b) { return __uint_as_float(b); }
__device__ __forceinline__ double mag_value(uint64_t b) { return __longlong_as_double((long long)b); }

// lane holding the largest magnitude, the smallest position among equals
// (all 32 lanes take part; the result is the same in every lane)
template <typename M> __device__ __forceinline__ int warp_argbest(M m, int pos) {
    bool tie;
    if constexpr (sizeof(M) == 8) {
        const uint32_t hi = (uint32_t)(m >> 32), lo = (uint32_t)m;
        const uint32_t mhi = __reduce_max_sync(0xffffffffu, hi);
        const uint32_t mlo = __reduce_max_sync(0xffffffffu, hi == mhi ? lo : 0u);
        tie = hi == mhi && lo == mlo;
    } else {
        tie = m == __reduce_max_sync(0xffffffffu, m);
    }
    const unsigned ties = __ballot_sync(0xffffffffu, tie);
    if ((ties & (ties - 1u)) == 0u) return __ffs(ties) - 1;  // one largest magnitude: no position to compare
    const int mpos = __reduce_min_sync(0xffffffffu, tie ? pos : CP_NONE);
    return __ffs(__ballot_sync(0xffffffffu, tie && pos == mpos)) - 1;
}

// Two columns of a row, real and imaginary parts as packed pairs, and a
// multiplier for them.  FP32 packs a pair into one 64-bit register operand
// (fma.rn.f32x2).  In shared memory a pair is (re0, re1, im0, im1).
template <typename T> struct ColPair;
template <typename T> struct ColMult;
template <> struct alignas(16) ColPair<float> { unsigned long long re, im; };
template <> struct alignas(16) ColPair<double> { double re[2], im[2]; };
template <> struct ColMult<float> { unsigned long long nr, i, ni; };  // (-l.re, -l.re), (l.im, l.im), (-l.im, -l.im)
template <> struct ColMult<double> { double r, i; };
__device__ __forceinline__ unsigned long long f2_pack(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void f2_unpack(unsigned long long v, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ unsigned long long f2_fma(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ unsigned long long f2_mul(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long f2_add(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ ColPair<float> pair_ld(const unsigned char *p, float) {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(p);
    return ColPair<float>{v.x, v.y};
}
__device__ __forceinline__ ColPair<double> pair_ld(const unsigned char *p, double) {
    const double2 a = reinterpret_cast<const double2 *>(p)[0], b = reinterpret_cast<const double2 *>(p)[1];
    return ColPair<double>{{a.x, a.y}, {b.x, b.y}};
}
__device__ __forceinline__ void pair_st(unsigned char *p, const ColPair<float> &v) {
    *reinterpret_cast<ulonglong2 *>(p) = make_ulonglong2(v.re, v.im);
}
__device__ __forceinline__ void pair_st(unsigned char *p, const ColPair<double> &v) {
    reinterpret_cast<double2 *>(p)[0] = make_double2(v.re[0], v.re[1]);
    reinterpret_cast<double2 *>(p)[1] = make_double2(v.im[0], v.im[1]);
}
template <int H> __device__ __forceinline__ Cx<float> pair_get(const ColPair<float> &v) {
    float r0, r1, i0, i1;
    f2_unpack(v.re, r0, r1);
    f2_unpack(v.im, i0, i1);
    return H ? Cx<float>{r1, i1} : Cx<float>{r0, i0};
}
template <int H> __device__ __forceinline__ Cx<double> pair_get(const ColPair<double> &v) {
    return Cx<double>{v.re[H], v.im[H]};
}
__device__ __forceinline__ ColPair<float> pair_make(Cx<float> a, Cx<float> b) {
    return ColPair<float>{f2_pack(a.re, b.re), f2_pack(a.im, b.im)};
}
__device__ __forceinline__ ColPair<double> pair_make(Cx<double> a, Cx<double> b) {
    return ColPair<double>{{a.re, b.re}, {a.im, b.im}};
}
__device__ __forceinline__ ColMult<float> pair_mult(Cx<float> l) {
    return ColMult<float>{f2_pack(-l.re, -l.re), f2_pack(l.im, l.im), f2_pack(-l.im, -l.im)};
}
__device__ __forceinline__ ColMult<double> pair_mult(Cx<double> l) { return ColMult<double>{l.re, l.im}; }
// x - l u, the product apart: one rounding at the entry's magnitude.  (Two fused
// steps on x round there twice: unrefined FP32 solutions at 82 to 2,524 unknowns
// were 2 to 9 % less exact; LU 2.48 -> 2.50 ms at N = 1,390.)
__device__ __forceinline__ ColPair<float> pair_cms(const ColPair<float> &x, const ColMult<float> &l,
                                                   const ColPair<float> &u) {
    return ColPair<float>{f2_add(x.re, f2_fma(l.i, u.im, f2_mul(l.nr, u.re))),
                          f2_add(x.im, f2_fma(l.ni, u.re, f2_mul(l.nr, u.im)))};
}
__device__ __forceinline__ ColPair<double> pair_cms(const ColPair<double> &x, const ColMult<double> &l,
                                                    const ColPair<double> &u) {
    ColPair<double> d;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        d.re[h] = x.re[h] + fma(l.i, u.im[h], -l.r * u.re[h]);
        d.im[h] = x.im[h] + fma(-l.i, u.re[h], -l.r * u.im[h]);
    }
    return d;
}

// 16 bytes of a pair of columns, x - l u: a whole FP32 pair, or one half (0:
// real parts, 1: imaginary parts) of an FP64 pair
__device__ __forceinline__ uint4 finish16(uint4 x, const ColMult<float> &l, const ColPair<float> &u, int) {
    const ulonglong2 b = *reinterpret_cast<const ulonglong2 *>(&x);
    const ColPair<float> v = pair_cms(ColPair<float>{b.x, b.y}, l, u);
    return make_uint4((uint32_t)v.re, (uint32_t)(v.re >> 32), (uint32_t)v.im, (uint32_t)(v.im >> 32));
}
__device__ __forceinline__ uint4 finish16(uint4 x, const ColMult<double> &l, const ColPair<double> &u, int half) {
    double v[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const double xh = h ? __hiloint2double((int)x.w, (int)x.z) : __hiloint2double((int)x.y, (int)x.x);
        v[h] = xh + (half ? fma(-l.i, u.re[h], -l.r * u.im[h]) : fma(l.i, u.im[h], -l.r * u.re[h]));
    }
    return make_uint4((uint32_t)__double2loint(v[0]), (uint32_t)__double2hiint(v[0]), (uint32_t)__double2loint(v[1]),
                      (uint32_t)__double2hiint(v[1]));
}
// 16 bytes (part 0, and in FP64 part 1) of a candidate's key: magnitude,
// position, reciprocal of the pivot
__device__ __forceinline__ uint4 key16(uint32_t m, int pos, Cx<float> inv, int) {
    return make_uint4(m, (uint32_t)pos, __float_as_uint(inv.re), __float_as_uint(inv.im));
}
__device__ __forceinline__ uint4 key16(uint64_t m, int pos, Cx<double> inv, int part) {
    if (part == 0) return make_uint4((uint32_t)m, (uint32_t)(m >> 32), (uint32_t)pos, 0u);
    return make_uint4((uint32_t)__double2loint(inv.re), (uint32_t)__double2hiint(inv.re),
                      (uint32_t)__double2loint(inv.im), (uint32_t)__double2hiint(inv.im));
}


template <typename T, int RPT>
__global__ void __launch_bounds__(CP_THREADS, 1) cluster_panel_kernel(ClusterPanelArgs<T> a) {
    using S = CpShape<T>;
    using M = decltype(mag_bits(T(0)));
    constexpr int W = S::W, NPM = S::NP, PB = S::PB, KB = S::KB, RSL = S::RSL;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, NT = (int)blockDim.x, NW = NT >> 5;
    const uint32_t rank = cl_rank();
    const int C = (int)gridDim.x;  // one cluster
    unsigned char *slot_row = smem_raw;                            // [CP_SLOTS][C][RSL]
    unsigned char *stage = slot_row + (size_t)CP_SLOTS * C * RSL;  // [2][RSL]
    unsigned char *slot_key = stage + 2 * RSL;                     // [CP_SLOTS][C][KB]
    unsigned char *stage_key = slot_key + (size_t)CP_SLOTS * C * KB;  // [2][KB]
    Cx<T> *l11 = reinterpret_cast<Cx<T> *>(stage_key + 2 * KB);    // W x (W + 1): L11 (rank 0)
    Cx<T> *y11 = l11 + W * (W + 1);                                // W x (W + 1): its inverse
    unsigned char *P = reinterpret_cast<unsigned char *>(y11 + W * (W + 1));  // rpc rows of CP_ROW_BYTES, complex
    struct alignas(16) Key {  // a warp's best row
        M m;
        int pos, li;
    };
    __shared__ uint64_t mbar[CP_SLOTS];
    __shared__ uint64_t ldbar;  // the sub-panel's rows landed in shared memory
    __shared__ Key red[2][CP_WARPS];
    __shared__ int s_abort[2];
    const int gr0 = a.k + (int)rank * a.rpc;
    const int nrows = max(0, min(a.rpc, a.n - gr0));
    const int jmax = min(W, a.n - a.k);
    const unsigned step_bytes = (unsigned)C * (256 + KB);
    auto row_at = [&](int i) { return reinterpret_cast<Cx<T> *>(P + (size_t)i * CP_ROW_BYTES); };
    if (tid == 0) {
        mb_init(&ldbar, 1);
        for (int b = 0; b < CP_SLOTS; ++b) mb_init(&mbar[b], 1);
        mb_init_fence();
        mb_arrive_expect(&ldbar, (unsigned)nrows * 256u);
        for (int b = 0; b < CP_SLOTS; ++b) mb_arrive_expect(&mbar[b], step_bytes);  // columns 0, 1, 2
        s_abort[0] = s_abort[1] = 0;
    }
    __syncthreads();
    if (C > 1) cl_arrive();
    for (int i = tid; i < nrows; i += NT)  // rows in flight all at once
        bulk_g2s(sm_addr(row_at(i)), a.A + (int64_t)(gr0 + i) * a.ld + a.k, 256u, sm_addr(&ldbar));
    if (!mb_try(&ldbar, 0u)) {
        const uint64_t t0 = global_ns();
        while (!mb_try(&ldbar, 0u))
            if (global_ns() - t0 > a.timeout_ns) {
                atomicOr(a.status, (int)DEV_BARRIER_TIMEOUT);
                break;
            }
    }
    // logical positions of this thread's rows (local rows tid + r NT; -1: none)
    int mp[RPT];
    ColPair<T> A[RPT][NPM];
#pragma unroll
    for (int r = 0; r < RPT; ++r) {
        const int i = tid + r * NT;
        mp[r] = i < nrows ? gr0 + i : -1;
#pragma unroll
        for (int q = 0; q < NPM; ++q) {
            const Cx<T> z{T(0), T(0)};
            A[r][q] = mp[r] >= 0 ? pair_make(row_at(i)[2 * q], row_at(i)[2 * q + 1]) : pair_make(z, z);
        }
    }

    // a thread's best row: magnitude, position, local row, the entry itself and
    // the multiplier that finishes the row
    struct Best {
        M m = 0;
        int pos = CP_NONE, li = 0;
        Cx<T> y{T(0), T(0)}, l{T(0), T(0)};
        __device__ __forceinline__ void offer(Cx<T> y1, Cx<T> l1, int pos1, int li1) {
            const M m1 = mag_bits(cabs1(y1));
            if (pos == CP_NONE || m1 > m || (m1 == m && pos1 < pos)) {
                m = m1;
                pos = pos1;
                li = li1;
                y = y1;
                l = l1;
            }
        }
    };
    Key cand{0, CP_NONE, 0};  // the CTA's best row for the next column
    // The CTA's candidate for column s (each thread's best in `b`) to every CTA
    // (C = 1: to the staging buffer).  prow: the pivot row of step s - 1, which
    // finishes the candidate's pairs (nullptr: the rows are as loaded).  SH, NP:
    // this thread's pairs, A[r][i] at pair (s >> 1) + i - SH.
    auto publish = [&](auto shc, auto npc, int s, int slot, const Best &b, const unsigned char *prow) -> bool {
        constexpr int SH = decltype(shc)::value, NP = decltype(npc)::value;
        const int pb = s & 1, base = s >> 1;
        const int wl = warp_argbest(b.m, b.pos);
        if (lane == wl) red[pb][warp] = Key{b.m, b.pos, b.li};
        __syncthreads();
        if (s_abort[pb ^ 1]) return false;  // set before the barrier: uniform
        const int bw = [&] {
            const Key r = lane < NW ? red[pb][lane] : Key{0, CP_NONE, 0};
            return warp_argbest(r.m, r.pos);
        }();
        cand = red[pb][bw];
        unsigned char *buf = stage + pb * RSL;
        if (warp == bw) {
            const bool some = cand.pos != CP_NONE;
            if (some && lane == wl) {
#pragma unroll
                for (int r = 0; r < RPT; ++r)
                    if (cand.li == tid + r * NT) {
#pragma unroll
                        for (int i = SH; i < NP; ++i)  // (past the row's end: the slot's padding)
                            pair_st(buf + (base + i - SH) * PB, A[r][i]);
                    }
            }
            const Cx<T> l{__shfl_sync(0xffffffffu, b.l.re, wl), __shfl_sync(0xffffffffu, b.l.im, wl)};
            const Cx<T> y{__shfl_sync(0xffffffffu, b.y.re, wl), __shfl_sync(0xffffffffu, b.y.im, wl)};
            const T den = y.re * y.re + y.im * y.im;
            const T rd = den > T(0) ? rcp_rn(den) : T(0);
            const Cx<T> inv{y.re * rd, -y.im * rd};
            __syncwarp();
            // lane q < 16: 16 bytes of the row, finished; of its first s / 2
            // pairs (multipliers, complex entries) from the sub-panel's copy
            const int q = lane * 16 / PB;  // the pair they belong to
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if (some && lane < 16) {
                v = reinterpret_cast<const uint4 *>(q < base ? P + (size_t)cand.li * CP_ROW_BYTES : buf)[lane];
                if (prow && q >= base + (s & 1)) v = finish16(v, pair_mult(l), pair_ld(prow + q * PB, T(0)), lane & 1);
            } else if (lane >= 16) {
                v = key16(some ? cand.m : M(0), cand.pos, some ? inv : Cx<T>{T(0), T(0)}, lane - 16);
            }
            if (C == 1) {
                if (lane < 16 && q >= base) reinterpret_cast<uint4 *>(buf)[lane] = v;
                if (lane >= 16 && lane < 16 + KB / 16) reinterpret_cast<uint4 *>(stage_key + pb * KB)[lane - 16] = v;
            } else if (lane < 16 + KB / 16) {
                const uint32_t dst = lane < 16 ? sm_addr(slot_row) + (uint32_t)(slot * C + rank) * RSL + 16u * lane
                                               : sm_addr(slot_key) + (uint32_t)(slot * C + rank) * KB + 16u * (lane - 16);
                const uint32_t to_bar = sm_addr(&mbar[slot]) - dst;  // the same distance in every CTA
#pragma unroll
                for (int peer = 0; peer < CP_CTAS; ++peer) {
                    const uint32_t d = cl_map(dst, peer);
                    st_async16(d, v, d + to_bar);
                }
            }
        }
        if (C == 1) __syncthreads();
        return true;
    };

    int par = 0;            // slot of the current column
    unsigned phase = 0;     // parity of its mbarrier phase
    bool stop = false;
    // one column; ODD: the pivot column is the second of the first pair
    auto step = [&](auto npc, auto oddc, int j) {
        constexpr int NP = decltype(npc)::value;
        constexpr int ODD = decltype(oddc)::value;
        const int jr = a.k + j, pb = j & 1;
        const unsigned char *prow = stage + pb * RSL, *pkey = stage_key + pb * KB;
        const unsigned char *lrow = P + (size_t)cand.li * CP_ROW_BYTES;  // the pivot row's multipliers
        int p = cand.pos;
        M wm = cand.m;
        if (C > 1) {
            if (!mb_try(&mbar[par], phase)) {
                const uint64_t t0 = global_ns();
                while (!mb_try(&mbar[par], phase)) {
                    if (global_ns() - t0 > a.timeout_ns) {
                        s_abort[pb] = 1;
                        atomicOr(a.status, (int)DEV_BARRIER_TIMEOUT);
                        break;
                    }
                }
            }
            if (tid == 0 && !s_abort[pb]) mb_arrive_expect(&mbar[par], step_bytes);  // next phase: column j + 3
            // the same winner in every warp
            const M *km = reinterpret_cast<const M *>(slot_key + (size_t)(par * C + (lane & (C - 1))) * KB);
            const M m = lane < C ? km[0] : M(0);
            const int pos = lane < C ? reinterpret_cast<const int *>(km + 1)[0] : CP_NONE;
            const int wc = warp_argbest(m, pos) & (C - 1);
            prow = lrow = slot_row + (size_t)(par * C + wc) * RSL;
            pkey = slot_key + (size_t)(par * C + wc) * KB;
            wm = reinterpret_cast<const M *>(pkey)[0];
            p = reinterpret_cast<const int *>(pkey + sizeof(M))[0];
        }
        const Cx<T> inv = *reinterpret_cast<const Cx<T> *>(pkey + KB / 2);
        const unsigned char *up = prow + (j >> 1) * PB;  // the pair A[r][0] stands for
        // the pivot row's column j + 1
        const Cx<T> un = pair_get<1 - ODD>(pair_ld(up + ODD * PB, T(0)));
        if (p < jr || p >= a.n) {  // no candidate (or a damaged slot): keep the row in place
            p = jr;
            wm = 0;
        }
        const bool more = j + 1 < jmax;
        // the interchange of positions jr and p (the pivot row retires at
        // jr), then the look-ahead: multiplier and column j + 1 of each row
        // (a row that is not active has multiplier 0 and keeps its values)
        Cx<T> l[RPT];
        Best best;
#pragma unroll
        for (int r = 0; r < RPT; ++r) {
            if (mp[r] == p)
                mp[r] = jr;
            else if (mp[r] == jr)
                mp[r] = p;
            const bool act = mp[r] > jr;
            const Cx<T> x = pair_get<ODD>(A[r][0]);
            l[r] = cmul(x, inv);
            if (!act) l[r] = Cx<T>{T(0), T(0)};
            const Cx<T> y = cms(ODD ? pair_get<0>(A[r][NP > 1 ? 1 : 0]) : pair_get<1>(A[r][0]), l[r], un);
            // the first column is final (the multiplier, or the pivot row's own entry)
            if constexpr (!ODD) A[r][0] = pair_make(act ? l[r] : x, y);
            if (act && more) best.offer(y, l[r], mp[r], tid + r * NT);
            if (act) row_at(tid + r * NT)[j] = l[r];  // read by the push of the candidate that holds it
        }
        const int nslot = par == CP_SLOTS - 1 ? 0 : par + 1;
        if (more && !publish(oddc, npc, j + 1, nslot, best, prow)) {
            stop = true;
            return;
        }
        // the rest of this step; a retiring pivot row goes to the sub-panel's copy first
#pragma unroll
        for (int r = 0; r < RPT; ++r)
            if (mp[r] == jr) {
                Cx<T> *row = row_at(tid + r * NT);
#pragma unroll
                for (int i = 0; i < NP; ++i) {
                    const int q = (j >> 1) + i;
                    if (q < NPM) {
                        row[2 * q] = pair_get<0>(A[r][i]);
                        row[2 * q + 1] = pair_get<1>(A[r][i]);
                    }
                }
            }
        ColMult<T> lm[RPT];
#pragma unroll
        for (int r = 0; r < RPT; ++r) lm[r] = pair_mult(l[r]);
#pragma unroll
        for (int i = 1; i < NP; ++i) {
            const ColPair<T> u = pair_ld(up + i * PB, T(0));
#pragma unroll
            for (int r = 0; r < RPT; ++r) A[r][i - ODD] = pair_cms(A[r][i], lm[r], u);
        }
        // the pivot's index; L11's row j (complex entries in the pairs before
        // j / 2, then the first half of pair j / 2)
        if (rank == 0 && warp == NW - 1) {
            if (lane == 0) {
                if (!(mag_value(wm) > T(0))) atomicOr(a.status, (int)DEV_ZERO_PIVOT);
                a.ipiv[jr] = p;
            }
            if (lane < W)
                l11[j * (W + 1) + lane] = lane >= j                    ? Cx<T>{T(lane == j), T(0)}
                                          : (lane >> 1) < (j >> 1) ? reinterpret_cast<const Cx<T> *>(lrow)[lane]
                                                                       : pair_get<0>(pair_ld(up, T(0)));
        }
        if (!more) {
            stop = true;
            return;
        }
        par = nslot;
        phase ^= nslot == 0 ? 1u : 0u;
    };
    // candidate of column 0
    {
        Best best;
        const Cx<T> z{T(0), T(0)};
#pragma unroll
        for (int r = 0; r < RPT; ++r)
            if (mp[r] >= 0) best.offer(pair_get<0>(A[r][0]), z, mp[r], tid + r * NT);
        if (C > 1) cl_wait();  // every CTA's mbarriers are initialised before any remote store
        publish(std::integral_constant<int, 0>{}, std::integral_constant<int, NPM>{}, 0, 0, best, nullptr);
    }
    auto run_phase = [&](auto npc, int j0) {
#pragma unroll 1
        for (int j = j0; j < j0 + W / 4 && !stop; j += 2) {
            step(npc, std::integral_constant<int, 0>{}, j);
            if (!stop) step(npc, std::integral_constant<int, 1>{}, j + 1);
        }
    };
    run_phase(std::integral_constant<int, NPM>{}, 0);
    run_phase(std::integral_constant<int, NPM * 3 / 4>{}, W / 4);
    run_phase(std::integral_constant<int, NPM / 2>{}, W / 2);
    run_phase(std::integral_constant<int, NPM / 4>{}, W * 3 / 4);

    // each row to its final position, by the bulk-copy engine
    fence_proxy_async_smem();
    __syncthreads();
    auto each_row = [&](auto &&fn) {
#pragma unroll
        for (int r = 0; r < RPT; ++r)
            if (mp[r] >= a.k && mp[r] < a.n) fn(tid + r * NT, mp[r]);
    };
    each_row([&](int i, int pos) { bulk_s2g(a.A + (int64_t)pos * a.ld + a.k, sm_addr(row_at(i)), 256u); });
    // the same interchanges on the panel's other columns: every CTA reads its
    // moved rows there before the cluster barrier and writes them at their
    // final positions after it (a permutation: every destination is some moved
    // row's origin, read before the barrier)
    __shared__ int mv_src[2 * W], mv_dst[2 * W], mv_n;
    constexpr int MVC = S::MVC, MVT = S::MVT, E = 16 / sizeof(Cx<T>);
    const int nleft = (a.k - a.xc0) / E, nother = a.xc1 > a.xc0 ? nleft + max(0, a.xc1 - a.k - W) / E : 0;
    const int mc = tid % MVC, mr0 = tid / MVC, mrs = NT / MVC;
    const int mcol = mc < nleft ? a.xc0 + mc * E : a.k + W + (mc - nleft) * E;
    uint4 mvv[MVT];
    int nmoved = 0;
    if (nother > 0) {
        if (tid == 0) mv_n = 0;
        __syncthreads();
        each_row([&](int i, int pos) {
            if (pos != gr0 + i) {
                const int slot = atomicAdd(&mv_n, 1);
                if (slot < 2 * W) {
                    mv_src[slot] = gr0 + i;
                    mv_dst[slot] = pos;
                }
            }
        });
        __syncthreads();
        nmoved = mc < nother ? min(mv_n, 2 * W) : 0;
#pragma unroll
        for (int u = 0; u < MVT; ++u)
            if (mr0 + u * mrs < nmoved)
                mvv[u] = *reinterpret_cast<const uint4 *>(a.A + (int64_t)mv_src[mr0 + u * mrs] * a.ld + mcol);
    }
    if (rank == 0 && a.dinv) {
        // The inverse of L11 (identity past jmax): the 8 x 8 diagonal blocks'
        // by substitution, a column per lane, then doubling: with the b x b
        // diagonal blocks inverted, Y21 = -Y22 (L21 Y11) for each pair of
        // them, L21 Y11 kept above l11's diagonal.
        for (int e = tid; e < W * W; e += NT) {
            const int i = e / W, c = e % W;
            if (i / 8 != c / 8) y11[i * (W + 1) + c] = Cx<T>{T(0), T(0)};
            if (i >= jmax) l11[i * (W + 1) + c] = Cx<T>{T(i == c), T(0)};
        }
        __syncthreads();
        if (tid < W) {
            const int d = tid & ~7;
            const Cx<T> *L = l11 + d * (W + 1) + d;
            Cx<T> v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                v[i] = Cx<T>{T(i == (tid & 7)), T(0)};
#pragma unroll
                for (int t = 0; t < i; ++t) v[i] = cms(v[i], L[i * (W + 1) + t], v[t]);
                y11[(d + i) * (W + 1) + tid] = v[i];
            }
        }
        __syncthreads();
#pragma unroll 1
        for (int b = 8, lb = 3; b < W; b *= 2, ++lb)
#pragma unroll 1
            for (int pass = 0; pass < 2; ++pass) {
                for (int e = tid; e < W / 2 * b; e += NT) {
                    const int d = (e >> (2 * lb)) * 2 * b, i = (e >> lb) & (b - 1), c = e & (b - 1);
                    const Cx<T> *left = (pass ? y11 + (d + b + i) * (W + 1) + d + b : l11 + (d + b + i) * (W + 1) + d);
                    const Cx<T> *right = (pass ? l11 + b : y11) + d * (W + 1) + d + c;
                    Cx<T> s0{T(0), T(0)}, s1{T(0), T(0)};
#pragma unroll 4
                    for (int t = 0; t < b; t += 2) {
                        s0 = cms(s0, left[t], right[t * (W + 1)]);
                        s1 = cms(s1, left[t + 1], right[(t + 1) * (W + 1)]);
                    }
                    const Cx<T> v{s0.re + s1.re, s0.im + s1.im};  // -(left right)
                    if (pass == 0)
                        l11[(d + i) * (W + 1) + d + b + c] = Cx<T>{-v.re, -v.im};
                    else
                        y11[(d + b + i) * (W + 1) + d + c] = v;
                }
                __syncthreads();
            }
        for (int e = tid; e < W * W; e += NT) {
            const int i = e / W, c = e % W;
            a.dinv[e] = y11[i * (W + 1) + c];
        }
    }
    bulk_commit_wait_all();
    cl_sync();  // every CTA's reads are done; no CTA leaves while a peer may still store into its shared memory
#pragma unroll
    for (int u = 0; u < MVT; ++u)
        if (mr0 + u * mrs < nmoved)
            *reinterpret_cast<uint4 *>(a.A + (int64_t)mv_dst[mr0 + u * mrs] * a.ld + mcol) = mvv[u];
}

template <> const void *cluster_panel_entry<BB_T, BB_ROWS>() {
    return reinterpret_cast<const void *>(cluster_panel_kernel<BB_T, BB_ROWS>);
}

}  // namespace bb
