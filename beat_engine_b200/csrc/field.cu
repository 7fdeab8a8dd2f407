// field.cu -- observation-point pressure and far-field pattern for all right
// hand sides in one pass over the boundary sources.
//
// Reference: build_field_evaluation_cache (src/BeatEngineCore.jl:1770-1810),
// _cuda_weighted_field_sources_kernel! (src/BeatEngineCudaField.jl:161-197),
// _cuda_field_eval_kernel! (:240-327), evaluate_galerkin_field_cpu
// (src/BeatEngineCpuField.jl:1-49):
//     p(x) = sum_src w [ G (ik - 1/r)(r.n / r) p_src - G q_src ],  r = y - x
// The far-field pattern has no reference counterpart; it is the r -> inf limit
// of the same sum with the same signed k:
//     p_inf(d) = sum_src exp(-ik d.y)/(4 pi) [ (-ik)(d.n) p_src - q_src ].
//
// The reference launches one field kernel per excitation and output; here one
// kernel evaluates G once per (point, source) for every column.  A CTA takes
// 32 points and a part of the sources, staged through shared memory in chunks
// that its warps share out; the CTAs add their partial sums with
// red.global.add.  FP64 in both precision forms.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <utility>
#include <vector>

#include "internal.cuh"
#include "phase.cuh"

namespace bb {

constexpr int FLD_CHUNK = 32;    // sources per shared-memory chunk
constexpr int FLD_THREADS = 128;
constexpr int FLD_POINTS = 32;   // points per CTA

struct FieldImages {
    int n;            // copies: the mesh itself, then its symmetry images
    double s[4][3];   // per copy: signs of x, y, z
};

// per source: position, normal, p-density and q-density for R columns, for
// the mesh and each symmetry image (reflected position and normal, the same
// densities); copy ix of source s is entry ix * F Q + s of arrays of stride
// ST = images.n F Q
__global__ void field_sources_kernel(const double *qpts, const double *normals, const double *areas,
                                     const int *faces, int F, int Q, const double *rule_w3, int N,
                                     const double2 *p, const double2 *q, int R, double *ys, double *ns,
                                     double2 *ps, double2 *qs, FieldImages images) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    const int S = F * Q, ST = S * images.n;
    if (s >= S) return;
    const int f = s / Q, qi = s % Q;
    const double w = rule_w3[4 * qi] * 2.0 * areas[f];
    const double b0 = rule_w3[4 * qi + 1], b1 = rule_w3[4 * qi + 2], b2 = rule_w3[4 * qi + 3];
    for (int ix = 0; ix < images.n; ++ix)
        for (int c = 0; c < 3; ++c) {
            ys[3 * ((size_t)ix * S + s) + c] = images.s[ix][c] * qpts[3 * (size_t)s + c];
            ns[3 * ((size_t)ix * S + s) + c] = images.s[ix][c] * normals[3 * f + c];
        }
    const int v0 = faces[3 * f], v1 = faces[3 * f + 1], v2 = faces[3 * f + 2];
    for (int r = 0; r < R; ++r) {
        const double2 a = p[(size_t)r * N + v0], b = p[(size_t)r * N + v1], c = p[(size_t)r * N + v2];
        const double2 pv = make_double2((b0 * a.x + b1 * b.x + b2 * c.x) * w, (b0 * a.y + b1 * b.y + b2 * c.y) * w);
        const double2 qq = q[(size_t)r * F + f];
        const double2 qv = make_double2(qq.x * w, qq.y * w);
        for (int ix = 0; ix < images.n; ++ix) {
            ps[(size_t)r * ST + (size_t)ix * S + s] = pv;
            qs[(size_t)r * ST + (size_t)ix * S + s] = qv;
        }
    }
}

// Green factor (gr, gi) and double-layer factor (dr, di) of one (point,
// source): G and G (ik - 1/r) (r.n) / r, r = y - x; FAR: E = exp(-ik d.y) / 4 pi
// and E (-ik d.n).  Zero at r = 0.
template <bool FAR>
__device__ __forceinline__ void field_factors(const double (&x)[3], const double *y, const double *n, double k,
                                              double &gr, double &gi, double &dr, double &di) {
    const double inv4pi = 0.07957747154594767;
    double s, c;
    if (FAR) {
        sincos_cw(-k * (x[0] * y[0] + x[1] * y[1] + x[2] * y[2]), &s, &c);
        gr = c * inv4pi;
        gi = s * inv4pi;
        const double dn = k * (x[0] * n[0] + x[1] * n[1] + x[2] * n[2]);
        dr = gi * dn;
        di = -gr * dn;
    } else {
        const double rx = y[0] - x[0], ry = y[1] - x[1], rz = y[2] - x[2];
        const double r2 = rx * rx + ry * ry + rz * rz;
        // (the series wants a normal number; r = 0 contributes nothing)
        const double ir = r2 < 2.2250738585072014e-308 ? (r2 == 0.0 ? 0.0 : rsqrt(r2)) : rsqrt_series(r2);
        sincos_cw(k * (r2 * ir), &s, &c);
        const double a = inv4pi * ir, proj = (rx * n[0] + ry * n[1] + rz * n[2]) * ir;
        gr = c * a;
        gi = s * a;
        dr = (-gr * ir - gi * k) * proj;
        di = (gr * k - gi * ir) * proj;
    }
}

__device__ __forceinline__ void field_point(const double *pts, int m, int M, bool unit, double (&x)[3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) x[i] = m < M ? pts[3 * (size_t)m + i] : (i == 0 ? 1.0 : 0.0);
    if (unit) {
        const double nn = sqrt(x[0] * x[0] + x[1] * x[1] + x[2] * x[2]);
#pragma unroll
        for (int i = 0; i < 3; ++i) x[i] /= nn;
    }
}

// Up to two right-hand sides: a lane per point, the warps take every fourth
// source.  Bound: the FP64 units, about 45 + 8 RC instructions per (point,
// source).
template <bool FAR, int RC>
__global__ void __launch_bounds__(FLD_THREADS) field_eval_kernel(const double *pts, int M, const double *ys,
                                                                 const double *ns, const double2 *ps,
                                                                 const double2 *qs, int S, int R, int r0,
                                                                 int per_cta, double k, double2 *out) {
    __shared__ __align__(16) double sg[FLD_CHUNK][6];  // y, n
    __shared__ double2 sp[FLD_CHUNK][RC], sq[FLD_CHUNK][RC];
    __shared__ double2 part[FLD_THREADS / 32][RC][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int m = blockIdx.x * FLD_POINTS + lane;
    const int s_begin = blockIdx.y * per_cta, s_end = min(S, s_begin + per_cta);
    double x[3];
    field_point(pts, m, M, FAR, x);
    double ar[RC], ai[RC];
#pragma unroll
    for (int r = 0; r < RC; ++r) ar[r] = ai[r] = 0.0;
    for (int c0 = s_begin; c0 < s_end; c0 += FLD_CHUNK) {
        const int cn = min(FLD_CHUNK, s_end - c0);
        __syncthreads();
        for (int i = threadIdx.x; i < cn * 3; i += FLD_THREADS) {
            sg[i / 3][i % 3] = ys[3 * (size_t)c0 + i];
            sg[i / 3][3 + i % 3] = ns[3 * (size_t)c0 + i];
        }
        for (int i = threadIdx.x; i < RC * FLD_CHUNK; i += FLD_THREADS) {
            const int r = i / FLD_CHUNK, j = i % FLD_CHUNK;
            const bool ok = r0 + r < R && j < cn;
            sp[j][r] = ok ? ps[(size_t)(r0 + r) * S + c0 + j] : make_double2(0, 0);
            sq[j][r] = ok ? qs[(size_t)(r0 + r) * S + c0 + j] : make_double2(0, 0);
        }
        __syncthreads();
#pragma unroll 2
        for (int j = warp; j < cn; j += FLD_THREADS / 32) {
            double gr, gi, dr, di;
            field_factors<FAR>(x, sg[j], sg[j] + 3, k, gr, gi, dr, di);
#pragma unroll
            for (int r = 0; r < RC; ++r) {
                const double2 pv = sp[j][r], qv = sq[j][r];
                ar[r] += dr * pv.x - di * pv.y - (gr * qv.x - gi * qv.y);
                ai[r] += dr * pv.y + di * pv.x - (gr * qv.y + gi * qv.x);
            }
        }
    }
#pragma unroll
    for (int r = 0; r < RC; ++r) part[warp][r][lane] = make_double2(ar[r], ai[r]);
    __syncthreads();
    for (int i = threadIdx.x; i < RC * 32; i += FLD_THREADS) {
        const int r = i / 32, mm = blockIdx.x * FLD_POINTS + i % 32;
        double2 v = make_double2(0, 0);
#pragma unroll
        for (int w = 0; w < FLD_THREADS / 32; ++w) {
            v.x += part[w][r][i % 32].x;
            v.y += part[w][r][i % 32].y;
        }
        if (mm < M && r0 + r < R) {
            atomicAdd(&out[(size_t)(r0 + r) * M + mm].x, v.x);
            atomicAdd(&out[(size_t)(r0 + r) * M + mm].y, v.y);
        }
    }
}

// Three and more right-hand sides: the sums over the sources are a real matrix
// product, points x (4 factors per source) times (4 per source) x (2 R), on
// the FP64 tensor cores (mma.sync.m8n8k4.f64; operand places as in the LU's
// FP64 update).  A warp takes 8 points x 4 sources at a time: lane (g, t)
// evaluates point g and source t once, and its factor i (dr, di, gr, gi) is its
// A operand of the i-th product, whose K index is the source; the B operand is
// then row i of source t,
//     p, ip (real parts of i p), -q, -iq,   columns (re, im) of each side,
// staged once per chunk.  So neither factors nor sums move between lanes.
// NB: blocks of 8 real columns, 4 NB right-hand sides.  Each warp holds PG
// groups of 8 points.  The four products of four sources are summed from zero
// and added to the running sum once: with the running sum as their accumulator
// it is rounded 16 times for four sources, and the error against long double was
// 10 % above a thread per point's (F = 11,864, 16 sides: 4.4 -> 4.9e-13; this 4.2).
// Bound: the FP64 units (about 45 + 34 NB FP64 instructions' worth per (point,
// source)); a thread per point with 16 sides in registers read 32 broadcast
// 16-byte values of shared memory per source and was held by those: field at
// 2,000 points, 16 sides, 71,184 sources 2.9 ms, this 2.2.  Three CTAs per SM
// with 16 sides, by registers.
constexpr int FLD_PG = FLD_POINTS / 8;
template <int NB> struct FieldB {
    static constexpr int LD = NB == 1 ? 8 : 8 * NB + 8;  // row stride: 8 mod 16 doubles, two wavefronts a load
};
template <bool FAR, int NB>
__global__ void __launch_bounds__(FLD_THREADS, NB == 4 ? 3 : 4) field_mma_kernel(const double *pts, int M, const double *ys,
                                                                const double *ns, const double2 *ps,
                                                                const double2 *qs, int S, int R, int r0, int per_cta,
                                                                double k, double2 *out) {
    constexpr int RC = 4 * NB, LD = FieldB<NB>::LD, WARPS = FLD_THREADS / 32, PART = 2 * RC + 1;
    __shared__ double sg[FLD_CHUNK][7];  // y, n; odd stride
    union Chunk {
        double b[4][FLD_CHUNK * LD];               // B rows of the chunk's sources
        double part[WARPS][FLD_POINTS * PART / 2];  // (half the warps' sums at a time)
    };
    __shared__ Chunk ch;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int s_begin = blockIdx.y * per_cta, s_end = min(S, s_begin + per_cta);
    double x[FLD_PG][3], c[FLD_PG][NB][2];
#pragma unroll
    for (int a = 0; a < FLD_PG; ++a) {
        field_point(pts, blockIdx.x * FLD_POINTS + 8 * a + g, M, FAR, x[a]);
#pragma unroll
        for (int b = 0; b < NB; ++b) c[a][b][0] = c[a][b][1] = 0.0;
    }
    for (int c0 = s_begin; c0 < s_end; c0 += FLD_CHUNK) {
        const int cn = min(FLD_CHUNK, s_end - c0);
        __syncthreads();
        for (int i = threadIdx.x; i < FLD_CHUNK * 3; i += FLD_THREADS) {
            const bool ok = i < cn * 3;
            sg[i / 3][i % 3] = ok ? ys[3 * (size_t)c0 + i] : 0.0;
            sg[i / 3][3 + i % 3] = ok ? ns[3 * (size_t)c0 + i] : 0.0;
        }
        for (int i = threadIdx.x; i < RC * FLD_CHUNK; i += FLD_THREADS) {
            const int r = i / FLD_CHUNK, j = i % FLD_CHUNK;
            const bool ok = r0 + r < R && j < cn;
            const double2 p = ok ? ps[(size_t)(r0 + r) * S + c0 + j] : make_double2(0, 0);
            const double2 q = ok ? qs[(size_t)(r0 + r) * S + c0 + j] : make_double2(0, 0);
            const int o = j * LD + 2 * r;
            ch.b[0][o] = p.x, ch.b[0][o + 1] = p.y;
            ch.b[1][o] = -p.y, ch.b[1][o + 1] = p.x;
            ch.b[2][o] = -q.x, ch.b[2][o + 1] = -q.y;
            ch.b[3][o] = q.y, ch.b[3][o + 1] = -q.x;
        }
        __syncthreads();
        for (int j0 = 4 * warp; j0 < cn; j0 += 4 * WARPS) {
            const double *sj = sg[j0 + t];
            const double y[3] = {sj[0], sj[1], sj[2]}, n[3] = {sj[3], sj[4], sj[5]};
            double f[FLD_PG][4];
#pragma unroll
            for (int a = 0; a < FLD_PG; ++a) field_factors<FAR>(x[a], y, n, k, f[a][2], f[a][3], f[a][0], f[a][1]);
            if (j0 + 4 > cn && j0 + t >= cn) {  // past the last source
#pragma unroll
                for (int a = 0; a < FLD_PG; ++a)
#pragma unroll
                    for (int i = 0; i < 4; ++i) f[a][i] = 0.0;
            }
#pragma unroll
            for (int b = 0; b < NB; ++b) {
                double bv[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) bv[i] = ch.b[i][(j0 + t) * LD + 8 * b + g];
#pragma unroll
                for (int a = 0; a < FLD_PG; ++a) {
                    double d[2] = {0.0, 0.0};  // four sources' sum, apart from the others'
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                            : "+d"(d[0]), "+d"(d[1])
                            : "d"(f[a][i]), "d"(bv[i]));
                    c[a][b][0] += d[0];
                    c[a][b][1] += d[1];
                }
            }
        }
    }
    // the warps' sums meet in shared memory, half of the points at a time:
    // lane (g, t) holds point 8 a + g, real columns 8 b + 2 t, 8 b + 2 t + 1
    constexpr int HALF = FLD_PG / 2;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        __syncthreads();
#pragma unroll
        for (int a = 0; a < HALF; ++a)
#pragma unroll
            for (int b = 0; b < NB; ++b)
#pragma unroll
                for (int e = 0; e < 2; ++e)
                    ch.part[warp][(8 * a + g) * PART + 8 * b + 2 * t + e] = c[h * HALF + a][b][e];
        __syncthreads();
        for (int i = threadIdx.x; i < 8 * HALF * 2 * RC; i += FLD_THREADS) {
            const int col = i / (8 * HALF), pt = i % (8 * HALF), r = r0 + col / 2;
            const int m = blockIdx.x * FLD_POINTS + 8 * HALF * h + pt;
            double v = 0.0;
#pragma unroll
            for (int w = 0; w < WARPS; ++w) v += ch.part[w][pt * PART + col];
            if (m < M && r < R) atomicAdd(reinterpret_cast<double *>(&out[(size_t)r * M + m]) + (col & 1), v);
        }
    }
}

// boundary sources of the mesh and its images, staged in c->ws.field
struct StagedSources {
    const double *ys = nullptr, *ns = nullptr, *pts = nullptr;
    const double2 *ps = nullptr, *qs = nullptr;
    const double2 *q = nullptr;  // the Neumann data used (admittance term included)
    int S = 0;                   // sources per column
};

static StagedSources stage_sources(beat_b200_ctx *c, int M, const double *pts_host, int R, const double *p_dev,
                                   const double *q_dev) {
    const int F = c->F, Q = c->Q, N = c->V;
    FieldImages images;
    images.n = 1 + c->nimg;
    for (int i = 0; i < 3; ++i) images.s[0][i] = 1.0;
    for (int ix = 0; ix < c->nimg; ++ix)
        for (int i = 0; i < 3; ++i) images.s[1 + ix][i] = c->img_sign[ix][i];
    const int S = F * Q * images.n;  // sources of the mesh and its images
    if (c->adm_set) {  // the boundary's Neumann data include the admittance term
        c->ws.qeff.alloc(sizeof(double2) * (size_t)F * R);
        effective_neumann(c, R, p_dev, q_dev, c->ws.qeff.as<double>());
        q_dev = c->ws.qeff.as<double>();
    }
    // rule weight + basis per point
    std::vector<double> rw3(4 * (size_t)Q);
    for (int q = 0; q < Q; ++q) {
        rw3[4 * q] = c->rule_w[q];
        rw3[4 * q + 1] = 1.0 - c->rule_pts[2 * q] - c->rule_pts[2 * q + 1];
        rw3[4 * q + 2] = c->rule_pts[2 * q];
        rw3[4 * q + 3] = c->rule_pts[2 * q + 1];
    }
    DevBuf &scratch = c->ws.field;  // kept across calls: no allocation on the steady path
    // doubles before the double2 arrays, rounded up to an even count so the
    // double2 arrays start on a 16-byte boundary
    const size_t nd = (4 * (size_t)Q + 6 * (size_t)S + 3 * (size_t)M + 1) & ~(size_t)1;
    const size_t bytes = sizeof(double) * nd + sizeof(double2) * 2 * (size_t)S * R;
    scratch.alloc(bytes);
    double *d_rw = scratch.as<double>();
    double *ys = d_rw + 4 * Q, *ns = ys + 3 * (size_t)S, *d_pts = ns + 3 * (size_t)S;
    double2 *ps = reinterpret_cast<double2 *>(d_rw + nd), *qs = ps + (size_t)S * R;
    BB_CUDA(cudaMemcpyAsync(d_rw, rw3.data(), sizeof(double) * 4 * Q, cudaMemcpyHostToDevice, c->stream));
    BB_CUDA(cudaMemcpyAsync(d_pts, pts_host, sizeof(double) * 3 * M, cudaMemcpyHostToDevice, c->stream));
    field_sources_kernel<<<(F * Q + 255) / 256, 256, 0, c->stream>>>(
        c->d_qpts.as<double>(), c->d_normals.as<double>(), c->d_areas.as<double>(), c->d_faces.as<int>(), F, Q, d_rw,
        N, reinterpret_cast<const double2 *>(p_dev), reinterpret_cast<const double2 *>(q_dev), R, ys, ns, ps, qs,
        images);
    BB_CUDA(cudaGetLastError());
    StagedSources st;
    st.ys = ys;
    st.ns = ns;
    st.pts = d_pts;
    st.ps = ps;
    st.qs = qs;
    st.q = reinterpret_cast<const double2 *>(q_dev);
    st.S = S;
    return st;
}

// The source range in as many parts as fill whole waves of resident CTAs best
// (a part has at least two chunks; with four, one point's gradient at F = 300
// took 79 us instead of 76, ten points' 78 instead of 67): with 63 tiles of points and 444 CTAs
// resident, 9 parts leave the second wave 28 % full (2.68 ms for the product
// kernel above with one running sum), 7 make one wave (2.05 ms).
struct SourceSplit {
    dim3 grid;
    int per;  // sources per CTA
};
template <typename K> static SourceSplit resident_split(const beat_b200_ctx *c, K *kernel, int M, int S) {
    int per_sm = 1;
    BB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, FLD_THREADS, 0));
    const int mt = (M + FLD_POINTS - 1) / FLD_POINTS, chunks = (S + FLD_CHUNK - 1) / FLD_CHUNK;
    const int per = chunks_per_slice(mt, chunks, (int64_t)std::max(1, per_sm) * c->sm_count, 2) * FLD_CHUNK;
    return {dim3(mt, (S + per - 1) / per), per};
}

void farfield(beat_b200_ctx *c, double k, int M, const double *pts_host, int R, const double *p_dev,
              const double *q_dev, double *out_dev, bool far) {
    BB_REQUIRE(c->F > 0, BEAT_B200_STATE, "no mesh: call beat_b200_set_mesh first");
    BB_REQUIRE(M >= 0 && R >= 1, BEAT_B200_INVALID_ARG, "field: M must be >= 0 and R >= 1");
    if (M == 0) return;
    const StagedSources st = stage_sources(c, M, pts_host, R, p_dev, q_dev);
    BB_CUDA(cudaMemsetAsync(out_dev, 0, sizeof(double2) * (size_t)M * R, c->stream));
    // by the columns left: one or two in registers (the products would spend 8
    // real columns on 2 or 4: 45 + 32 against 45 + 8 instructions for one),
    // then products of 4, 8 and 16
    auto pass = [&](auto *kernel, int r0) {
        const SourceSplit sp = resident_split(c, kernel, M, st.S);
        kernel<<<sp.grid, FLD_THREADS, 0, c->stream>>>(st.pts, M, st.ys, st.ns, st.ps, st.qs, st.S, R, r0, sp.per, k,
                                                       reinterpret_cast<double2 *>(out_dev));
        BB_CUDA(cudaGetLastError());
    };
    for (int r0 = 0; r0 < R; r0 += 16) {
        const int left = R - r0;
        if (left == 1)
            pass(far ? field_eval_kernel<true, 1> : field_eval_kernel<false, 1>, r0);
        else if (left == 2)
            pass(far ? field_eval_kernel<true, 2> : field_eval_kernel<false, 2>, r0);
        else if (left <= 4)
            pass(far ? field_mma_kernel<true, 1> : field_mma_kernel<false, 1>, r0);
        else if (left <= 8)
            pass(far ? field_mma_kernel<true, 2> : field_mma_kernel<false, 2>, r0);
        else
            pass(far ? field_mma_kernel<true, 4> : field_mma_kernel<false, 4>, r0);
    }
    BB_CUDA(cudaStreamSynchronize(c->stream));
}

// ---------------------------------------------------------------------------
// pressure and its gradient (pressure_gradient_v1)
//
// Reference: field_value_gradient, _gradient_triangle,
// _adaptive_gradient_triangle, correct_field_gradient!,
// evaluate_galerkin_field_gradient_cpu (src/BeatEngineFieldGradient.jl:1-88),
// evaluate_galerkin_field_gradient_cuda (src/BeatEngineCudaFieldGradient.jl:
// 1-38).  With r = y - x, u = r / |r|, G = exp(ik|r|) / (4 pi |r|),
// a = ik - 1/|r|, b = 3/|r|^2 - k^2 - 3ik/|r|:
//     value    = G (a (u.n) p - q)
//     gradient = G (a q u - p (b (u.n) u + (a / |r|) n))
// summed over the regular sources, then for every face (and symmetry image)
// whose centroid lies within 3 diameters of the point, the face's regular
// contribution is replaced by adaptive quadrature: the face is split into
// four by its edge midpoints until a piece's diameter is at most 0.4 x the
// distance from the point to its centroid and |k| x diameter <= 0.7, each
// leaf taking the fourth-order rule; a piece still too large at depth 12
// means the point is too close to the boundary (an error, as in the
// reference).  The reference runs that correction on host threads after the
// device sum; here both run on the device, the correction one warp per (point,
// near face) with an explicit subdivision stack, a piece per lane.
//
// Output layout: M x 4 x R complex, column-major, component d (0 value,
// 1..3 d/dx, d/dy, d/dz) of column r at out[m + M (d + 4 r)].
// ---------------------------------------------------------------------------
constexpr int FG_RC = 4;          // right-hand sides per pass
constexpr int FG_CHUNK = 32;
constexpr int FG_THREADS = 128;
constexpr int FG_MAX_DEPTH = 12;
constexpr int FG_STACK = 32 * (3 * FG_MAX_DEPTH + 1);  // pending pieces of a split taken 32 at a time, at most
constexpr int FG_NEAR_WARPS = 2;                     // near pairs per CTA of the correction
constexpr int FG_SCALE = 1 << FG_MAX_DEPTH;      // piece vertices are multiples of 1/4096 in face coordinates
constexpr long long FG_PIECE_BUDGET = 1 << 22;   // pieces per (point, face): a bound on runaway refinement
constexpr int FG_ERR_TOO_CLOSE = 1, FG_ERR_BUDGET = 2;

struct GradRule {
    int n;
    double w[8];      // weights (summing to 1/2)
    double b[8][3];   // barycentric coordinates of the points
};

// contribution of one source (weight w) to value + gradient of rc columns;
// P[c], Qn[c]: p and q of column c at the source
template <int RC>
__device__ __forceinline__ void grad_source(double x0, double x1, double x2, double y0, double y1, double y2, double n0,
                                            double n1, double n2, double w, double k, const double2 *P,
                                            const double2 *Qn, double (&acc)[RC][8]) {
    const double rx = y0 - x0, ry = y1 - x1, rz = y2 - x2;
    const double r2 = rx * rx + ry * ry + rz * rz;
    if (r2 == 0.0) return;
    const double ir = r2 < 2.2250738585072014e-308 ? rsqrt(r2) : rsqrt_series(r2), rad = r2 * ir;
    const double u[3] = {rx * ir, ry * ir, rz * ir}, nn[3] = {n0, n1, n2};
    double sn_, cs_;
    sincos_cw(k * rad, &sn_, &cs_);
    const double gs = w * 0.07957747154594767 * ir;
    const double gr = cs_ * gs, gi = sn_ * gs;
    // Ga = G a, a = (-1/r, k); Gb = G b, b = (3/r^2 - k^2, -3k/r)
    const double gar = -gr * ir - gi * k, gai = gr * k - gi * ir;
    const double br = 3.0 * ir * ir - k * k, bi = -3.0 * k * ir;
    const double gbr = gr * br - gi * bi, gbi = gr * bi + gi * br;
    const double proj = u[0] * n0 + u[1] * n1 + u[2] * n2;
    double cdr[3], cdi[3];  // G b proj u_d + G a n_d / r
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        cdr[d] = gbr * proj * u[d] + gar * ir * nn[d];
        cdi[d] = gbi * proj * u[d] + gai * ir * nn[d];
    }
#pragma unroll
    for (int cc = 0; cc < RC; ++cc) {
        const double2 p = P[cc], q = Qn[cc];
        acc[cc][0] += (gar * p.x - gai * p.y) * proj - (gr * q.x - gi * q.y);
        acc[cc][1] += (gar * p.y + gai * p.x) * proj - (gr * q.y + gi * q.x);
        const double aqr = gar * q.x - gai * q.y, aqi = gar * q.y + gai * q.x;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            acc[cc][2 + 2 * d] += u[d] * aqr - (cdr[d] * p.x - cdi[d] * p.y);
            acc[cc][3 + 2 * d] += u[d] * aqi - (cdr[d] * p.y + cdi[d] * p.x);
        }
    }
}

// regular sum over the staged sources (weights and densities premultiplied):
// a lane per point, the CTA's warps take every fourth source, as in the field
template <int RC>
__global__ void __launch_bounds__(FG_THREADS) field_grad_kernel(const double *pts, int M, const double *ys,
                                                                const double *ns, const double2 *ps,
                                                                const double2 *qs, int S, int R, int r0, int per_cta,
                                                                double k, double2 *out) {
    __shared__ double sg[FG_CHUNK][6];  // y, n
    __shared__ double2 sp[FG_CHUNK][RC], sq[FG_CHUNK][RC];
    __shared__ double part[FG_THREADS / 32][RC * 8][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int m = blockIdx.x * FLD_POINTS + lane;
    const int s_begin = blockIdx.y * per_cta, s_end = min(S, s_begin + per_cta);
    double x[3];
    field_point(pts, m, M, false, x);
    double acc[RC][8];
#pragma unroll
    for (int r = 0; r < RC; ++r)
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[r][e] = 0.0;
    for (int c0 = s_begin; c0 < s_end; c0 += FG_CHUNK) {
        const int cn = min(FG_CHUNK, s_end - c0);
        __syncthreads();
        for (int i = threadIdx.x; i < cn * 3; i += FG_THREADS) {
            sg[i / 3][i % 3] = ys[3 * (size_t)c0 + i];
            sg[i / 3][3 + i % 3] = ns[3 * (size_t)c0 + i];
        }
        for (int i = threadIdx.x; i < RC * FG_CHUNK; i += FG_THREADS) {
            const int r = i / FG_CHUNK, j = i % FG_CHUNK;
            const bool ok = r0 + r < R && j < cn;
            sp[j][r] = ok ? ps[(size_t)(r0 + r) * S + c0 + j] : make_double2(0, 0);
            sq[j][r] = ok ? qs[(size_t)(r0 + r) * S + c0 + j] : make_double2(0, 0);
        }
        __syncthreads();
#pragma unroll 2
        for (int j = warp; j < cn; j += FG_THREADS / 32)
            grad_source<RC>(x[0], x[1], x[2], sg[j][0], sg[j][1], sg[j][2], sg[j][3], sg[j][4], sg[j][5], 1.0, k,
                            sp[j], sq[j], acc);
    }
#pragma unroll
    for (int r = 0; r < RC; ++r)
#pragma unroll
        for (int e = 0; e < 8; ++e) part[warp][8 * r + e][lane] = acc[r][e];
    __syncthreads();
    for (int i = threadIdx.x; i < RC * 8 * 32; i += FG_THREADS) {
        const int e = i / 32, mm = blockIdx.x * FLD_POINTS + i % 32, r = r0 + e / 8, d = e % 8 / 2;
        double v = 0.0;
#pragma unroll
        for (int w = 0; w < FG_THREADS / 32; ++w) v += part[w][e][i % 32];
        if (mm < M && r < R)
            atomicAdd(reinterpret_cast<double *>(&out[(size_t)mm + (size_t)M * (d + 4 * (size_t)r)]) + (e & 1), v);
    }
}

__device__ __forceinline__ void face_corners(const double *verts, const int *faces, int f, const double *sg,
                                             double (&v)[3][3]) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const int vi = faces[3 * f + a];
#pragma unroll
        for (int d = 0; d < 3; ++d) v[a][d] = sg[d] * verts[3 * (size_t)vi + d];
    }
}

__device__ __forceinline__ double tri_diameter(const double (&v)[3][3]) {
    double e[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const int b = (a + 1) % 3;
        const double dx = v[a][0] - v[b][0], dy = v[a][1] - v[b][1], dz = v[a][2] - v[b][2];
        e[a] = sqrt(dx * dx + dy * dy + dz * dz);
    }
    return fmax(fmax(e[0], e[1]), e[2]);
}

__device__ __forceinline__ double dist_to_centroid(const double (&v)[3][3], double x0, double x1, double x2) {
    const double cx = (v[0][0] + v[1][0] + v[2][0]) / 3.0, cy = (v[0][1] + v[1][1] + v[2][1]) / 3.0,
                 cz = (v[0][2] + v[1][2] + v[2][2]) / 3.0;
    const double dx = x0 - cx, dy = x1 - cy, dz = x2 - cz;
    return sqrt(dx * dx + dy * dy + dz * dz);
}

// (point, face copy) pairs with the face's centroid within 3 diameters of the
// point; item = m * (F * copies) + copy * F + f, written while slots last.  A
// thread per face copy, so that its diameter and centroid are formed once, and
// a part of the points per blockIdx.y.
__global__ void near_pairs_kernel(const double *pts, int M, const double *verts, const int *faces, int F,
                                  FieldImages images, int per, long long *items, long long cap,
                                  unsigned long long *count) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= F * images.n) return;
    double v[3][3];
    face_corners(verts, faces, e % F, images.s[e / F], v);
    const double reach = 3.0 * tri_diameter(v), bound = 1.000001 * reach * reach;
    const double cx = (v[0][0] + v[1][0] + v[2][0]) / 3.0, cy = (v[0][1] + v[1][1] + v[2][1]) / 3.0,
                 cz = (v[0][2] + v[1][2] + v[2][2]) / 3.0;
    const int m1 = min(M, ((int)blockIdx.y + 1) * per);
    for (int m = blockIdx.y * per; m < m1; ++m) {
        const double dx = pts[3 * m] - cx, dy = pts[3 * m + 1] - cy, dz = pts[3 * m + 2] - cz;
        const double d2 = dx * dx + dy * dy + dz * dz;
        if (d2 <= bound && sqrt(d2) <= reach) {
            const unsigned long long slot = atomicAdd(count, 1ull);
            if ((long long)slot < cap) items[slot] = (long long)m * F * images.n + e;
        }
    }
}

// Adds adaptive - regular for every near pair of columns [r0, r0 + RC), r0 =
// RC blockIdx.y: a warp per pair, grid-strided over the *count listed pairs
// (nothing is done when the list overflowed its cap).  The split's pending
// pieces are a stack in shared memory; each round the warp takes up to 32 from
// its top, a lane each: a leaf is integrated, another piece leaves its four
// children.  (One thread per pair walked its pieces alone: 0.78 ms for 2,300
// pairs, this 0.05.)
template <int RC>
__global__ void __launch_bounds__(32 * FG_NEAR_WARPS) near_correction_kernel(
    const double *pts, int M, const double *verts, const int *faces, const double *normals, int F, int N,
    FieldImages images, const long long *items, const unsigned long long *count, long long cap, const double2 *p,
    const double2 *q, int R, GradRule coarse, GradRule fine, double k, double2 *out, int *err) {
    // a piece: three corners in face coordinates, multiples of 1/4096 while
    // depth <= 12 (so exact in 16-bit integers)
    struct Piece {
        unsigned short c[3][2];
        unsigned short depth;
    };
    __shared__ Piece stacks[FG_NEAR_WARPS][FG_STACK];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    Piece *stack = stacks[warp];
    const int r0 = blockIdx.y * RC, rc = min(RC, R - r0);
    const long long nitems = (long long)*count;
    if (nitems > cap) return;
    for (long long it = (long long)blockIdx.x * FG_NEAR_WARPS + warp; it < nitems;
         it += (long long)gridDim.x * FG_NEAR_WARPS) {
        const long long t = items[it];
        const int f = (int)(t % F);
        const long long rest = t / F;
        const int ix = (int)(rest % images.n), m = (int)(rest / images.n);
        const double *sg = images.s[ix];
        const double x0 = pts[3 * m], x1 = pts[3 * m + 1], x2 = pts[3 * m + 2];
        double v[3][3];
        face_corners(verts, faces, f, sg, v);
        const double n0 = sg[0] * normals[3 * f], n1 = sg[1] * normals[3 * f + 1], n2 = sg[2] * normals[3 * f + 2];
        double2 pv[3][RC], qv[RC];
#pragma unroll
        for (int cc = 0; cc < RC; ++cc) {
            const bool ok = cc < rc;
#pragma unroll
            for (int a = 0; a < 3; ++a)
                pv[a][cc] = ok ? p[(size_t)(r0 + cc) * N + faces[3 * f + a]] : make_double2(0, 0);
            qv[cc] = ok ? q[(size_t)(r0 + cc) * F + f] : make_double2(0, 0);
        }
        const double e1[3] = {v[1][0] - v[0][0], v[1][1] - v[0][1], v[1][2] - v[0][2]};
        const double e2[3] = {v[2][0] - v[0][0], v[2][1] - v[0][1], v[2][2] - v[0][2]};
        double acc[RC][8];  // adaptive minus regular, this lane's part
#pragma unroll
        for (int cc = 0; cc < RC; ++cc)
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[cc][e] = 0.0;

        // points [j0, j1) of the rule (scaled by sign) on the piece with
        // corners pc, which are s[0..2] in face coordinates
        auto integrate = [&](const double (&pc)[3][3], const double (&s)[3][2], const GradRule &rule, double sign,
                             int j0, int j1) {
            const double a1[3] = {pc[1][0] - pc[0][0], pc[1][1] - pc[0][1], pc[1][2] - pc[0][2]};
            const double a2[3] = {pc[2][0] - pc[0][0], pc[2][1] - pc[0][1], pc[2][2] - pc[0][2]};
            const double cx = a1[1] * a2[2] - a1[2] * a2[1], cy = a1[2] * a2[0] - a1[0] * a2[2],
                         cz = a1[0] * a2[1] - a1[1] * a2[0];
            const double jac = sqrt(cx * cx + cy * cy + cz * cz);
            for (int j = j0; j < j1; ++j) {
                const double b0 = rule.b[j][0], b1 = rule.b[j][1], b2 = rule.b[j][2];
                const double y0 = b0 * pc[0][0] + b1 * pc[1][0] + b2 * pc[2][0];
                const double y1 = b0 * pc[0][1] + b1 * pc[1][1] + b2 * pc[2][1];
                const double y2 = b0 * pc[0][2] + b1 * pc[1][2] + b2 * pc[2][2];
                // P1 basis of the face at the point
                const double xi = b0 * s[0][0] + b1 * s[1][0] + b2 * s[2][0];
                const double et = b0 * s[0][1] + b1 * s[1][1] + b2 * s[2][1];
                const double l0 = 1.0 - xi - et;
                double2 P[RC];
#pragma unroll
                for (int cc = 0; cc < RC; ++cc)
                    P[cc] = make_double2(l0 * pv[0][cc].x + xi * pv[1][cc].x + et * pv[2][cc].x,
                                         l0 * pv[0][cc].y + xi * pv[1][cc].y + et * pv[2][cc].y);
                grad_source<RC>(x0, x1, x2, y0, y1, y2, n0, n1, n2, sign * jac * rule.w[j], k, P, qv, acc);
            }
        };

        if (lane < coarse.n) {  // the regular rule on the whole face, a point per lane: what the regular sum added
            const double s[3][2] = {{0, 0}, {1, 0}, {0, 1}};
            integrate(v, s, coarse, -1.0, lane, lane + 1);
        }
        __syncwarp();
        if (lane == 0) stack[0] = Piece{{{0, 0}, {FG_SCALE, 0}, {0, FG_SCALE}}, 0};
        int top = 1;
        long long pieces = 0;
        const double inv = 1.0 / FG_SCALE;
        bool failed = false;
        while (top > 0) {
            __syncwarp();
            const int take = min(top, 32);
            top -= take;
            Piece pc;
            bool split = false;
            if (lane < take) {
                pc = stack[top + lane];
                double s[3][2], g[3][3];
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    s[a][0] = pc.c[a][0] * inv;
                    s[a][1] = pc.c[a][1] * inv;
#pragma unroll
                    for (int d = 0; d < 3; ++d) g[a][d] = v[0][d] + s[a][0] * e1[d] + s[a][1] * e2[d];
                }
                const double diam = tri_diameter(g);
                split = !(diam <= 0.4 * dist_to_centroid(g, x0, x1, x2) && fabs(k) * diam <= 0.7);
                if (!split) integrate(g, s, fine, 1.0, 0, fine.n);
            }
            const unsigned mask = __ballot_sync(0xffffffffu, split);
            if (__ballot_sync(0xffffffffu, split && pc.depth >= FG_MAX_DEPTH)) {
                if (lane == 0) atomicOr(err, FG_ERR_TOO_CLOSE);
                failed = true;
                break;
            }
            pieces += __popc(mask);
            if (pieces > FG_PIECE_BUDGET) {
                if (lane == 0) atomicOr(err, FG_ERR_BUDGET);
                failed = true;
                break;
            }
            __syncwarp();  // the popped pieces are read: their places may be written
            if (split) {
                unsigned short mid[3][2];  // ab, bc, ca
#pragma unroll
                for (int a = 0; a < 3; ++a)
#pragma unroll
                    for (int d = 0; d < 2; ++d)
                        mid[a][d] = (unsigned short)((pc.c[a][d] + pc.c[(a + 1) % 3][d]) / 2);
                const unsigned short dd = pc.depth + 1;
                Piece *to = stack + top + 4 * __popc(mask & ((1u << lane) - 1u));
                // children (a, ab, ca), (ab, b, bc), (ca, bc, c), (ab, bc, ca)
                to[0] = Piece{{{mid[0][0], mid[0][1]}, {mid[1][0], mid[1][1]}, {mid[2][0], mid[2][1]}}, dd};
                to[1] = Piece{{{mid[2][0], mid[2][1]}, {mid[1][0], mid[1][1]}, {pc.c[2][0], pc.c[2][1]}}, dd};
                to[2] = Piece{{{mid[0][0], mid[0][1]}, {pc.c[1][0], pc.c[1][1]}, {mid[1][0], mid[1][1]}}, dd};
                to[3] = Piece{{{pc.c[0][0], pc.c[0][1]}, {mid[0][0], mid[0][1]}, {mid[2][0], mid[2][1]}}, dd};
            }
            top += 4 * __popc(mask);
        }
        if (failed) continue;
#pragma unroll
        for (int cc = 0; cc < RC; ++cc)
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                double a = acc[cc][e];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
                if (lane == 0 && cc < rc)
                    atomicAdd(reinterpret_cast<double *>(
                                  &out[(size_t)m + (size_t)M * (e / 2 + 4 * (size_t)(r0 + cc))]) +
                                  (e & 1),
                              a);
            }
    }
}

static GradRule grad_rule(const std::vector<double> &pts, const std::vector<double> &w) {
    GradRule r{};
    r.n = (int)w.size();
    for (int j = 0; j < r.n; ++j) {
        r.w[j] = w[j];
        r.b[j][0] = 1.0 - pts[2 * j] - pts[2 * j + 1];
        r.b[j][1] = pts[2 * j];
        r.b[j][2] = pts[2 * j + 1];
    }
    return r;
}

void field_gradient(beat_b200_ctx *c, double k, int M, const double *pts_host, int R, const double *p_dev,
                    const double *q_dev, double *out_dev) {
    BB_REQUIRE(c->F > 0, BEAT_B200_STATE, "no mesh: call beat_b200_set_mesh first");
    BB_REQUIRE(M >= 0 && R >= 1, BEAT_B200_INVALID_ARG, "field gradient: M must be >= 0 and R >= 1");
    if (M == 0) return;
    const int F = c->F, N = c->V;
    const StagedSources st = stage_sources(c, M, pts_host, R, p_dev, q_dev);
    double2 *out = reinterpret_cast<double2 *>(out_dev);
    BB_CUDA(cudaMemsetAsync(out, 0, sizeof(double2) * 4 * (size_t)M * R, c->stream));
    auto regular = [&](auto *kernel, int r0) {
        const SourceSplit sp = resident_split(c, kernel, M, st.S);
        kernel<<<sp.grid, FG_THREADS, 0, c->stream>>>(st.pts, M, st.ys, st.ns, st.ps, st.qs, st.S, R, r0, sp.per, k,
                                                      out);
        BB_CUDA(cudaGetLastError());
    };
    for (int r0 = 0; r0 < R; r0 += FG_RC) regular(R == 1 ? field_grad_kernel<1> : field_grad_kernel<FG_RC>, r0);
    FieldImages images;
    images.n = 1 + c->nimg;
    for (int i = 0; i < 3; ++i) images.s[0][i] = 1.0;
    for (int ix = 0; ix < c->nimg; ++ix)
        for (int i = 0; i < 3; ++i) images.s[1 + ix][i] = c->img_sign[ix][i];
    // near pairs listed, then corrected, without a wait between: the correction
    // reads the count on the device and does nothing when the list overflowed;
    // then both run once more with room for every pair
    DevBuf &nb = c->ws.grad;  // [count u64][error int, pad][items i64 ...], grow-only
    const size_t head = 16;
    long long cap = nb.bytes > head ? (long long)((nb.bytes - head) / sizeof(long long)) : 0;
    if (cap < 1024) {
        nb.alloc(head + 1024 * sizeof(long long));
        cap = 1024;
    }
    std::vector<double> p4, w4;
    triangle_rule(4, p4, w4);
    const GradRule coarse = grad_rule(c->rule_pts, c->rule_w), fine = grad_rule(p4, w4);
    const int face_blocks = (int)(((int64_t)F * images.n + 255) / 256);
    const int parts = std::min(M, std::max(1, 8 * c->sm_count / face_blocks)), per = (M + parts - 1) / parts;
    const int near_blocks = (int)std::min<int64_t>(
        4 * c->sm_count, ((int64_t)M * F * images.n + FG_NEAR_WARPS - 1) / FG_NEAR_WARPS);  // a warp per possible pair
    struct {
        unsigned long long count;
        int err, pad;
    } got{};
    for (int pass = 0; pass < 2; ++pass) {
        BB_CUDA(cudaMemsetAsync(nb.p, 0, head, c->stream));
        unsigned long long *d_count = static_cast<unsigned long long *>(nb.p);
        int *d_err = reinterpret_cast<int *>(static_cast<char *>(nb.p) + 8);
        long long *items = reinterpret_cast<long long *>(static_cast<char *>(nb.p) + head);
        near_pairs_kernel<<<dim3(face_blocks, (M + per - 1) / per), 256, 0, c->stream>>>(
            st.pts, M, c->d_verts.as<double>(), c->d_faces.as<int>(), F, images, per, items, cap, d_count);
        BB_CUDA(cudaGetLastError());
        auto correct = [&](auto *kernel, int groups) {
            kernel<<<dim3(near_blocks, groups), 32 * FG_NEAR_WARPS, 0, c->stream>>>(
                st.pts, M, c->d_verts.as<double>(), c->d_faces.as<int>(), c->d_normals.as<double>(), F, N, images,
                items, d_count, cap, reinterpret_cast<const double2 *>(p_dev), st.q, R, coarse, fine, k, out, d_err);
            BB_CUDA(cudaGetLastError());
        };
        if (R == 1)
            correct(near_correction_kernel<1>, 1);
        else
            correct(near_correction_kernel<FG_RC>, (R + FG_RC - 1) / FG_RC);
        static_assert(sizeof(got) == head, "the list's head");
        BB_CUDA(cudaMemcpyAsync(&got, nb.p, head, cudaMemcpyDeviceToHost, c->stream));
        BB_CUDA(cudaStreamSynchronize(c->stream));
        if ((long long)got.count <= cap) break;
        BB_REQUIRE(pass == 0, BEAT_B200_CUDA_ERROR, "field gradient: near-pair list overflowed twice");
        cap = (long long)got.count;
        nb.alloc(head + (size_t)cap * sizeof(long long));
    }
    const int err = got.err;
    BB_REQUIRE(!(err & FG_ERR_TOO_CLOSE), BEAT_B200_INVALID_ARG,
               "field gradient: a point is too close to the boundary for reliable evaluation");
    BB_REQUIRE(!(err & FG_ERR_BUDGET), BEAT_B200_INVALID_ARG,
               "field gradient: adaptive refinement exceeded its piece budget (mesh too coarse for k)");
}

}  // namespace bb
