// lu.cuh -- shared by the LU's translation units (lu.cu, cluster_panel.cu).
#pragma once

#include "internal.cuh"

namespace bb {

template <typename T> __device__ __forceinline__ T cabs1(Cx<T> v) { return fabs(v.re) + fabs(v.im); }
// correctly rounded reciprocal (the same value as 1 / x)
__device__ __forceinline__ float rcp_rn(float x) { return __frcp_rn(x); }
__device__ __forceinline__ double rcp_rn(double x) { return __drcp_rn(x); }
template <typename T> __device__ __forceinline__ Cx<T> cms(Cx<T> x, Cx<T> l, Cx<T> u) {  // x - l u
    return Cx<T>{x.re - (l.re * u.re - l.im * u.im), x.im - (l.re * u.im + l.im * u.re)};
}

// The cluster panel kernel (cluster_panel.cu): constants, arguments, shapes.
constexpr int CP_CTAS = 16, CP_THREADS = 256, CP_WARPS = CP_THREADS / 32, CP_ROW_BYTES = 272, CP_SLOTS = 3;
// rows up to which one CTA alone factors the sub-panel: at one row per thread
// it saves the exchange (31 against 44 us a sub-panel in FP32); with two rows
// per thread (49 us) sixteen CTAs of one are faster
constexpr int CP_ONE_CTA = 128;
constexpr int CP_NONE = 0x7fffffff;  // position of "no candidate"

template <typename T> struct ClusterPanelArgs {
    Cx<T> *A;
    int64_t ld;
    int n, k;     // sub-panel: rows [k, n), columns [k, k + W), W = 256 / sizeof(Cx<T>)
    int rpc;      // rows per CTA
    int *ipiv;
    int *status;
    Cx<T> *dinv;  // inverse of the unit lower W x W diagonal block (nullptr: not wanted)
    int xc0, xc1; // the panel's columns: the interchanges go to [xc0, xc1) outside [k, k + W) as well
                  // (xc0 == xc1: the caller swaps the other columns itself)
    uint64_t timeout_ns;
};

template <typename T> struct CpShape {
    static constexpr int W = 256 / sizeof(Cx<T>);        // columns
    static constexpr int NP = W / 2;                      // column pairs
    static constexpr int PB = 256 / NP;                   // bytes of a pair
    static constexpr int KB = sizeof(T) == 4 ? 16 : 32;   // bytes of a key: magnitude, position, reciprocal
    // a slot's row: NP pairs, then the pairs a phase's last columns read past the row's end (unused values)
    static constexpr int RSL = 256 + (NP / 4 - 1) * PB;
    // The interchange of the panel's other columns: at most 2 W moved rows, MVC
    // 16-byte chunks (or fewer) each, MVT values per thread of 128 or more
    static constexpr int MVC = sizeof(T) == 4 ? 64 : 128, MVT = 2 * W * MVC / 128;
    // shared memory for rpc rows on C CTAs
    static size_t smem(int rpc, int C) {
        return (size_t)rpc * CP_ROW_BYTES + (size_t)(RSL + KB) * (CP_SLOTS * C + 2) +
               sizeof(Cx<T>) * 2 * W * (W + 1);
    }
};

// the kernel with RPT rows per thread, one translation unit each (cluster_panel.cu)
template <typename T, int RPT> const void *cluster_panel_entry();

}  // namespace bb
