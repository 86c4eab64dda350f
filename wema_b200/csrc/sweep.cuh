// sweep.cuh - the strips that the DWT kernels sweep (dwt.cu).
//
// A warp owns a strip of 32 Q neighbouring pairs of columns (lane k the
// pairs Q k .. Q k + Q - 1 of the strip, 2 Q neighbouring samples) and sweeps pairs of rows
// from top to bottom.  Both lifting directions run in registers: across
// a row a lane lifts its own samples and takes one neighbour's from the
// next lane per step (a shuffle for 2 Q samples); down the columns each step of
// the lifting keeps its last value, so a pair of rows that enters moves every
// step on by one and a finished pair of rows, two behind, comes out.
// There is no staging, no block barrier and no shared memory but the forward's
// rings of incoming rows and state, which are a warp's own.
//
// Every output depends on samples within 4 of it.  Strips overlap by one
// lane on either side (30 lanes write; the garbage that lane 0 and lane 31 take
// from their missing neighbours moves inward by two pairs), segments of rows by
// two pairs of rows.  Above and below the image the rows are the mirrored
// rows, which lift to the mirrored values, so the column direction has no border
// case; across a row the border's mirror (dwt.c:63-98, 126-160) is a
// select of the lane's own neighbour.
#pragma once

#include "common.cuh"

namespace wema {

constexpr int SW_WARPS = 4;              // warps per CTA
constexpr int SW_THREADS = 32 * SW_WARPS;
constexpr int SW_LANES = 30;             // lanes of a strip that write
constexpr unsigned SW_FULL = 0xffffffffu;

// A CTA's warps take neighbouring strips over the same rows (the samples two
// strips share then come from the first-level cache) where a level has three strips
// or more; of one or two, the warps take a part of the rows each (with two or
// three of them idle, eight 64x8192 streams in colour took 730 us a tick, so 354).
inline __host__ __device__ int sweep_across(int pairs, int q) {   // strips of a CTA side by side: 1, 2 or 4
    return pairs <= SW_LANES * q ? 1 : pairs <= 2 * SW_LANES * q ? 2 : SW_WARPS;
}
inline __host__ __device__ int sweep_groups(int pairs, int q) {
    const int most = sweep_across(pairs, q) * SW_LANES * q;
    return (pairs + most - 1) / most;
}
// this warp's strip and rows of rows a .. b - 1 of a CTA's group of strips
template <bool NARROW>
struct WarpRows {
    int strip, ya, yb;
    __device__ __forceinline__ WarpRows(int group, int across, int a, int b) {
        const int w = threadIdx.x >> 5;
        if constexpr (NARROW) {
            const int down = SW_WARPS / across, r = w / across;
            strip = group * across + w % across;
            ya = a + (b - a) * r / down;
            yb = a + (b - a) * (r + 1) / down;
        } else {
            strip = group * SW_WARPS + w;
            ya = a;
            yb = b;
        }
    }
};

// strip s of a level of `sw` pairs: its first pair, and the range of its pairs
// (from the first one) that it writes
template <int Q>
struct Strip {
    int p0, lo, hi;
    __device__ __forceinline__ Strip(int s, int sw) {
        const int out = s * SW_LANES * Q;
        p0 = s ? out - Q : 0;
        lo = out - p0;
        hi = min(out + SW_LANES * Q, sw) - p0;
    }
};

// the sample that stands for sample i of a line of n beyond its ends
// (whole-sample mirror); the parity stays
__device__ __forceinline__ int mirror(int i, int n) {
    if (i < 0) i = -i;
    if (i < n) return i;
    if (n == 1) return 0;
    const int p = 2 * (n - 1);
    i %= p;
    return i < n ? i : p - i;
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// One lifting step across a row.  g: the lane's first pair, n the line's length.
// EDGE: the line may end inside a lane (the last pair at any of its places, an
// odd length); else it ends with a lane's last sample or further right.
// predict: o += c (e + right e); update: e += c (left o + o)
template <int Q, bool EDGE>
__device__ __forceinline__ void lift_predict(const float (&e)[Q], float (&o)[Q], float c, int g, int n) {
    const float t = __shfl_down_sync(SW_FULL, e[0], 1);
#pragma unroll
    for (int k = 0; k < Q; k++) {
        float r = k < Q - 1 ? e[k + 1 < Q ? k + 1 : k] : t;
        if (EDGE || k == Q - 1) r = 2 * (g + k) + 2 < n ? r : e[k];
        o[k] = __fmaf_rn(__fadd_rn(e[k], r), c, o[k]);
    }
}
template <int Q, bool EDGE>
__device__ __forceinline__ void lift_update(float (&e)[Q], const float (&o)[Q], float c, int g, int n) {
    const float t = __shfl_up_sync(SW_FULL, o[Q - 1], 1);
#pragma unroll
    for (int k = 0; k < Q; k++) {
        float l = k > 0 ? o[k > 0 ? k - 1 : 0] : t, r = o[k];
        if (k == 0) l = g > 0 ? l : o[0];
        if (EDGE) r = 2 * (g + k) + 1 < n ? r : l;
        e[k] = __fmaf_rn(__fadd_rn(l, r), c, e[k]);
    }
}
template <int Q, bool EDGE>
__device__ __forceinline__ void row_forward(float (&e)[Q], float (&o)[Q], int g, int n) {
    if (EDGE && n < 2) return;
    lift_predict<Q, EDGE>(e, o, kAlpha, g, n);
    lift_update<Q, EDGE>(e, o, kBeta, g, n);
    lift_predict<Q, EDGE>(e, o, kGamma, g, n);
    lift_update<Q, EDGE>(e, o, kDelta, g, n);
#pragma unroll
    for (int k = 0; k < Q; k++) {
        e[k] = __fmul_rn(e[k], kKInv);
        o[k] = __fmul_rn(o[k], kK);
    }
}
template <int Q, bool EDGE>
__device__ __forceinline__ void row_inverse(float (&e)[Q], float (&o)[Q], int g, int n) {
    if (EDGE && n < 2) return;
#pragma unroll
    for (int k = 0; k < Q; k++) {
        e[k] = __fmul_rn(e[k], kK);
        o[k] = __fmul_rn(o[k], kKInv);
    }
    lift_update<Q, EDGE>(e, o, -kDelta, g, n);
    lift_predict<Q, EDGE>(e, o, -kGamma, g, n);
    lift_update<Q, EDGE>(e, o, -kBeta, g, n);
    lift_predict<Q, EDGE>(e, o, -kAlpha, g, n);
}

// The column direction of Q columns, one pair of rows (e, o) at a time; the
// finished pair, two rows of pairs behind, replaces it.  live: the level has at
// least two rows (else its one row passes through).
template <int Q>
struct ColumnInverse {
    float o0[Q], e1[Q], o1[Q], e2[Q];    // odd as entered, even and odd after one step, even finished
    __device__ __forceinline__ void step(float (&e)[Q], float (&o)[Q], bool live) {
#pragma unroll
        for (int k = 0; k < Q; k++) {
            const float a = live ? __fmul_rn(e[k], kK) : e[k], b = __fmul_rn(o[k], kKInv);
            const float ne1 = live ? __fmaf_rn(__fadd_rn(o0[k], b), -kDelta, a) : a;
            const float no1 = __fmaf_rn(__fadd_rn(e1[k], ne1), -kGamma, o0[k]);
            const float ne2 = live ? __fmaf_rn(__fadd_rn(o1[k], no1), -kBeta, e1[k]) : e1[k];
            o[k] = __fmaf_rn(__fadd_rn(e2[k], ne2), -kAlpha, o1[k]);
            e[k] = e2[k];
            o0[k] = b;
            e1[k] = ne1;
            o1[k] = no1;
            e2[k] = ne2;
        }
    }
};
template <int Q>
struct ColumnForward {
    float e0[Q], o0[Q], o1[Q], e1[Q], o2[Q];
    __device__ __forceinline__ void step(float (&e)[Q], float (&o)[Q], bool live) {
#pragma unroll
        for (int k = 0; k < Q; k++) {
            const float no1 = __fmaf_rn(__fadd_rn(e0[k], e[k]), kAlpha, o0[k]);
            const float ne1 = live ? __fmaf_rn(__fadd_rn(o1[k], no1), kBeta, e0[k]) : e0[k];
            const float no2 = __fmaf_rn(__fadd_rn(e1[k], ne1), kGamma, o1[k]);
            const float ne2 = live ? __fmaf_rn(__fadd_rn(o2[k], no2), kDelta, e1[k]) : e1[k];
            e0[k] = e[k];
            o0[k] = o[k];
            o1[k] = no1;
            e1[k] = ne1;
            o2[k] = no2;
            e[k] = live ? __fmul_rn(ne2, kKInv) : ne2;
            o[k] = __fmul_rn(no2, kK);
        }
    }
};

}  // namespace wema
