// window.cu - the window ("--haar") temporal filter (temporal_filter.c:139-319);
// its deltas are amplified like the IIR's (phase_amp.c:12-56) where the
// inverse DWT stages the coefficients.
//
// The ring holds the last ws frames of every unique coefficient, slot-major
// ([ws][Pu]), so a push is one contiguous plane copy and each thread reads
// its position's history with coalesced loads.  For position u, with the
// window in chronological order x_0..x_{ws-1} (oldest first, centre c = ws/2):
//   delta = x_c - mean(x);
//   bilateral: sigma = max(0.5 * mean|x_t - x_c|, 1e-3),
//              w_t = exp(-(x_t-x_c)^2 / (2 sigma^2)) * exp(-(t-c)^2 / (2 (0.15 ws)^2)),
//              delta = sum w_t (x_t - mean) / sum w_t  (if sum w_t > 1e-8).
// The reference's vectorised reductions and vector expf order these sums
// differently; deltas agree to a few ulp, the bar for this stage.
//
// Precision variant (fp16): the ring's samples are stored as FP16 (rounded to
// nearest on the push) and widened to FP32 as they are read; every sum, the
// mean, the weights and the delta stay FP32.  The ring is the window mode's
// dominant traffic (ws reads per position per frame), so this halves it.
#include <cuda_fp16.h>

#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace wema {

constexpr int WIN_THREADS = 256;

__device__ __forceinline__ void put(float* p, float v) { *p = v; }
__device__ __forceinline__ void put(__half* p, float v) { *p = __float2half_rn(v); }
__device__ __forceinline__ float get(const float* p) { return *p; }
__device__ __forceinline__ float get(const __half* p) { return __half2float(*p); }

template <class T>
__global__ void k_ring_push(WindowParams w) {
    const int c = blockIdx.y;
    const float* coef = w.coef[c];
    T* dst = static_cast<T*>(w.ring[c]) + (long long)w.newest * w.pu;
    for (long long u = blockIdx.x * (long long)blockDim.x + threadIdx.x; u < w.pu;
         u += (long long)gridDim.x * blockDim.x)
        put(dst + u, pl_ld(coef, u, w.h16));
}

// The frame's push is in the filter kernels: the newest sample comes from the
// coefficient plane and goes to its ring slot (no coefficient plane: it is
// there already).  As the ring holds it: FP16-rounded where it is.
template <class T>
__device__ __forceinline__ T newest_sample(const WindowParams& w, int c, long long u) {
    T* const slot = static_cast<T*>(w.ring[c]) + (long long)w.newest * w.pu + u;
    if (!w.coef[c]) return *slot;
    T v;
    put(&v, pl_ld(w.coef[c], u, w.h16));
    *slot = v;
    return v;
}

// V consecutive ring elements in one load
template <class T, int V>
struct __align__(V * sizeof(T)) Pack {
    T v[V];
};

// ---- delta = centre sample - mean: one pass over the ring, V positions per
// thread (V > 1 where every slot's row starts aligned, so a sample costs a
// quarter of the loads and addresses).  1280x720, window 32: 47 -> 25 us.
template <class T, int V>
__global__ void __launch_bounds__(WIN_THREADS) k_window_mean(WindowParams w) {
    const int c = blockIdx.y;
    const long long pu = w.pu;
    const int ws = w.ws, center = ws / 2, wrap = ws - w.head;   // sample `wrap` is slot 0
    const float inv_ws = __fdiv_rn(1.0f, (float)ws);
    const T* const ring = static_cast<const T*>(w.ring[c]);
    for (long long u = V * (blockIdx.x * (long long)WIN_THREADS + threadIdx.x); u < pu;
         u += V * ((long long)gridDim.x * WIN_THREADS)) {
        float sum[V], cur[V];
#pragma unroll
        for (int k = 0; k < V; k++) sum[k] = cur[k] = 0.0f;
        auto take = [&](const Pack<T, V>& x, int t) {
#pragma unroll
            for (int k = 0; k < V; k++) {
                const float v = get(&x.v[k]);
                sum[k] = __fadd_rn(sum[k], v);
                if (t == center) cur[k] = v;
            }
        };
        // samples 0 .. ws-2 in the ring's two runs, then the newest
        auto run = [&](int t0, int t1, long long slot) {
            const T* q = ring + slot * pu + u;
#pragma unroll 8
            for (int t = t0; t < t1; t++, q += pu) take(*reinterpret_cast<const Pack<T, V>*>(q), t);
        };
        run(0, min(wrap, ws - 1), w.head);
        run(wrap, ws - 1, 0);
        Pack<T, V> last;
#pragma unroll
        for (int k = 0; k < V; k++) last.v[k] = newest_sample<T>(w, c, u + k);
        take(last, ws - 1);
#pragma unroll
        for (int k = 0; k < V; k++)
            pl_st(w.delta[c], u + k, __fadd_rn(cur[k], -__fmul_rn(inv_ws, sum[k])), w.h16);
    }
}

// ---- bilateral: a tile of positions with its whole window in shared memory
// ([sample][position], oldest first), read from the ring once; two positions
// per thread.  The mean and the mean deviation share a pass (the centre sample
// is known by then), the weights take the second.  Instruction-bound: about 20 per
// sample and position, 8 of them the exponential, against 64 with the ring
// read in each of three passes and indexed modulo its size.
// 1280x720, window 32: 74 -> 44 us a frame (push included), 118 MB of ring.
// WIDE: windows whose tiles leave at most 7 CTAs per SM get the registers for
// more samples in flight (window 64: 104 -> 91 us; at 32 it costs 1-5 us).
// VEC: every slot's row starts at 16 bytes, so the tile comes in by 16-byte
// asynchronous copies (else by loads, eight samples at a time).
template <class T, bool WIDE, bool VEC>
__global__ void __launch_bounds__(WIN_THREADS / 2, WIDE ? 7 : VEC ? 16 : 10) k_window_bilateral(WindowParams w) {
    extern __shared__ __align__(16) unsigned char win_smem[];
    T* const tile = reinterpret_cast<T*>(win_smem);
    const int c = blockIdx.y, P = 2 * blockDim.x, tid = threadIdx.x;
    const long long pu = w.pu;
    const int ws = w.ws, head = w.head, center = ws / 2;
    const float inv_ws = __fdiv_rn(1.0f, (float)ws);
    const T* const ring = static_cast<const T*>(w.ring[c]);
    constexpr int EPC = 16 / sizeof(T);                 // elements per 16-byte copy
    for (long long u0 = (long long)blockIdx.x * P; u0 < pu; u0 += (long long)gridDim.x * P) {
        const int np = (int)min((long long)P, pu - u0);
        if constexpr (VEC) {   // (np is a multiple of EPC too)
            const int pieces = P / EPC, e = (tid % pieces) * EPC;
            for (int t = tid / pieces; t < ws - 1; t += blockDim.x / pieces) {
                int slot = head + t;
                if (slot >= ws) slot -= ws;
                if (e < np) {
                    const unsigned d = (unsigned)__cvta_generic_to_shared(tile + t * P + e);
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d),
                                 "l"(ring + (long long)slot * pu + u0 + e) : "memory");
                }
            }
            asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
        } else {
            const bool a = tid < np, b = tid + (int)blockDim.x < np;
            for (int t0 = 0; t0 < ws - 1; t0 += 8) {   // 8 samples' loads in flight
                T v[8][2];
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    int slot = head + min(t0 + i, ws - 2);
                    if (slot >= ws) slot -= ws;
                    const T* q = ring + (long long)slot * pu + u0 + tid;
                    if (a) v[i][0] = __ldg(q);
                    if (b) v[i][1] = __ldg(q + blockDim.x);
                }
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const int t = min(t0 + i, ws - 2);
                    if (a) tile[t * P + tid] = v[i][0];
                    if (b) tile[t * P + tid + blockDim.x] = v[i][1];
                }
            }
        }
        const int k0 = 2 * tid;
        if (k0 < np) tile[(ws - 1) * P + k0] = newest_sample<T>(w, c, u0 + k0);
        if (k0 + 1 < np) tile[(ws - 1) * P + k0 + 1] = newest_sample<T>(w, c, u0 + k0 + 1);
        __syncthreads();
        const Pack<T, 2>* const col = reinterpret_cast<const Pack<T, 2>*>(tile + k0);   // next sample: P / 2 on
        const int step = P / 2;
        float cur[2], sum[2] = {0.0f, 0.0f}, mad[2] = {0.0f, 0.0f};
        float mean[2], inv2[2], wsum[2] = {0.0f, 0.0f}, res[2] = {0.0f, 0.0f};
#pragma unroll
        for (int k = 0; k < 2; k++) cur[k] = get(&col[center * step].v[k]);
#pragma unroll 8
        for (int t = 0; t < ws; t++) {
            const Pack<T, 2> x = col[t * step];
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const float v = get(&x.v[k]);
                sum[k] = __fadd_rn(sum[k], v);
                mad[k] = __fadd_rn(mad[k], fabsf(__fadd_rn(v, -cur[k])));
            }
        }
#pragma unroll
        for (int k = 0; k < 2; k++) {
            mean[k] = __fmul_rn(inv_ws, sum[k]);
            const float sigma = fmaxf(__fmul_rn(__fmul_rn(inv_ws, 0.5f), mad[k]), 0.001f);
            inv2[k] = __fdiv_rn(0.5f, __fmul_rn(sigma, sigma));
        }
#pragma unroll 8
        for (int t = 0; t < ws; t++) {
            const Pack<T, 2> x = col[t * step];
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const float v = get(&x.v[k]);
                const float df = __fadd_rn(v, -cur[k]);
                const float wt = __fmul_rn(expf(-__fmul_rn(__fmul_rn(df, df), inv2[k])), w.time_w[t]);
                wsum[k] = __fadd_rn(wsum[k], wt);
                res[k] = __fmaf_rn(wt, __fadd_rn(v, -mean[k]), res[k]);
            }
        }
#pragma unroll
        for (int k = 0; k < 2; k++) {
            float d = __fadd_rn(cur[k], -mean[k]);
            if (wsum[k] > 1e-8f) d = __fmul_rn(res[k], __fdiv_rn(1.0f, wsum[k]));
            if (k0 + k < np) pl_st(w.delta[c], u0 + k0 + k, d, w.h16);
        }
        __syncthreads();   // the tile is free for the next
    }
}

static dim3 win_grid(long long pu, int channels, int most) {
    const long long b = (pu + WIN_THREADS - 1) / WIN_THREADS;
    return dim3((unsigned)(b < most ? (b > 0 ? b : 1) : most), (unsigned)channels);
}

cudaError_t window_prepare_device() {
    const int most = 256 * 128 * (int)sizeof(float);   // the longest window over 128 positions
    cudaError_t e = cudaSuccess;
    for (const void* k :
         {(const void*)k_window_bilateral<float, false, false>, (const void*)k_window_bilateral<float, false, true>,
          (const void*)k_window_bilateral<float, true, false>, (const void*)k_window_bilateral<float, true, true>,
          (const void*)k_window_bilateral<__half, false, false>, (const void*)k_window_bilateral<__half, false, true>,
          (const void*)k_window_bilateral<__half, true, false>, (const void*)k_window_bilateral<__half, true, true>})
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    return e;
}

cudaError_t launch_ring_push(const WindowParams& wp, int channels, cudaStream_t st) {
    const dim3 g = win_grid(wp.pu, channels, 148 * 8);
    if (wp.fp16) k_ring_push<__half><<<g, WIN_THREADS, 0, st>>>(wp);
    else k_ring_push<float><<<g, WIN_THREADS, 0, st>>>(wp);
    return cudaGetLastError();
}

// every slot's row of every channel's ring starts at a multiple of `bytes`
static bool rows_aligned(const WindowParams& wp, int channels, size_t esz, size_t bytes) {
    bool ok = (size_t)wp.pu * esz % bytes == 0;
    for (int c = 0; c < channels; c++) ok = ok && reinterpret_cast<uintptr_t>(wp.ring[c]) % bytes == 0;
    return ok;
}

template <class T>
static void launch_window_t(const WindowParams& wp, int channels, cudaStream_t st) {
    if (wp.bilateral) {
        // tiles of 256 positions up to 32 KB of window, 128 beyond
        const bool wide = (size_t)wp.ws * 256 * sizeof(T) > 32768;
        const int P = wide ? 128 : 256;
        const long long b = (wp.pu + P - 1) / P;
        const dim3 g((unsigned)std::max<long long>(std::min<long long>(b, 148 * 64), 1), (unsigned)channels);
        const size_t smem = (size_t)wp.ws * P * sizeof(T);
        const bool vec = rows_aligned(wp, channels, sizeof(T), 16);
        if (wide && vec) k_window_bilateral<T, true, true><<<g, P / 2, smem, st>>>(wp);
        else if (wide) k_window_bilateral<T, true, false><<<g, P / 2, smem, st>>>(wp);
        else if (vec) k_window_bilateral<T, false, true><<<g, P / 2, smem, st>>>(wp);
        else k_window_bilateral<T, false, false><<<g, P / 2, smem, st>>>(wp);
        return;
    }
    if (rows_aligned(wp, channels, sizeof(T), 4 * sizeof(T)))
        k_window_mean<T, 4><<<win_grid((wp.pu + 3) / 4, channels, 148 * 16), WIN_THREADS, 0, st>>>(wp);
    else
        k_window_mean<T, 1><<<win_grid(wp.pu, channels, 148 * 16), WIN_THREADS, 0, st>>>(wp);
}

cudaError_t launch_window(const WindowParams& wp, int channels, cudaStream_t st) {
    if (wp.fp16) launch_window_t<__half>(wp, channels, st);
    else launch_window_t<float>(wp, channels, st);
    return cudaGetLastError();
}

}  // namespace wema
