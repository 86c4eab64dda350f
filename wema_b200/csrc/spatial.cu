// spatial.cu - luma-delta smoothing and transfer to RGB, fused with the u8
// output (wema.c:289-335, wema_batch.c:311-346).
//
// guide I = luma of the input frame (same evaluation as the DWT input),
// p = gray_out - I, smoothed by the guided filter (radius 4, eps 0.01,
// wema.c:173-230) or, with edge-aware off, the 5-tap [1 4 6 4 1]/16 blur
// with border renormalisation (wema.c:236-283); then
// out = clamp01(RGB + smooth) and u8 = (uint8)(v*255 + 0.5).
//
// Guided filter: one warp sweeps a strip of the frame from top to bottom
// (see guided_sweep).  Every box mean is the clipped window's sum divided by
// the clipped count (the reference's definition); the sums here are
// vertical running sums over a 9-row ring and horizontal window sums across
// the warp's lanes, not the reference's FP32 running prefix sums - the two
// differ in the last bits only, which the u8 output absorbs (<= 1 LSB).
#include "common.cuh"
#include "kernels.h"
#include "multi.cuh"

#include <algorithm>
#include <atomic>
#include <type_traits>

namespace wema {

constexpr int TS = 32;                  // Gaussian fallback: output tile
constexpr int SP_THREADS = 256;         // Gaussian fallback: threads per tile

struct SpArgs { TransferParams p; };

__device__ __forceinline__ void load_rgb(const TransferParams& p, const float* lut, int pi,
                                         float& r, float& g, float& b) {
    if (p.src_u8) {
        const uint8_t* q = p.src_u8 + 3 * pi;
        r = lut[q[0]]; g = lut[q[1]]; b = lut[q[2]];
    } else {
        const float* q = p.src_f32 + 3 * pi;
        r = q[0]; g = q[1]; b = q[2];
    }
}

__device__ __forceinline__ void store_rgb(const TransferParams& p, int pi, float r, float g,
                                          float b, float dy) {
    r = clamp01(__fadd_rn(r, dy));
    g = clamp01(__fadd_rn(g, dy));
    b = clamp01(__fadd_rn(b, dy));
    if (p.out_u8) {
        uint8_t* d = p.out_u8 + 3 * pi;
        d[0] = quant_u8(r); d[1] = quant_u8(g); d[2] = quant_u8(b);
    }
    if (p.out_f32) {
        float* d = p.out_f32 + 3 * pi;
        d[0] = r; d[1] = g; d[2] = b;
    }
}

// ---- guided filter: a vertical sweep per warp --------------------------------
//
// A warp owns a strip of 128 input columns, 4 consecutive columns per lane,
// and sweeps a segment of output rows from top to bottom.  The
// strip's first and last 8 columns are the halo of the two radius-4 rounds,
// so a strip produces 112 output columns (lanes 2..29); strips overlap by 16
// columns and segments by 16 rows (the vertical halo).  Per input
// row r entering the sweep:
//   I, p of row r (0 outside the image) go into a 9-row ring in shared
//   memory; vertical running sums of I, p, I*I, I*p over rows r-8..r add
//   row r and drop row r-9 (read back from the ring);
//   the first round at row r-4: horizontal 9-column window sums of those
//   vertical sums, exchanged with the neighbouring lanes by shuffles, times
//   1/(clipped column count x clipped row count) give mean_I, mean_p,
//   corr_II, corr_Ip and then a, b (0 outside the image, wema.c:206-217);
//   the horizontal window sums of a and b go into a second 9-row ring, whose
//   vertical running sums over rows r-12..r-4 give the second round at row
//   r-8: dy = mean_a * I + mean_b (wema.c:218-229, I read back from the
//   first ring), added to the row's RGB, clamped and quantised.
// Every running sum is recomputed from its ring, oldest row first, at rows
// fixed in the frame (first round: window ends r = 0 mod 16; second round:
// c1 = 4 mod 16) and slides from there, so a row's sums do not depend on
// where its segment starts: any segment that starts at a multiple of 16 rows
// gives bit-identical output, and rounding drift spans at most 15 slides.
//
// What bounds it: instruction issue and latency at 12 warps per SM (18.4 KB of
// rings per warp) - 460 instructions per row of a strip at 64% of the issue slots,
// DRAM at 19%.  So the work per pixel is cut (fewer halo rows by segments as long
// as an even split allows, quant12, shared quad sums) and the loop body is
// kept in few branch-free pieces: rows come in pairs whose second never
// recomputes its sums.  A 3840x8640 frame: 203 us against 248 (fixed segments
// of 64 rows, every byte through the float steps); fixed segments of 128 rows 241.
constexpr int GR = 4;                   // guided-filter radius (wema.c:314)
constexpr int GS_IN = 128;              // input columns per strip (4 per lane)
constexpr int GS_OUT = GS_IN - 4 * GR;  // output columns per strip
constexpr int GS_RING = 2 * GR + 1;     // rows in each ring
constexpr int GS_WARPS = 2;             // strips per CTA (one per warp)
constexpr int GS_THREADS = 32 * GS_WARPS;
constexpr int GS_UNIT = 16;              // segments start at multiples of this
constexpr int GS_ROWS_DEFAULT = 64;      // the setting that stands for an even split
constexpr float kEps = 0.01f;           // wema.c:315
constexpr unsigned kFull = 0xffffffffu;

struct SweepRing {                      // one warp's rings
    float4 ip[GS_RING][2][32];          // I, p of rows r-8..r; lane l holds columns 4l..4l+3
    float4 ab[GS_RING][2][32];          // horizontal window sums of a, b
};

// 1/k for the clipped window counts k = 1 .. 2 GR + 1 (index 0 unused),
// correctly rounded (the compiler's IEEE division)
__constant__ float c_rcp[2 * GR + 2] = {0.f, 1.f / 1, 1.f / 2, 1.f / 3, 1.f / 4, 1.f / 5,
                                         1.f / 6, 1.f / 7, 1.f / 8, 1.f / 9};

// 1 / (clipped count of a radius-4 window at coordinate c of a line of n);
// 0 for c outside the line
__device__ __forceinline__ float inv_count(int c, int n) {
    if (c < 0 || c >= n) return 0.f;
    return c_rcp[min(c + GR, n - 1) - max(c - GR, 0) + 1];
}

// The 9-column window sums centred on a lane's 4 columns: its own 4 values
// and its neighbours', by shuffles (lanes 0 and 31 get garbage, which only
// halo columns use).  The left neighbour's four values are needed as their
// sum and one by one: its sum comes with the shuffles (it made it for itself)
// instead of being added up again.
__device__ __forceinline__ void hwin(const float v[4], float o[4]) {
    const float t = __fadd_rn(__fadd_rn(v[0], v[1]), __fadd_rn(v[2], v[3]));
    const float tl = __shfl_up_sync(kFull, t, 1);
    float L[3], R[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        if (j < 3) L[j] = __shfl_up_sync(kFull, v[j], 1);
        R[j] = __shfl_down_sync(kFull, v[j], 1);
    }
    float s = __fadd_rn(__fadd_rn(tl, t), R[0]);
    o[0] = s;
#pragma unroll
    for (int j = 1; j < 4; j++) {
        s = __fadd_rn(__fsub_rn(s, L[j - 1]), R[j]);
        o[j] = s;
    }
}

__device__ __forceinline__ float max_nan(float a, float b) {   // NaN if either is
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

// How a sweep reads and writes its rows (chosen per stream, sweep_mode):
//   kRowsWords   RGB24 rows word-aligned (width a multiple of 4 and aligned
//                buffers): the 4 pixels of a lane are 3 words, all in or all
//                out of the image;
//   kRowsWords16 the same with an FP16 reconstruction (planes_fp16): its loads
//                are kept as they came and widened a row later, when they
//                are used;
//   kRowsRagged  RGB24 of any width >= 4 and alignment: a lane's 12 bytes are
//                cut from 4 aligned words by a funnel shift (the shift is the
//                row's: lanes are 12 bytes apart), and the output's words are
//                put together across lanes the same way, with byte stores
//                only at the two ends of the strip's row.  3839x2160 in
//                64-row segments: 105 us a frame, 180 pixel by pixel;
//   kRowsFloat   float RGB frames;
//   kRowsAny     RGB24 pixel by pixel: widths below 4 and frames of 2^29
//                pixels or more (64-bit indices).
enum { kRowsWords = 0, kRowsWords16 = 1, kRowsRagged = 2, kRowsFloat = 3, kRowsAny = 4, kRowsMixed = -1 };

// One row of 4 pixels of a lane: the loads of row r, issued a row ahead,
// and their decoding; with them the RGB of row r - 2 GR, the step's output row
// (loaded as input 2 GR rows earlier, so mostly cache hits).  A lane outside
// the image keeps stale values, which decode() and the writers leave out.
template <int MODE>
struct RowLoad;

// guide I and p = gray - I of 4 pixels; in[j]: pixel j lies in the image.
// vec: all four in the vector body's evaluation order
__device__ __forceinline__ void guide4(const float (&c)[12], const float (&gy)[4], const bool (&in)[4], bool vec,
                                       long long pi0, long long vec_end, float I[4], float P[4]) {
    float Iv[4];
    if (vec) {
#pragma unroll
        for (int j = 0; j < 4; j++) Iv[j] = luma_vec(c[3 * j], c[3 * j + 1], c[3 * j + 2]);
    } else {
#pragma unroll
        for (int j = 0; j < 4; j++)
            Iv[j] = pi0 + j < vec_end ? luma_vec(c[3 * j], c[3 * j + 1], c[3 * j + 2])
                                      : luma_tail(c[3 * j], c[3 * j + 1], c[3 * j + 2]);
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
        I[j] = in[j] ? Iv[j] : 0.f;
        P[j] = in[j] ? __fadd_rn(gy[j], -Iv[j]) : 0.f;
    }
}

// The output bytes of 4 pixels: quant(clamp01(fl(b / 255) + dy)) of the 12
// bytes b in w.  In exact arithmetic that is floor(b + 255 dy + 1/2) clamped to
// 0..255, and the float steps' roundings stay below 3.1e-5 in those units
// (fl(b / 255) and its sum with dy 2^-25 each where the sum is not clamped,
// times 255; the product and the sum with 1/2 2^-17 each).  So where 255 dy is
// further than 1e-4 from an exact half and below 20000, all three channels
// of the pixel are b + n clamped with n = round(255 dy): two channels per
// 16-bit-pair add, minimum and maximum.  A warp with another pixel (about one
// row in 40) takes the float steps for the lanes that hold one; the clamps
// send a NaN to 0 (SAT) or 255.
template <bool SAT>
__device__ __forceinline__ void quant12(const uint32_t (&w)[3], const float (&dy)[4], uint32_t (&o)[3]) {
    constexpr float M = 12582912.0f;    // 1.5 * 2^23: the low bits of x + M hold round(x)
    uint32_t n[4];
    float dm = 0.f, nm = 0.f;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const float rb = __fmaf_rn(dy[j], 255.0f, M);
        const float nf = __fsub_rn(rb, M);
        dm = max_nan(dm, fabsf(__fmaf_rn(dy[j], 255.0f, -nf)));
        nm = max_nan(nm, fabsf(nf));
        n[j] = __float_as_uint(rb);
    }
    // the channels' pairs: (r g)(b r') (g' b')(r" g") (b" r"')(g"' b"')
    const uint32_t add[6] = {__byte_perm(n[0], n[0], 0x1010), __byte_perm(n[0], n[1], 0x5410),
                             __byte_perm(n[1], n[1], 0x1010), __byte_perm(n[2], n[2], 0x1010),
                             __byte_perm(n[2], n[3], 0x5410), __byte_perm(n[3], n[3], 0x1010)};
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const uint32_t lo = __viaddmin_s16x2_relu(__byte_perm(w[k], 0u, 0x4140), add[2 * k], 0x00ff00ffu);
        const uint32_t hi = __viaddmin_s16x2_relu(__byte_perm(w[k], 0u, 0x4342), add[2 * k + 1], 0x00ff00ffu);
        o[k] = __byte_perm(lo, hi, 0x6420);
    }
    const bool ok = dm < 0.4999f && nm < 20000.0f;
    if (__any_sync(kFull, !ok)) {       // (uniform)
#pragma unroll
        for (int k = 0; k < 3; k++) {
            uint32_t q[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float v = __fadd_rn(byte_of(w[k], i), dy[(4 * k + i) / 3]);
                q[i] = quant_bits(SAT ? __saturatef(v) : clamp01(v));
            }
            // low bytes of four quantised values into one word
            const uint32_t f = __byte_perm(__byte_perm(q[0], q[1], 0x0040u), __byte_perm(q[2], q[3], 0x0040u), 0x5410u);
            o[k] = ok ? o[k] : f;
        }
    }
}

template <bool H16>
struct RowLoadWords {
    uint32_t w[3];
    std::conditional_t<H16, uint2, float4> g;
    uint32_t ow[3];
    bool any;

    __device__ __forceinline__ void issue(const TransferParams& p, int r, int cx) {
        any = r >= 0 && r < p.h && cx + 3 >= 0 && cx < p.w;
        const int y = r - 2 * GR;
        if (y >= 0 && y < p.h && cx >= 0 && cx < p.w) {
            const uint32_t* q = reinterpret_cast<const uint32_t*>(p.src_u8) + 3 * ((y * p.w + cx) >> 2);
            ow[0] = __ldg(q);
            ow[1] = __ldg(q + 1);
            ow[2] = __ldg(q + 2);
        }
        if (any) {
            const int pi = r * p.w + cx;
            const uint32_t* q = reinterpret_cast<const uint32_t*>(p.src_u8) + 3 * (pi >> 2);
            w[0] = __ldg(q);
            w[1] = __ldg(q + 1);
            w[2] = __ldg(q + 2);
            if constexpr (H16) g = __ldg(reinterpret_cast<const uint2*>(reinterpret_cast<const __half*>(p.gray_out) + pi));
            else g = __ldg(reinterpret_cast<const float4*>(p.gray_out + pi));
        }
    }
    __device__ __forceinline__ void decode(const TransferParams& p, int r, int cx, float I[4], float P[4]) const {
        float c[12];
#pragma unroll
        for (int k = 0; k < 12; k++) c[k] = byte_of(w[k >> 2], k & 3);
        float gy[4];
        if constexpr (H16) {
            const float2 lo = __half22float2(*reinterpret_cast<const __half2*>(&g.x));
            const float2 hi = __half22float2(*reinterpret_cast<const __half2*>(&g.y));
            gy[0] = lo.x; gy[1] = lo.y; gy[2] = hi.x; gy[3] = hi.y;
        } else {
            gy[0] = g.x; gy[1] = g.y; gy[2] = g.z; gy[3] = g.w;
        }
        const bool in[4] = {any, any, any, any};
        const long long pi0 = (long long)r * p.w + cx;
        // every row but the last lies in the vector body: it ends at most 3 pixels
        // before the frame's end, and 4 | w
        guide4(c, gy, in, r + 1 < p.h || pi0 + 3 < p.vec_end, pi0, p.vec_end, I, P);
    }
    // out = clamp01(RGB + dy) of the lane's 4 output pixels of row y, in the
    // strip whose output columns start at x0; called by every lane
    __device__ __forceinline__ void put(const TransferParams& p, int y, int cx, int x0, const float (&dy)[4]) const {
        const int lane = threadIdx.x & 31;
        const bool mine = lane >= 2 && lane < 30 && cx >= 0 && cx < p.w;   // not a halo lane
        const int pi0 = y * p.w + cx;
        uint32_t o[3];
        quant12<true>(ow, dy, o);
        if (mine && p.out_u8) {
            uint32_t* d = reinterpret_cast<uint32_t*>(p.out_u8) + 3 * (pi0 >> 2);
            d[0] = o[0];
            d[1] = o[1];
            d[2] = o[2];
        }
        if (mine && p.out_f32) {
            float4* d = reinterpret_cast<float4*>(p.out_f32 + 3 * pi0);
#pragma unroll
            for (int k = 0; k < 3; k++) {
                float v[4];
#pragma unroll
                for (int i = 0; i < 4; i++) v[i] = __saturatef(__fadd_rn(byte_of(ow[k], i), dy[(4 * k + i) / 3]));
                d[k] = make_float4(v[0], v[1], v[2], v[3]);
            }
        }
    }
};

template <>
struct RowLoad<kRowsWords> : RowLoadWords<false> {};
template <>
struct RowLoad<kRowsWords16> : RowLoadWords<true> {};

template <>
struct RowLoad<kRowsRagged> {
    uint32_t w[4], ow[4];
    int sh, osh;                        // bit shift of the lane's first byte in w[0], ow[0]
    float g[4];
    bool any;

    // the four aligned words from the one that holds byte 3 * pi of the
    // frame; words past the frame's last byte are not read
    static __device__ __forceinline__ void words4(const TransferParams& p, int pi, uint32_t (&v)[4], int& shift) {
        const unsigned off = (unsigned)(reinterpret_cast<uintptr_t>(p.src_u8) & 3);
        const uint32_t* base = reinterpret_cast<const uint32_t*>(p.src_u8 - off);
        const unsigned b = off + 3u * (unsigned)pi;
        const unsigned nw = (off + 3u * (unsigned)(p.w * p.h) + 3u) >> 2;
        shift = 8 * (int)(b & 3);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const unsigned i = (b >> 2) + k;
            v[k] = 0u;
            if (i < nw) v[k] = __ldg(base + i);
        }
    }
    static __device__ __forceinline__ void bytes12(const uint32_t (&v)[4], int shift, uint32_t (&o)[3]) {
#pragma unroll
        for (int k = 0; k < 3; k++) o[k] = __funnelshift_r(v[k], v[k + 1], shift);
    }

    __device__ __forceinline__ void issue(const TransferParams& p, int r, int cx) {
        // (cx is a multiple of 4: a lane with pixels in the image has cx >= 0)
        any = r >= 0 && r < p.h && cx >= 0 && cx < p.w;
        const int y = r - 2 * GR;
        if (y >= 0 && y < p.h && cx >= 0 && cx < p.w) words4(p, y * p.w + cx, ow, osh);
        if (any) {
            const int pi = r * p.w + cx;
            words4(p, pi, w, sh);
            if (p.h16) {
#pragma unroll
                for (int j = 0; j < 4; j++)
                    g[j] = cx + j < p.w ? __half2float(__ldg(reinterpret_cast<const __half*>(p.gray_out) + pi + j)) : 0.f;
            } else {
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    g[j] = 0.f;
                    if (cx + j < p.w) g[j] = __ldg(p.gray_out + pi + j);
                }
            }
        }
    }
    __device__ __forceinline__ void decode(const TransferParams& p, int r, int cx, float I[4], float P[4]) const {
        uint32_t b[3];
        bytes12(w, sh, b);
        float c[12];
#pragma unroll
        for (int k = 0; k < 12; k++) c[k] = byte_of(b[k >> 2], k & 3);
        const bool in[4] = {any, any && cx + 1 < p.w, any && cx + 2 < p.w, any && cx + 3 < p.w};
        const long long pi0 = (long long)r * p.w + cx;
        guide4(c, g, in, r + 1 < p.h || pi0 + 3 < p.vec_end, pi0, p.vec_end, I, P);   // (w >= 4)
    }
    __device__ __forceinline__ void put(const TransferParams& p, int y, int cx, int x0, const float (&dy)[4]) const {
        uint32_t b[3], o[3];
        bytes12(ow, osh, b);
        quant12<false>(b, dy, o);
        const uint32_t left = __shfl_up_sync(kFull, o[2], 1);
        // the strip's bytes of the row, and the lane's three aligned words of them
        const int off = (int)(reinterpret_cast<uintptr_t>(p.out_u8) & 3);
        uint8_t* const base = p.out_u8 - off;
        const int row = y * p.w;
        const int bs = off + 3 * (row + x0), be = off + 3 * (row + min(x0 + GS_OUT, p.w));
        const int b0 = off + 3 * (row + cx);
        const int s = 8 * (b0 & 3);
        const uint32_t v[3] = {__funnelshift_l(left, o[0], s), __funnelshift_l(o[0], o[1], s),
                               __funnelshift_l(o[1], o[2], s)};
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const int at = (b0 & ~3) + 4 * k;
            if (at >= bs && at + 4 <= be) {
                *reinterpret_cast<uint32_t*>(base + at) = v[k];
            } else if (at + 4 > bs && at < be) {
#pragma unroll
                for (int i = 0; i < 4; i++)
                    if (at + i >= bs && at + i < be) base[at + i] = (uint8_t)(v[k] >> (8 * i));
            }
        }
    }
};

// one pixel at a time: U8 RGB24, else float RGB
template <bool U8>
struct RowLoadPixels {
    float rgb[12], g[4];
    bool any;

    __device__ __forceinline__ void issue(const TransferParams& p, int r, int cx) {
        any = r >= 0 && r < p.h && cx + 3 >= 0 && cx < p.w;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int x = cx + j;
            const long long pi = (long long)r * p.w + x;
            g[j] = 0.f;
#pragma unroll
            for (int c = 0; c < 3; c++) rgb[3 * j + c] = 0.f;
            if (any && x >= 0 && x < p.w) {
                g[j] = pl_ld(p.gray_out, pi, p.h16);
#pragma unroll
                for (int c = 0; c < 3; c++)
                    rgb[3 * j + c] = U8 ? u8f(__ldg(p.src_u8 + 3 * pi + c)) : __ldg(p.src_f32 + 3 * pi + c);
            }
        }
    }
    __device__ __forceinline__ void decode(const TransferParams& p, int r, int cx, float I[4], float P[4]) const {
        bool in[4];
#pragma unroll
        for (int j = 0; j < 4; j++) in[j] = any && cx + j >= 0 && cx + j < p.w;
        const long long pi0 = (long long)r * p.w + cx;
        guide4(rgb, g, in, pi0 + 3 < p.vec_end, pi0, p.vec_end, I, P);
    }
    __device__ __forceinline__ void put(const TransferParams& p, int y, int cx, int x0, const float (&dy)[4]) const {
        const int lane = threadIdx.x & 31;
        if (lane < 2 || lane >= 30) return;
        const long long pi0 = (long long)y * p.w + cx;
        float v[12];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if (cx + j < 0 || cx + j >= p.w) continue;
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const long long e = 3 * (pi0 + j) + c;
                v[3 * j + c] = U8 ? u8f(__ldg(p.src_u8 + e)) : __ldg(p.src_f32 + e);
            }
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if (cx + j < 0 || cx + j >= p.w) continue;
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const long long e = 3 * (pi0 + j) + c;
                const float q = clamp01(__fadd_rn(v[3 * j + c], dy[j]));
                if (p.out_u8) p.out_u8[e] = quant_u8(q);
                if (p.out_f32) p.out_f32[e] = q;
            }
        }
    }
};
template <>
struct RowLoad<kRowsFloat> : RowLoadPixels<false> {};
template <>
struct RowLoad<kRowsAny> : RowLoadPixels<true> {};

// output rows ys .. ye-1 (ys a multiple of GS_UNIT) of one strip
template <int MODE>
__device__ __forceinline__ void guided_sweep(const TransferParams& pg, SweepRing& R, int strip, int ys, int ye) {
    // the parameters in registers: read through the reference, every field the
    // loop uses would be loaded again after each output store, which may alias
    // the parameter table as far as the compiler knows (measured 0.58 -> 0.55 ms)
    const TransferParams p = pg;
    const int W = p.w, H = p.h;
    const int lane = threadIdx.x & 31;
    const int x0 = strip * GS_OUT;
    const int cx = x0 - 2 * GR + 4 * lane;          // this lane's first column

    float icx[4];
#pragma unroll
    for (int j = 0; j < 4; j++) icx[j] = inv_count(cx + j, W);
    const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int k = 0; k < GS_RING; k++) {
        R.ip[k][0][lane] = z4; R.ip[k][1][lane] = z4;
        R.ab[k][0][lane] = z4; R.ab[k][1][lane] = z4;
    }
    float vI[4] = {0.f, 0.f, 0.f, 0.f}, vP[4] = {0.f, 0.f, 0.f, 0.f};
    float vII[4] = {0.f, 0.f, 0.f, 0.f}, vIP[4] = {0.f, 0.f, 0.f, 0.f};
    float uA[4] = {0.f, 0.f, 0.f, 0.f}, uB[4] = {0.f, 0.f, 0.f, 0.f};
    int s1 = 0, s2 = 0;                             // ring slots of the row entering

    // one input row through the sweep (the row's loads were issued a row ahead).
    // Both sums' anchors lie at even rows, and the sweep starts at one
    auto step = [&](const RowLoad<MODE>& in, int r, auto even_row) {
        constexpr bool EVEN = decltype(even_row)::value;
        float I[4], P[4];
        in.decode(p, r, cx, I, P);
        // ring of I, p; vertical sums over rows r-8..r
        {
            const float4 oI = R.ip[s1][0][lane], oP = R.ip[s1][1][lane];
            R.ip[s1][0][lane] = make_float4(I[0], I[1], I[2], I[3]);
            R.ip[s1][1][lane] = make_float4(P[0], P[1], P[2], P[3]);
            const float ofI[4] = {oI.x, oI.y, oI.z, oI.w}, ofP[4] = {oP.x, oP.y, oP.z, oP.w};
#pragma unroll
            for (int j = 0; j < 4; j++) {
                vI[j] = __fsub_rn(__fadd_rn(vI[j], I[j]), ofI[j]);
                vP[j] = __fsub_rn(__fadd_rn(vP[j], P[j]), ofP[j]);
                vII[j] = __fmaf_rn(-ofI[j], ofI[j], __fmaf_rn(I[j], I[j], vII[j]));
                vIP[j] = __fmaf_rn(-ofI[j], ofP[j], __fmaf_rn(I[j], P[j], vIP[j]));
            }
            if (EVEN && (r & 15) == 0) {                  // anchor: the window's sums afresh
#pragma unroll
                for (int j = 0; j < 4; j++) vI[j] = vP[j] = vII[j] = vIP[j] = 0.f;
#pragma unroll
                for (int k = 1; k <= GS_RING; k++) {   // slots s1+1 .. s1+9: rows r-8 .. r
                    const int sl = s1 + k < GS_RING ? s1 + k : s1 + k - GS_RING;
                    const float4 a4 = R.ip[sl][0][lane], b4 = R.ip[sl][1][lane];
                    const float ai[4] = {a4.x, a4.y, a4.z, a4.w}, bi[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        vI[j] = __fadd_rn(vI[j], ai[j]);
                        vP[j] = __fadd_rn(vP[j], bi[j]);
                        vII[j] = __fmaf_rn(ai[j], ai[j], vII[j]);
                        vIP[j] = __fmaf_rn(ai[j], bi[j], vIP[j]);
                    }
                }
            }
            s1 = s1 == GS_RING - 1 ? 0 : s1 + 1;
        }
        if (r < ys) return;                         // rows r-8..r not all in yet
        // first round at row c1 = r - 4: a, b
        float a[4], b[4];
        {
            float sI[4], sP[4], sII[4], sIP[4];
            hwin(vI, sI);
            hwin(vP, sP);
            hwin(vII, sII);
            hwin(vIP, sIP);
            const float icy = inv_count(r - GR, H);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float inv = __fmul_rn(icx[j], icy);
                const float mI = __fmul_rn(sI[j], inv), mP = __fmul_rn(sP[j], inv);
                const float cII = __fmul_rn(sII[j], inv), cIP = __fmul_rn(sIP[j], inv);
                // the denominator is >= eps + E[I^2] - E[I]^2 > 0; a within 2 ulp
                const float av = __fdividef(__fmaf_rn(-mI, mP, cIP), __fmaf_rn(-mI, mI, __fadd_rn(cII, kEps)));
                // outside the image 0 by selection: a sum that overflowed would make
                // its product with inv = 0 a NaN, which the windows inside would take in
                const bool inside = inv != 0.f;
                a[j] = inside ? av : 0.f;
                b[j] = inside ? __fmaf_rn(-av, mI, mP) : 0.f;
            }
        }
        // second round: horizontal sums of a, b into the ring; vertical sums over rows c1-8..c1
        {
            float hA[4], hB[4];
            hwin(a, hA);
            hwin(b, hB);
            const float4 oA = R.ab[s2][0][lane], oB = R.ab[s2][1][lane];
            R.ab[s2][0][lane] = make_float4(hA[0], hA[1], hA[2], hA[3]);
            R.ab[s2][1][lane] = make_float4(hB[0], hB[1], hB[2], hB[3]);
            const float ofA[4] = {oA.x, oA.y, oA.z, oA.w}, ofB[4] = {oB.x, oB.y, oB.z, oB.w};
#pragma unroll
            for (int j = 0; j < 4; j++) {
                uA[j] = __fsub_rn(__fadd_rn(uA[j], hA[j]), ofA[j]);
                uB[j] = __fsub_rn(__fadd_rn(uB[j], hB[j]), ofB[j]);
            }
            if (EVEN && ((r - GR) & 15) == 4) {            // anchor: first-round rows c1-8..c1 afresh
#pragma unroll
                for (int j = 0; j < 4; j++) uA[j] = uB[j] = 0.f;
#pragma unroll
                for (int k = 1; k <= GS_RING; k++) {
                    const int sl = s2 + k < GS_RING ? s2 + k : s2 + k - GS_RING;
                    const float4 a4 = R.ab[sl][0][lane], b4 = R.ab[sl][1][lane];
                    const float ai[4] = {a4.x, a4.y, a4.z, a4.w}, bi[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        uA[j] = __fadd_rn(uA[j], ai[j]);
                        uB[j] = __fadd_rn(uB[j], bi[j]);
                    }
                }
            }
            s2 = s2 == GS_RING - 1 ? 0 : s2 + 1;
        }
        if (r < ys + 2 * GR) return;                // first-round rows c1-8..c1 not all in yet
        // output row y = r - 8; its I is the oldest row of the first ring (slot s1)
        const int y = r - 2 * GR;
        const float icy = inv_count(y, H);
        const float4 Iy = R.ip[s1][0][lane];
        const float Iv[4] = {Iy.x, Iy.y, Iy.z, Iy.w};
        float dy[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float inv = __fmul_rn(icx[j], icy);
            dy[j] = __fmaf_rn(__fmul_rn(uA[j], inv), Iv[j], __fmul_rn(uB[j], inv));
        }
        in.put(p, y, cx, x0, dy);
    };

    // two load buffers in turn, so a row's loads are in flight while the
    // previous row is computed (no register copy that would wait on them)
    const int r0 = ys - 2 * GR, r1 = ye + 2 * GR;
    RowLoad<MODE> A, B;
    A.issue(p, r0, cx);
    for (int r = r0; r < r1; r += 2) {
        if (r + 1 < r1) B.issue(p, r + 1, cx);
        step(A, r, std::true_type{});
        if (r + 1 >= r1) break;
        if (r + 2 < r1) A.issue(p, r + 2, cx);
        step(B, r + 1, std::false_type{});
    }
}

__host__ __device__ inline int sweep_mode(const TransferParams& p) {
    if (!p.src_u8) return kRowsFloat;
    if (p.w < 4 || (long long)p.w * p.h >= (1LL << 29)) return kRowsAny;
    const bool words = !(p.w & 3) && !(reinterpret_cast<uintptr_t>(p.src_u8) & 3) &&
                       !(reinterpret_cast<uintptr_t>(p.gray_out) & 15) &&
                       !(reinterpret_cast<uintptr_t>(p.out_u8) & 3) && !(reinterpret_cast<uintptr_t>(p.out_f32) & 15);
    if (words) return p.h16 ? kRowsWords16 : kRowsWords;
    return p.out_f32 || !p.out_u8 ? kRowsAny : kRowsRagged;   // (ragged rows: RGB24 out only)
}
int transfer_rows_mode(const TransferParams& p) { return sweep_mode(p); }

// A launch's work in units of seg_rows output rows of a strip, a frame's units
// strip after strip; consecutive units of a strip that a warp holds are one
// segment.
__device__ __forceinline__ int units_per_strip(const TransferParams& p) { return (p.h + p.seg_rows - 1) / p.seg_rows; }

// the rare form out of line, so that the mixed kernel's registers go to the others
__device__ __noinline__ void sweep_any(const TransferParams& p, SweepRing& R, int strip, int ys, int ye) {
    guided_sweep<kRowsAny>(p, R, strip, ys, ye);
}

// units u0 .. u0 + n - 1 of a frame's strip, in the form its rows have
// (kRowsMixed: looked up)
template <int MODE>
__device__ __forceinline__ void guided_segment(const TransferParams& p, SweepRing& R, int strip, int u0, int n) {
    const int ys = u0 * p.seg_rows, ye = min(ys + n * p.seg_rows, p.h);
    if constexpr (MODE != kRowsMixed) {
        guided_sweep<MODE>(p, R, strip, ys, ye);
    } else {
        const int mode = sweep_mode(p);
        if (mode == kRowsWords) guided_sweep<kRowsWords>(p, R, strip, ys, ye);
        else if (mode == kRowsWords16) guided_sweep<kRowsWords16>(p, R, strip, ys, ye);
        else if (mode == kRowsRagged) guided_sweep<kRowsRagged>(p, R, strip, ys, ye);
        else sweep_any(p, R, strip, ys, ye);   // (batched frames are RGB24)
    }
}

// ---- rows per segment, per device (the autotuner may change it): the default
// splits the work evenly over the warps, any other height is fixed
static std::atomic<int> g_seg_rows[64];

int guided_rows(int dev) {
    const int v = (dev >= 0 && dev < 64) ? g_seg_rows[dev].load() : 0;
    return v > 0 ? v : GS_ROWS_DEFAULT;
}

static int fixed_rows(int dev) {        // 0: split evenly
    const int v = guided_rows(dev);
    return v == GS_ROWS_DEFAULT ? 0 : v;
}

bool guided_set_rows(int dev, int rows) {
    if (dev < 0 || dev >= 64 || rows < 16 || rows > 4096 || (rows & 15)) return false;
    g_seg_rows[dev].store(rows);
    return true;
}

static int current_device() {
    int d = 0;
    cudaGetDevice(&d);
    return d;
}

// 5-tap Gaussian fallback: halo 2
constexpr int GH = 2;
constexpr int RG = TS + 2 * GH;

__device__ __forceinline__ void gauss_body(const TransferParams& p, int bx, int by) {
    __shared__ float P[RG][RG + 1];
    __shared__ float T[RG][TS + 1];
    __shared__ float lut[256];
    for (int i = threadIdx.x; i < 256; i += SP_THREADS) lut[i] = __fdiv_rn((float)i, 255.0f);
    const int W = p.w, H = p.h;
    const int x0 = bx * TS, y0 = by * TS;
    const int gx0 = x0 - GH, gy0 = y0 - GH;
    const float kw[5] = {1.0f / 16.0f, 4.0f / 16.0f, 6.0f / 16.0f, 4.0f / 16.0f, 1.0f / 16.0f};
    __syncthreads();
    for (int k = threadIdx.x; k < RG * RG; k += SP_THREADS) {
        const int ly = k / RG, lx = k % RG;
        const int gx = gx0 + lx, gy = gy0 + ly;
        float v = 0.f;
        if (gx >= 0 && gx < W && gy >= 0 && gy < H) {
            const long long pi = (long long)gy * W + gx;
            float r, g, b;
            load_rgb(p, lut, pi, r, g, b);
            const float I = pi < p.vec_end ? luma_vec(r, g, b) : luma_tail(r, g, b);
            v = __fadd_rn(pl_ld(p.gray_out, pi, p.h16), -I);
        }
        P[ly][lx] = v;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < RG * TS; k += SP_THREADS) {
        const int ly = k / TS, tx = k % TS;
        const int gx = x0 + tx, gy = gy0 + ly;
        if (gx >= W || gy < 0 || gy >= H) continue;
        float s = 0.f, wsum = 0.f;
#pragma unroll
        for (int d = -2; d <= 2; d++) {
            const int xx = gx + d;
            if (xx >= 0 && xx < W) {
                s = __fmaf_rn(P[ly][xx - gx0], kw[d + 2], s);
                wsum = __fadd_rn(wsum, kw[d + 2]);
            }
        }
        T[ly][tx] = __fdiv_rn(s, wsum);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < TS * TS; k += SP_THREADS) {
        const int ty = k / TS, tx = k % TS;
        const int gx = x0 + tx, gy = y0 + ty;
        if (gx >= W || gy >= H) continue;
        float s = 0.f, wsum = 0.f;
#pragma unroll
        for (int d = -2; d <= 2; d++) {
            const int yy = gy + d;
            if (yy >= 0 && yy < H) {
                s = __fmaf_rn(T[yy - gy0][tx], kw[d + 2], s);
                wsum = __fadd_rn(wsum, kw[d + 2]);
            }
        }
        const float dy = __fdiv_rn(s, wsum);
        const long long pi = (long long)gy * W + gx;
        float r, g, b;
        load_rgb(p, lut, pi, r, g, b);
        store_rgb(p, pi, r, g, b, dy);
    }
}

template <int MODE>
__global__ void __launch_bounds__(GS_THREADS) k_guided_transfer(SpArgs args, int units, int warps) {
    __shared__ SweepRing rings[GS_WARPS];
    const int per = units_per_strip(args.p);
    int2 u = unit_share(units, blockIdx.x * GS_WARPS + (threadIdx.x >> 5), warps);
    while (u.x < u.y) {
        const int strip = u.x / per, u0 = u.x - strip * per, n = min(u.y - u.x, per - u0);
        guided_segment<MODE>(args.p, rings[threadIdx.x >> 5], strip, u0, n);
        u.x += n;
    }
}
__global__ void __launch_bounds__(SP_THREADS) k_gauss_transfer(SpArgs args) {
    gauss_body(args.p, blockIdx.x, blockIdx.y);
}
// batched: task = one stream (edge-aware and Gaussian streams in separate
// launches); the guided map counts units, not blocks.  MODE: the one form of
// the launch's rows, or kRowsMixed, chosen per segment.  6 CTAs per SM is
// what the rings allow; the mixed kernel would take registers for 4 otherwise.
template <int MODE>
__global__ void __launch_bounds__(GS_THREADS, 6)
    k_guided_transfer_multi(const TransferParams* __restrict__ ps, const int* __restrict__ map, int warps) {
    __shared__ SweepRing rings[GS_WARPS];
    int2 u = unit_share(map[1 + map[0]], blockIdx.x * GS_WARPS + (threadIdx.x >> 5), warps);
    while (u.x < u.y) {
        const TaskBlock t = task_block(map, u.x);       // x: unit in the strip, y: strip
        const TransferParams& p = ps[t.task];
        const int n = min(u.y - u.x, units_per_strip(p) - t.x);
        guided_segment<MODE>(p, rings[threadIdx.x >> 5], t.y, t.x, n);
        u.x += n;
    }
}
__global__ void __launch_bounds__(SP_THREADS)
    k_gauss_transfer_multi(const TransferParams* __restrict__ ps, const int* __restrict__ map) {
    const TaskBlock t = task_block(map, blockIdx.x);
    gauss_body(ps[t.task], t.x, t.y);
}

__global__ void k_passthrough(SpArgs args) {
    const TransferParams& p = args.p;
    const long long n = (long long)p.w * p.h * 3;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        float v = p.src_u8 ? __fdiv_rn((float)p.src_u8[i], 255.0f) : p.src_f32[i];
        if (p.out_u8) p.out_u8[i] = p.src_u8 ? p.src_u8[i] : quant_u8(v);
        if (p.out_f32) p.out_f32[i] = v;
    }
}

template <class K>
static cudaError_t prefer_shared(K k) {
    return cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
}

cudaError_t spatial_prepare_device() {
    // the sweep's rings are static shared memory; prefer shared memory over L1
    cudaError_t e = prefer_shared(k_guided_transfer<kRowsWords>);
    if (e == cudaSuccess) e = prefer_shared(k_guided_transfer<kRowsWords16>);
    if (e == cudaSuccess) e = prefer_shared(k_guided_transfer<kRowsRagged>);
    if (e == cudaSuccess) e = prefer_shared(k_guided_transfer<kRowsFloat>);
    if (e == cudaSuccess) e = prefer_shared(k_guided_transfer<kRowsAny>);
    if (e == cudaSuccess) e = prefer_shared(k_guided_transfer_multi<kRowsWords>);
    if (e == cudaSuccess) e = prefer_shared(k_guided_transfer_multi<kRowsWords16>);
    if (e == cudaSuccess) e = prefer_shared(k_guided_transfer_multi<kRowsMixed>);
    return e;
}

// Warps of a guided launch over `units` units.  fixed: one segment per unit.
// Else the units are 16 rows (GS_UNIT) and a warp takes m or m - 1 of them in
// a row, for a segment of 16 m rows and 16 rows of halo.  A row costs a warp
// about 0.45 + 0.06 k us (x 1.2) with k warps on its SM (measured: 0.55 us at
// 1 to 4, 1.0 at 8, 1.17 at 12, the rings' limit), so few strips want short
// segments over many SMs and many want one long segment per warp: of the
// splits with at most 2, 4, .. 12 warps per SM the one with the least
// (m + 1) (0.45 + 0.06 k) is taken.  A launch with more work than fits in
// short segments still is one wave, without a partly filled last one.  A plain
// session's frame shares the GPU with its other frames' kernels, which need the
// shared memory and issue slots that fewer, longer segments leave: the fewest
// warps within `slack` percent of the least (3840x2160, frames in flight:
// 8 warps per SM 217 us a frame, the 11 of the least 227).
static int guided_warps(int units, bool fixed, int slack) {
    if (fixed) return units;
    constexpr int kSm = 148;
    int warps[6];
    long long cost[6], least = -1;
    for (int i = 0; i < 6; i++) {
        const int most = kSm * 2 * (i + 1);
        const int m = std::max(1, (units + most - 1) / most);
        warps[i] = (units + m - 1) / m;
        cost[i] = (m + 1LL) * (45 + 6LL * ((warps[i] + kSm - 1) / kSm));
        if (least < 0 || cost[i] < least) least = cost[i];
    }
    int i = 0;
    while (cost[i] * 100 > least * (100 + slack)) i++;
    return warps[i];
}

// guided filter: units of seg_rows rows of a strip (gx units per strip, gy
// strips; seg_rows filled in when 0); Gaussian: 32x32 tiles
unsigned transfer_grid(TransferParams& p, unsigned& gx, unsigned& gy) {
    if (p.edge_aware) {
        if (p.seg_rows <= 0) {
            const int f = fixed_rows(current_device());
            p.seg_rows = f > 0 ? f : GS_UNIT;
        }
        gx = (unsigned)((p.h + p.seg_rows - 1) / p.seg_rows);
        gy = (unsigned)((p.w + GS_OUT - 1) / GS_OUT);
    } else {
        gx = (unsigned)((p.w + TS - 1) / TS);
        gy = (unsigned)((p.h + TS - 1) / TS);
    }
    return gx * gy;
}

cudaError_t launch_transfer_multi(int edge_aware, const TransferParams* d_params, const int* d_map,
                                  unsigned blocks, int mode, cudaStream_t st) {
    if (blocks == 0) return cudaSuccess;
    if (!edge_aware) {
        k_gauss_transfer_multi<<<blocks, SP_THREADS, 0, st>>>(d_params, d_map);
        return cudaGetLastError();
    }
    const int warps = guided_warps((int)blocks, fixed_rows(current_device()) > 0, 0);
    const unsigned grid = (unsigned)((warps + GS_WARPS - 1) / GS_WARPS);
    if (mode == kRowsWords) k_guided_transfer_multi<kRowsWords><<<grid, GS_THREADS, 0, st>>>(d_params, d_map, warps);
    else if (mode == kRowsWords16) k_guided_transfer_multi<kRowsWords16><<<grid, GS_THREADS, 0, st>>>(d_params, d_map, warps);
    else k_guided_transfer_multi<kRowsMixed><<<grid, GS_THREADS, 0, st>>>(d_params, d_map, warps);
    return cudaGetLastError();
}

static cudaError_t launch_guided(const SpArgs& a, int units, bool fixed, cudaStream_t st) {
    const int warps = guided_warps(units, fixed, 10);
    const unsigned grid = (unsigned)((warps + GS_WARPS - 1) / GS_WARPS);
    switch (sweep_mode(a.p)) {
        case kRowsWords: k_guided_transfer<kRowsWords><<<grid, GS_THREADS, 0, st>>>(a, units, warps); break;
        case kRowsWords16: k_guided_transfer<kRowsWords16><<<grid, GS_THREADS, 0, st>>>(a, units, warps); break;
        case kRowsRagged: k_guided_transfer<kRowsRagged><<<grid, GS_THREADS, 0, st>>>(a, units, warps); break;
        case kRowsFloat: k_guided_transfer<kRowsFloat><<<grid, GS_THREADS, 0, st>>>(a, units, warps); break;
        default: k_guided_transfer<kRowsAny><<<grid, GS_THREADS, 0, st>>>(a, units, warps); break;
    }
    return cudaGetLastError();
}

// One stream's frame.  The output is the same however it is split.
cudaError_t launch_transfer(const TransferParams& p0, cudaStream_t st) {
    SpArgs a{p0};
    const bool fixed = a.p.seg_rows > 0;
    if (a.p.edge_aware && !fixed) a.p.seg_rows = GS_UNIT;
    unsigned gx, gy;
    const unsigned units = transfer_grid(a.p, gx, gy);
    if (a.p.edge_aware) return launch_guided(a, (int)units, fixed, st);
    k_gauss_transfer<<<dim3(gx, gy), SP_THREADS, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_passthrough(const TransferParams& p, cudaStream_t st) {
    SpArgs a{p};
    const long long n = (long long)p.w * p.h * 3;
    int blocks = (int)((n + 255) / 256);
    if (blocks > 148 * 8) blocks = 148 * 8;
    k_passthrough<<<blocks, 256, 0, st>>>(a);
    return cudaGetLastError();
}

// ---- the autotuner's trial of the batched sweep's segment height: a 3840 x 8640
// RGB24 frame (four 2160-row frames' worth of strips and segments, about the
// batched tick's warp count at 128 rows) as one task of the batched launch, each
// candidate set on the device as a tick would find it and timed over five
// launches after one warm-up; the fastest is kept.  Outputs do not depend on the
// choice.
cudaError_t guided_autotune(int dev, const int* cand, int nc, float* ms, int* chosen) {
    cudaError_t e = cudaSetDevice(dev);
    if (e != cudaSuccess) return e;
    const int W = 3840, H = 4 * 2160;
    const size_t P = (size_t)W * H;
    uint8_t *in = nullptr, *out = nullptr;
    float* gray = nullptr;
    void *dp = nullptr, *dmap = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    cudaStream_t st = nullptr;
    const int keep = guided_rows(dev);
    auto done = [&](cudaError_t r) {
        for (void* p : {(void*)in, (void*)out, (void*)gray, dp, dmap})
            if (p) cudaFree(p);
        if (e0) cudaEventDestroy(e0);
        if (e1) cudaEventDestroy(e1);
        if (st) cudaStreamDestroy(st);
        if (r != cudaSuccess) guided_set_rows(dev, keep);   // leave the device's choice as it was
        return r;
    };
    if ((e = cudaMalloc(&in, 3 * P)) != cudaSuccess) return done(e);
    if ((e = cudaMalloc(&out, 3 * P)) != cudaSuccess) return done(e);
    if ((e = cudaMalloc(&gray, P * sizeof(float))) != cudaSuccess) return done(e);
    if ((e = cudaMalloc(&dp, sizeof(TransferParams))) != cudaSuccess) return done(e);
    if ((e = cudaMalloc(&dmap, 8 * sizeof(int))) != cudaSuccess) return done(e);
    if ((e = cudaMemset(in, 0x5a, 3 * P)) != cudaSuccess) return done(e);
    if ((e = cudaMemset(gray, 0, P * sizeof(float))) != cudaSuccess) return done(e);
    if ((e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking)) != cudaSuccess) return done(e);
    if ((e = cudaEventCreate(&e0)) != cudaSuccess || (e = cudaEventCreate(&e1)) != cudaSuccess) return done(e);
    if ((e = spatial_prepare_device()) != cudaSuccess) return done(e);
    int best = keep;
    float best_ms = 1e30f;
    for (int k = 0; k < nc; k++) {
        guided_set_rows(dev, cand[k]);
        TransferParams tp{};
        tp.w = W;
        tp.h = H;
        tp.vec_end = (long long)P;
        tp.src_u8 = in;
        tp.gray_out = gray;
        tp.out_u8 = out;
        tp.edge_aware = 1;
        unsigned gx, gy;
        const unsigned units = transfer_grid(tp, gx, gy);
        const int map[5] = {1, 0, (int)units, (int)gx, (int)gy};
        if ((e = cudaMemcpy(dp, &tp, sizeof tp, cudaMemcpyHostToDevice)) != cudaSuccess) return done(e);
        if ((e = cudaMemcpy(dmap, map, sizeof map, cudaMemcpyHostToDevice)) != cudaSuccess) return done(e);
        for (int rep = 0; rep < 6; rep++) {
            if (rep == 1 && (e = cudaEventRecord(e0, st)) != cudaSuccess) return done(e);
            e = launch_transfer_multi(1, (const TransferParams*)dp, (const int*)dmap, units, transfer_rows_mode(tp), st);
            if (e != cudaSuccess) return done(e);
        }
        if ((e = cudaEventRecord(e1, st)) != cudaSuccess) return done(e);
        if ((e = cudaEventSynchronize(e1)) != cudaSuccess) return done(e);
        float t = 0.f;
        if ((e = cudaEventElapsedTime(&t, e0, e1)) != cudaSuccess) return done(e);
        ms[k] = t / 5.f;
        if (ms[k] < best_ms) {
            best_ms = ms[k];
            best = cand[k];
        }
    }
    guided_set_rows(dev, best);
    *chosen = best;
    return done(cudaSuccess);
}

}  // namespace wema
