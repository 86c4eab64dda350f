// dwt.cu - 2D CDF 9/7 lifting DWT, forward and inverse, one fused kernel per
// pyramid level, swept strip by strip (sweep.cuh): a warp lifts two neighbouring
// pairs of columns per lane and a pair of rows at a time, both directions in
// registers.
//
// Forward: RGB (converted on the way in, a channel at a time) or the previous
// level's LL in; LL and the three bands out, with the temporal filter's step on
// each coefficient as it is written (batched streams with FP32 state, after their
// first frame).  Inverse: the bands are amplified as they come in; planes out, or
// for colour at level 0 RGB.
//
// Sample and pair indices are 32-bit: the runtime caps frames at 2^28 pixels.
// Arithmetic is the reference's: x = fma(left + right, c, x), scalings as
// separate multiplies (dwt.c:45-170 as GCC -Ofast evaluates it), so
// coefficients are bit-exact.
//
// What bounds them: the latency of their loads and HBM at the large levels, the
// chain of steps of a short segment at the small ones, which are a tile's
// (dwt_tiles.cu) where that is the faster form.  Measured against the tiles, which
// load and lift 1.4 times the area through shared memory (thread instructions per
// pixel: forward with the filter's step 93 against 171, inverse 37 against 91):
//   3840x4320, level 0   forward with the filter's step 140 -> 118 us; inverse 55 -> 42
//   the 48-stream tick   level 0 forward 0.615 -> 0.578 ms, inverse 0.279 -> 0.182,
//                        levels 3..1 inverse 0.116 -> 0.088
#include <algorithm>
#include <atomic>
#include <type_traits>

#include "cascade.cuh"
#include "common.cuh"
#include "kernels.h"
#include "multi.cuh"
#include "row_copy.h"
#include "sweep.cuh"

namespace wema {

constexpr int SQ = 2;                    // pairs of columns per lane

// ----------------------------------------------------------------- forward
// A warp's inputs of FWD_RING consecutive pairs of rows in shared memory, copied
// in asynchronously FWD_RING - 1 ahead in whole 16-byte pieces: the strip's part
// of the two rows, and the temporal filter's state of the row of positions that
// the step finishes.
constexpr int FWD_RING = 3;
template <int MODE>
struct RowRing {
    static constexpr int PX = MODE == kSrcRgbU8 ? 3 : MODE == kSrcRgbF32 ? 12 : 4;   // bytes per sample
    static constexpr int PIECES = 64 * SQ * PX / 16 + 1;                             // one more: any alignment
    uint4 v[FWD_RING][2][PIECES];
};
struct StateRing {
    float4 v[FWD_RING][3][32 * SQ];
};

// What a sweep of channel z of a level uses of its parameters; what it rarely
// uses stays in g.  (A colour frame's three channels are swept apart, each
// converting the pixels to its own: the pixels are 3 of a channel's 34 bytes per
// pixel, and three channels' rings and lifting state in one warp would leave one
// CTA per SM.)
template <int MODE, bool H16>
struct FwdSweep {
    const FwdLevelParams& g;
    int z, iw, ih, sw, sh, n, vec_end;
    int inner;                           // rows whose copies may be whole pieces (row_copy.h)
    const void* src;                     // RGB24, float RGB, or the channel's plane
    float *coef, *ll, *dl;
    void* st;
    float c[10];
    bool ivec, cvec, svec;               // rows of the input plane, the outputs, the state start at vectors
    template <class A>
    __device__ __forceinline__ auto pick(const A& a) const {
        return z == 0 ? a[0] : z == 1 ? a[1] : a[2];
    }
    __device__ __forceinline__ FwdSweep(const FwdLevelParams& g_, int z_)
        : g(g_), z(z_), iw(g.iw), ih(g.ih), sw(g.sw), sh(g.sh), n((int)g.n), vec_end((int)g.vec_end) {
        inner = inner_rows(ih, RowRing<MODE>::PX * iw);
        coef = pick(g.coef);
        ll = pick(g.ll_out);
        dl = pick(g.iir_delta);
        st = pick(g.iir_state);
        src = MODE == kSrcPlanes ? (const void*)pick(g.src_planes) : MODE == kSrcRgbU8 ? (const void*)g.src_u8
                                                                                     : (const void*)g.src_f32;
#pragma unroll
        for (int k = 0; k < 10; k++) c[k] = g.iir_c[k];
        const uintptr_t outs = (uintptr_t)coef << (H16 ? 1 : 0) | (uintptr_t)ll | (uintptr_t)dl << (H16 ? 1 : 0);
        ivec = MODE == kSrcPlanes && !(iw & 3) && !((uintptr_t)src & 15);
        cvec = !(sw & 1) && !(outs & 7);
        svec = cvec && !((uintptr_t)st & 31);
    }
};

// the address of the strip's first sample of image row `row`
template <int MODE, class S>
__device__ __forceinline__ const uint8_t* row_start(const S& p, int row, int p0) {
    return static_cast<const uint8_t*>(p.src) + (long long)RowRing<MODE>::PX * (row * p.iw + 2 * p0);
}
// a row's part in 4-byte words, where 16-byte pieces may reach past the frame; out
// of line, as only the frame's first and last rows come here
__device__ __noinline__ void row_words(uint8_t* d, const uint8_t* q, int bytes) {
    const int off = (int)(reinterpret_cast<uintptr_t>(q) & 15), at = off & ~3;
    const int words = (off - at + bytes + 3) >> 2;
    for (int k = threadIdx.x & 31; k < words; k += 32) cp_async4(d + at + 4 * k, q - off + at + 4 * k);
}
// the strip's part of the two rows of pair j (a plane lies in the library's own
// memory, on either side of it too)
template <int MODE, class S>
__device__ __forceinline__ void row_issue(const S& p, RowRing<MODE>& ring, int slot, int j, int p0) {
    const int bytes = RowRing<MODE>::PX * min(64 * SQ, p.iw - 2 * p0);
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int row = mirror(2 * j + h, p.ih);
        const uint8_t* q = row_start<MODE>(p, row, p0);
        if (MODE == kSrcPlanes || row_inner(row, p.inner)) {   // (uniform)
            const int off = (int)(reinterpret_cast<uintptr_t>(q) & 15);
            const int pieces = (off + bytes + 15) >> 4;
            for (int k = threadIdx.x & 31; k < pieces; k += 32) cp_async16(&ring.v[slot][h][k], q - off + 16 * k);
        } else {
            row_words(reinterpret_cast<uint8_t*>(ring.v[slot][h]), q, bytes);
        }
    }
}
// the samples of row h of the pair
template <int MODE, class S>
__device__ __forceinline__ void row_samples(const S& p, const RowRing<MODE>& ring, int slot, int h, int row, int p0, int g,
                                            float (&out)[2 * SQ]) {
    const int lane = threadIdx.x & 31;
    const int off = (int)(reinterpret_cast<uintptr_t>(row_start<MODE>(p, row, p0)) & 15);
    const uint8_t* at = reinterpret_cast<const uint8_t*>(ring.v[slot][h]) + off + 2 * SQ * RowRing<MODE>::PX * lane;
    if constexpr (MODE == kSrcPlanes) {
        if (p.ivec) {
            const float4 w = *reinterpret_cast<const float4*>(at);
            out[0] = w.x; out[1] = w.y; out[2] = w.z; out[3] = w.w;
        } else {
#pragma unroll
            for (int k = 0; k < 2 * SQ; k++) out[k] = reinterpret_cast<const float*>(at)[k];
        }
    } else {
        float rgb[6 * SQ];
        if constexpr (MODE == kSrcRgbU8) {
            const int sh = 8 * (int)(off & 3);   // (a lane's 12 bytes: the same place in its words)
            const uint32_t* q = reinterpret_cast<const uint32_t*>(at - (off & 3));
            uint32_t w[4];
#pragma unroll
            for (int k = 0; k < 4; k++) w[k] = q[k];
#pragma unroll
            for (int k = 0; k < 6 * SQ; k++)     // fl(byte / 255)
                rgb[k] = byte_of(__funnelshift_r(w[k >> 2], w[(k >> 2) + 1], sh), k & 3);
        } else {
#pragma unroll
            for (int k = 0; k < 6 * SQ; k++) rgb[k] = reinterpret_cast<const float*>(at)[k];
        }
        // the strip's row wholly in the vector body (every row but the frame's
        // last): no pixel needs the epilogue's form
        const bool all = row * p.iw + min(p.iw, 2 * (p0 + 32 * SQ)) <= p.vec_end;
        const int pi = row * p.iw + 2 * g;
#pragma unroll
        for (int k = 0; k < 2 * SQ; k++) {
            const float r = rgb[3 * k], gg = rgb[3 * k + 1], b = rgb[3 * k + 2];
            const bool vec = all || pi + k < p.vec_end;
            if (p.z == 0) {
                out[k] = vec ? luma_vec(r, gg, b) : luma_tail(r, gg, b);
            } else {                     // (uniform)
                float y, cb, cr;
                if (vec) ycbcr_vec(r, gg, b, y, cb, cr);
                else ycbcr_tail(r, gg, b, y, cb, cr);
                out[k] = p.z == 1 ? cb : cr;
            }
        }
    }
}
// the state of the strip's positions of row y
template <class S>
__device__ __forceinline__ void state_issue(const S& p, StateRing& ring, int slot, int y, const Strip<SQ>& s) {
    const int lane = threadIdx.x & 31;
    const float4* const st = static_cast<const float4*>(p.st);
#pragma unroll
    for (int b = 0; b < 3; b++)
#pragma unroll
        for (int i = 0; i < SQ; i++) {
            const int t = 32 * i + lane;
            if (t >= s.lo && t < s.hi) cp_async16(&ring.v[slot][b][t], st + (b * p.n + y * p.sw + s.p0 + t));
        }
}
// two positions' state out: 32 bytes in one store where aligned
__device__ __forceinline__ void st_state2(float4* s, bool vec, bool second, const float4& a, const float4& b) {
    if (vec) {
        asm volatile("st.global.cs.v8.f32 [%8], {%0,%1,%2,%3,%4,%5,%6,%7};" ::"f"(a.x), "f"(a.y), "f"(a.z), "f"(a.w),
                     "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w), "l"(s) : "memory");
    } else {
        __stcs(s, a);
        if (second) __stcs(s + 1, b);
    }
}
__device__ __forceinline__ void st_pair(float* p, int i, const float (&v)[SQ], bool h, bool vec, bool second) {
    if (vec && h) {
        *reinterpret_cast<__half2*>(reinterpret_cast<__half*>(p) + i) = __floats2half2_rn(v[0], v[1]);
    } else if (vec) {
        *reinterpret_cast<float2*>(p + i) = make_float2(v[0], v[1]);
    } else {
        pl_st(p, i, v[0], h);
        if (second) pl_st(p, i + 1, v[1], h);
    }
}

// an element that the same launch may have written (the levels of k_dwt_fwd_tail)
__device__ __forceinline__ float pl_ldcg(const float* p, int i, bool h) {
    return h ? __half2float(__ldcg(reinterpret_cast<const __half*>(p) + i)) : __ldcg(p + i);
}

// Write-out of a lane's SQ positions of row y of one channel: LL, the bands LH,
// HH, HL (v[0..2]), and the temporal filter's step on them (cascade.cuh): the
// filter reads the coefficient as stored (FP16-rounded in the planes_fp16
// variant), so the deltas equal those of the separate filter kernel bit for bit.
// tail: some coefficient of the row takes the scalar-tail form (uniform).
template <bool H16, class S>
__device__ __forceinline__ void put_level(const S& p, int y, int g, bool second, bool tail,
                                          const float4 (*state)[32 * SQ], const float (&ll)[SQ], float (&v)[3][SQ]) {
    const int o = y * p.sw + g, lane = threadIdx.x & 31;
    const bool cvec = p.cvec;
    st_pair(p.ll, o, ll, false, cvec, second);
#pragma unroll
    for (int b = 0; b < 3; b++) st_pair(p.coef, b * p.n + o, v[b], H16, cvec, second);
    if (!p.st) return;
#pragma unroll
    for (int b = 0; b < 3; b++) {
        const int u = b * p.n + o;
        if (H16) {
#pragma unroll
            for (int k = 0; k < SQ; k++) v[b][k] = __half2float(__float2half_rn(v[b][k]));
        }
        float4 s[SQ];
#pragma unroll
        for (int k = 0; k < SQ; k++) s[k] = state[b][SQ * lane + k];
        if (!tail) {
#pragma unroll
            for (int k = 0; k < SQ; k++) v[b][k] = cascade(p.c, s[k], v[b][k], false);
        } else {
            const long long u6 = p.g.iir_off6 + u;
#pragma unroll
            for (int k = 0; k < SQ; k++) v[b][k] = cascade(p.c, s[k], v[b][k], u6 + k >= p.g.iir_simd_end);
        }
        st_state2(static_cast<float4*>(p.st) + u, p.svec, second, s[0], s[1]);
        st_pair(p.dl, u, v[b], H16, cvec, second);
    }
}

template <int MODE, bool H16, bool EDGE>
__device__ __forceinline__ void fwd_sweep(const FwdSweep<MODE, H16>& p, RowRing<MODE>& rows, StateRing* states,
                                          const Strip<SQ>& s, int ya, int yb) {
    const int lane = threadIdx.x & 31;
    const int g = s.p0 + SQ * lane;
    const bool live = !EDGE || p.ih >= 2;
    const bool writer = SQ * lane >= s.lo && SQ * lane < s.hi;
    const bool second = SQ * lane + 1 < s.hi;
    ColumnForward<SQ> L, H;
#pragma unroll
    for (int k = 0; k < SQ; k++) {
        L.e0[k] = L.o0[k] = L.o1[k] = L.e1[k] = L.o2[k] = 0.0f;
        H.e0[k] = H.o0[k] = H.o1[k] = H.e1[k] = H.o2[k] = 0.0f;
    }
    const int j0 = ya - 2, j1 = yb + 2;
    auto issue = [&](int j, int slot) {
        if (j < j1) row_issue<MODE>(p, rows, slot, j, s.p0);
        if (p.st && j - 2 >= ya && j < j1) state_issue(p, *states, slot, j - 2, s);
        cp_commit();
    };
    __syncwarp();                            // the last segment's readers are done with the rings
#pragma unroll
    for (int i = 0; i < FWD_RING - 1; i++) issue(j0 + i, i);
    int slot = 0;
#pragma unroll 1
    for (int j = j0; j < j1; j++) {
        float a[2 * SQ], b[2 * SQ];
        cp_wait<FWD_RING - 2>();
        __syncwarp();                        // every lane's pieces are in, and the slot before is read
        row_samples<MODE>(p, rows, slot, 0, mirror(2 * j, p.ih), s.p0, g, a);
        row_samples<MODE>(p, rows, slot, 1, mirror(2 * j + 1, p.ih), s.p0, g, b);
        issue(j + FWD_RING - 1, slot == 0 ? FWD_RING - 1 : slot - 1);
        if (MODE != kSrcPlanes && p.g.plane_out[0] && writer && j >= ya && j < yb) {
            float* const plane = p.pick(p.g.plane_out);
#pragma unroll
            for (int k = 0; k < 2 * SQ; k++)
                if (2 * g + k < p.iw) {
                    plane[2 * j * p.iw + 2 * g + k] = a[k];
                    if (2 * j + 1 < p.ih) plane[(2 * j + 1) * p.iw + 2 * g + k] = b[k];
                }
        }
        const int y = j - 2, now = slot;
        slot = slot == FWD_RING - 1 ? 0 : slot + 1;
        float e[SQ], o[SQ], he[SQ], ho[SQ];
#pragma unroll
        for (int k = 0; k < SQ; k++) {
            e[k] = a[2 * k];
            he[k] = a[2 * k + 1];
            o[k] = b[2 * k];
            ho[k] = b[2 * k + 1];
        }
        row_forward<SQ, EDGE>(e, he, g, p.iw);
        row_forward<SQ, EDGE>(o, ho, g, p.iw);
        L.step(e, o, live);
        H.step(he, ho, live);
        if (y < ya || !writer) continue;
        float v[3][SQ];
#pragma unroll
        for (int k = 0; k < SQ; k++) {
            v[0][k] = o[k];
            v[1][k] = ho[k];
            v[2][k] = he[k];
        }
        // stale entries of odd-sized levels take the previous level's value at
        // the same index
        const bool hy = 2 * y + 1 < p.ih;
        if (EDGE || !hy) {
            const float* pv = p.pick(p.g.prev);
            const int pn = (int)p.g.prev_n;
#pragma unroll
            for (int k = 0; k < SQ; k++) {
                const bool hx = !EDGE || 2 * (g + k) + 1 < p.iw;
                const int at = y * p.sw + g + k;
                if (k && !second) break;
                if (!hy) v[0][k] = pv ? pl_ldcg(pv, at, H16) : 0.0f;
                if (!(hx && hy)) v[1][k] = pv ? pl_ldcg(pv, pn + at, H16) : 0.0f;
                if (!hx) v[2][k] = pv ? pl_ldcg(pv, 2 * pn + at, H16) : 0.0f;
            }
        }
        const bool tail = p.g.iir_off6 + 2 * p.n + (long long)y * p.sw + s.p0 + s.hi > p.g.iir_simd_end;
        put_level<H16>(p, y, g, second, tail, states->v[now], e, v);
    }
}

// whether a strip's rows need the border forms: the line ends inside a lane, or
// the level is a single row or column
__device__ __forceinline__ bool strip_edge(const Strip<SQ>& s, int w, int h, int pairs) {
    return (w % (2 * SQ) != 0 && s.p0 + 32 * SQ >= pairs) || w < 2 || h < 2;
}

// units u0 .. u0 + n - 1 (g.unit pairs of rows each) of a CTA's group of strips.
// NARROW: the level may be one or two strips wide, whose rows the warps share; a
// form of its own, as rows that differ from warp to warp make the wide levels'
// sweeps 5 to 8% longer.
template <int MODE, bool H16, bool NARROW>
__device__ __forceinline__ void fwd_segment(const FwdLevelParams& g, int z, RowRing<MODE>& rows, StateRing* states,
                                            int group, int u0, int n) {
    const FwdSweep<MODE, H16> p(g, z);
    const WarpRows<NARROW> r(group, sweep_across(p.sw, SQ), u0 * g.unit, min((u0 + n) * g.unit, p.sh));
    const Strip<SQ> s(r.strip, p.sw);
    if (s.hi <= s.lo || (NARROW && r.yb <= r.ya)) return;
    if (strip_edge(s, p.iw, p.ih, p.sw)) fwd_sweep<MODE, H16, true>(p, rows, states, s, r.ya, r.yb);
    else fwd_sweep<MODE, H16, false>(p, rows, states, s, r.ya, r.yb);
}

// ----------------------------------------------------------------- inverse
// what a sweep of a level uses of its parameters, for C channels from z on.
// OUT: kOutPlanes (one channel) or kOutRgb (three)
template <int C, bool H16>
struct InvSweep {
    int ow, oh, sw, sh, n;
    const float *ll[C], *coef[C], *delta[C];
    float* out[C];
    float thr[C], al[C];
    uint8_t* u8;
    float* f32;
    bool out16, vec, ovec, wvec;         // inputs, output planes, output bytes start at vectors
    __device__ __forceinline__ InvSweep(const InvLevelParams& g, int z)
        : ow(g.ow), oh(g.oh), sw(g.sw), sh(g.sh), n((int)g.n), u8(g.out_u8), f32(g.out_f32) {
        uintptr_t in = 0, planes = 0;
#pragma unroll
        for (int k = 0; k < C; k++) {
            const int i = C > 1 ? k : z;
            auto pick = [&](const auto& a) { return i == 0 ? a[0] : i == 1 ? a[1] : a[2]; };
            ll[k] = pick(g.ll);
            coef[k] = pick(g.coef);
            delta[k] = pick(g.delta);
            out[k] = pick(g.out_planes);
            al[k] = pick(g.alpha);
            thr[k] = g.thr[i];
            in |= (uintptr_t)ll[k] | (uintptr_t)coef[k] << (H16 ? 1 : 0) | (uintptr_t)delta[k] << (H16 ? 1 : 0);
            planes |= (uintptr_t)out[k];
        }
        out16 = H16 && g.out16;
        vec = !(sw & 1) && !(in & 7);
        ovec = !out16 && !(ow & 3) && !(planes & 15);
        wvec = !(ow & 3) && !((uintptr_t)u8 & 3);
    }
};

// SQ neighbouring elements of a plane as they were loaded: FP16 ones packed in
// w[0] (a vector load) or one by one, widened when they are used, a pair of rows
// later
// FRESH: the same launch may have written them (the levels of k_dwt_inv_tail):
// not through the read-only path
template <bool H16, bool FRESH = false>
struct Elems {
    float w[SQ];
    template <class T>
    static __device__ __forceinline__ T ld(const T* p) {
        if constexpr (FRESH) return __ldcg(p);
        else return __ldg(p);
    }
    __device__ __forceinline__ void load(const float* p, int i, bool vec, int n) {
        if (H16) {
            const __half* q = reinterpret_cast<const __half*>(p) + i;
            if (vec) {
                w[0] = ld(reinterpret_cast<const float*>(q));
            } else {
#pragma unroll
                for (int k = 0; k < SQ; k++)
                    if (k < n) w[k] = __uint_as_float(ld(reinterpret_cast<const unsigned short*>(q + k)));
            }
        } else if (vec) {
            const float2 a = ld(reinterpret_cast<const float2*>(p + i));
            w[0] = a.x; w[1] = a.y;
        } else {
#pragma unroll
            for (int k = 0; k < SQ; k++)
                if (k < n) w[k] = ld(p + i + k);
        }
    }
    __device__ __forceinline__ void get(bool vec, float (&v)[SQ]) const {
        if (H16) {
            const uint32_t a = __float_as_uint(w[0]);
            const uint32_t b = vec ? a : __byte_perm(a, __float_as_uint(w[1]), 0x5410);
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&b));
            v[0] = f.x; v[1] = f.y;
        } else {
            v[0] = w[0]; v[1] = w[1];
        }
    }
};

// The loads of one pair of rows: LL and the three bands (LH, HH, HL) with their
// deltas, per channel.
template <int C, bool H16, bool FRESH>
struct InvRows {
    Elems<false, FRESH> ll[C];
    Elems<H16> x[C][3], d[C][3];

    // row pair j; g: the lane's first pair
    __device__ __forceinline__ void issue(const InvSweep<C, H16>& p, int j, int g) {
        const int n = p.sw - g;
        if (n <= 0) return;
        const int ie = (mirror(2 * j, p.oh) >> 1) * p.sw + g, io = (mirror(2 * j + 1, p.oh) >> 1) * p.sw + g;
        const int at[3] = {io, p.n + io, 2 * p.n + ie};
#pragma unroll
        for (int c = 0; c < C; c++) {
            ll[c].load(p.ll[c], ie, p.vec, n);
#pragma unroll
            for (int b = 0; b < 3; b++) {
                x[c][b].load(p.coef[c], at[b], p.vec, n);
                d[c][b].load(p.delta[c], at[b], p.vec, n);
            }
        }
    }
    __device__ __forceinline__ void amplified(const InvSweep<C, H16>& p, int c, int b, float (&v)[SQ]) const {
        float dl[SQ];
        x[c][b].get(p.vec, v);
        d[c][b].get(p.vec, dl);
#pragma unroll
        for (int k = 0; k < SQ; k++) v[k] = fabsf(v[k]) > p.thr[c] ? __fmaf_rn(dl[k], p.al[c], v[k]) : v[k];
    }
};

// 2 SQ neighbouring samples of a row: even ones in a, odd ones in b
__device__ __forceinline__ void put_samples(float* out, int at, int left, bool vec, bool h16, const float (&a)[SQ],
                                            const float (&b)[SQ]) {
    if (vec) {
        *reinterpret_cast<float4*>(out + at) = make_float4(a[0], b[0], a[1], b[1]);
    } else {
#pragma unroll
        for (int k = 0; k < SQ; k++) {
            if (2 * k < left) pl_st(out, at + 2 * k, a[k], h16);
            if (2 * k + 1 < left) pl_st(out, at + 2 * k + 1, b[k], h16);
        }
    }
}

template <int C, int OUT, bool H16, bool EDGE, bool FRESH = false>
__device__ __forceinline__ void inv_sweep(const InvSweep<C, H16>& p, const Strip<SQ>& s, int ya, int yb) {
    const int lane = threadIdx.x & 31;
    const int g = s.p0 + SQ * lane;
    const int ow = p.ow, oh = p.oh;
    const bool live = !EDGE || oh >= 2;
    const bool writer = SQ * lane >= s.lo && SQ * lane < s.hi;
    ColumnInverse<SQ> L[C], H[C];
#pragma unroll
    for (int c = 0; c < C; c++)
#pragma unroll
        for (int k = 0; k < SQ; k++) {
            L[c].o0[k] = L[c].e1[k] = L[c].o1[k] = L[c].e2[k] = 0.0f;
            H[c].o0[k] = H[c].e1[k] = H[c].o1[k] = H[c].e2[k] = 0.0f;
        }
    InvRows<C, H16, FRESH> r;
    const int j1 = yb + 2;
    r.issue(p, ya - 2, g);
#pragma unroll 1
    for (int j = ya - 2; j < j1; j++) {
        // v[c][h]: row h of the pair, v[c][h][0] its even samples and [1] its odd
        float v[C][2][2][SQ];
#pragma unroll
        for (int c = 0; c < C; c++) {
#pragma unroll
            for (int k = 0; k < SQ; k++) v[c][0][0][k] = r.ll[c].w[k];
            r.amplified(p, c, 0, v[c][1][0]);
            r.amplified(p, c, 1, v[c][1][1]);
            r.amplified(p, c, 2, v[c][0][1]);
        }
        if (j + 1 < j1) r.issue(p, j + 1, g);   // in flight while this pair of rows is lifted
#pragma unroll
        for (int c = 0; c < C; c++) {
            L[c].step(v[c][0][0], v[c][1][0], live);
            H[c].step(v[c][0][1], v[c][1][1], live);
        }
        const int y = j - 2;
        if (y < ya) continue;
#pragma unroll
        for (int c = 0; c < C; c++) {
            row_inverse<SQ, EDGE>(v[c][0][0], v[c][0][1], g, ow);
            row_inverse<SQ, EDGE>(v[c][1][0], v[c][1][1], g, ow);
        }
        if (!writer) continue;
        const int left = ow - 2 * g;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            if (2 * y + h >= oh) break;
            const int at = (2 * y + h) * ow + 2 * g;
            if (OUT == kOutPlanes || p.out[0]) {
#pragma unroll
                for (int c = 0; c < C; c++) put_samples(p.out[c], at, left, p.ovec, p.out16, v[c][h][0], v[c][h][1]);
            }
            if constexpr (OUT == kOutRgb) {
                float rgb[6 * SQ];
#pragma unroll
                for (int k = 0; k < 2 * SQ; k++)
                    ycbcr_to_rgb(v[0][h][k & 1][k >> 1], v[1][h][k & 1][k >> 1], v[2][h][k & 1][k >> 1], rgb[3 * k],
                                 rgb[3 * k + 1], rgb[3 * k + 2]);
                if (p.u8 && p.wvec) {
                    uint32_t* w = reinterpret_cast<uint32_t*>(p.u8 + 3 * at);
#pragma unroll
                    for (int k = 0; k < 3; k++)   // low bytes of four quantised values into one word
                        w[k] = __byte_perm(__byte_perm(quant_bits(rgb[4 * k]), quant_bits(rgb[4 * k + 1]), 0x0040u),
                                           __byte_perm(quant_bits(rgb[4 * k + 2]), quant_bits(rgb[4 * k + 3]), 0x0040u),
                                           0x5410u);
                } else if (p.u8) {
#pragma unroll
                    for (int k = 0; k < 6 * SQ; k++)
                        if (k < 3 * left) p.u8[3 * at + k] = (uint8_t)quant_bits(rgb[k]);
                }
                if (p.f32) {
#pragma unroll
                    for (int k = 0; k < 6 * SQ; k++)
                        if (k < 3 * left) p.f32[3 * at + k] = rgb[k];
                }
            }
        }
    }
}

template <int C, int OUT, bool H16, bool NARROW>
__device__ __forceinline__ void inv_segment(const InvLevelParams& g, int z, int group, int u0, int n) {
    const InvSweep<C, H16> p(g, z);
    const WarpRows<NARROW> r(group, sweep_across(p.sw, SQ), u0 * g.unit, min((u0 + n) * g.unit, p.sh));
    const Strip<SQ> s(r.strip, p.sw);
    if (s.hi <= s.lo || (NARROW && r.yb <= r.ya)) return;
    if (strip_edge(s, p.ow, p.oh, p.sw)) inv_sweep<C, OUT, H16, true>(p, s, r.ya, r.yb);
    else inv_sweep<C, OUT, H16, false>(p, s, r.ya, r.yb);
}

// ------------------------------------------------------------- wrappers
// A launch's work is counted in units of `unit` pairs of rows of a CTA's group
// of strips; each CTA takes an even share of consecutive units, and those of one
// group are one segment.  The channel is the units' third index, but for the
// inverse's RGB out, which takes a colour frame's three channels together.
//
// CTAs per SM asked of the register allocator and counted on by the split:
// forward 5 (96 registers), 4 with the filter's rings beside it (47 KB of shared
// memory), 3 from float frames; inverse 5, RGB out 2.
constexpr int fwd_res(int mode, bool rings) { return mode == kSrcRgbF32 ? 3 : rings ? 4 : 5; }
constexpr int inv_res(int C) { return C == 3 ? 2 : 5; }

// Storage types: FP32, or the planes_fp16 variant's FP16 planes (H16): each launch's
// kernel is compiled for its own.
// f(first unit in the group, group, channel, units) for each segment of this CTA
template <class F>
__device__ __forceinline__ void each_segment(int units, int per, int groups, F f) {
    int2 u = unit_share(units, blockIdx.x, gridDim.x);
    while (u.x < u.y) {
        const int row = u.x % per, col = u.x / per, n = min(u.y - u.x, per - row);
        f(row, col % groups, col / groups, n);
        u.x += n;
    }
}

template <int MODE, bool H16>
__global__ void __launch_bounds__(SW_THREADS, fwd_res(MODE, false)) k_dwt_fwd(const __grid_constant__ FwdLevelParams g, int units) {
    __shared__ RowRing<MODE> rows[SW_WARPS];
    // (a plain session's filter is a launch of its own: no state here)
    each_segment(units, (g.sh + g.unit - 1) / g.unit, sweep_groups(g.sw, SQ), [&](int row, int group, int z, int n) {
        fwd_segment<MODE, H16, false>(g, z, rows[threadIdx.x >> 5], nullptr, group, row, n);
    });
}
template <int C, int OUT, bool H16>
__global__ void __launch_bounds__(SW_THREADS, inv_res(C)) k_dwt_inv(const __grid_constant__ InvLevelParams g, int units) {
    each_segment(units, (g.sh + g.unit - 1) / g.unit, sweep_groups(g.sw, SQ), [&](int row, int group, int z, int n) {
        inv_segment<C, OUT, H16, false>(g, z, group, row, n);
    });
}

// The coarser levels of a small frame in one launch: a cluster per channel takes
// them in turn, with a cluster barrier between two levels.  Warps of a sweep do not
// meet, so each takes an even share of a level's rows of strips.
// What bounds it: the chain of a warp's steps (rows + 4 of them at each level); a
// level of few rows launched apart costs more than that in the host's launch
// (about 2.5 us) and the wait for the kernel before.  12 warps: the rings' 38 KB.
constexpr int TAIL_CTAS = 8, TAIL_WARPS = 12;
template <class P>
struct LevelTail {
    P lv[3];                             // in the order they run
    int count;
};
// f(strip, first pair of rows, end) for each of this warp's shares
template <class F>
__device__ __forceinline__ void tail_shares(int sw, int sh, F f) {
    const int strips = (sw + SW_LANES * SQ - 1) / (SW_LANES * SQ);
    int2 u = unit_share(strips * sh, blockIdx.x * TAIL_WARPS + (threadIdx.x >> 5), TAIL_CTAS * TAIL_WARPS);
    while (u.x < u.y) {
        const int s = u.x / sh, y = u.x % sh, n = min(u.y - u.x, sh - y);
        f(Strip<SQ>(s, sw), y, y + n);
        u.x += n;
    }
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}
template <bool H16>
__global__ void __cluster_dims__(TAIL_CTAS, 1, 1) __launch_bounds__(32 * TAIL_WARPS)
    k_dwt_fwd_tail(const __grid_constant__ LevelTail<FwdLevelParams> t) {
    __shared__ RowRing<kSrcPlanes> rows[TAIL_WARPS];
#pragma unroll 1
    for (int l = 0; l < t.count; l++) {
        if (l) cluster_barrier();
        const FwdSweep<kSrcPlanes, H16> p(t.lv[l], blockIdx.y);
        tail_shares(p.sw, p.sh, [&](const Strip<SQ>& s, int ya, int yb) {
            fwd_sweep<kSrcPlanes, H16, true>(p, rows[threadIdx.x >> 5], nullptr, s, ya, yb);
        });
    }
}
template <bool H16>
__global__ void __cluster_dims__(TAIL_CTAS, 1, 1) __launch_bounds__(32 * TAIL_WARPS)
    k_dwt_inv_tail(const __grid_constant__ LevelTail<InvLevelParams> t) {
#pragma unroll 1
    for (int l = 0; l < t.count; l++) {
        if (l) cluster_barrier();
        const InvSweep<1, H16> p(t.lv[l], blockIdx.y);
        tail_shares(p.sw, p.sh, [&](const Strip<SQ>& s, int ya, int yb) {
            inv_sweep<1, kOutPlanes, H16, true, true>(p, s, ya, yb);
        });
    }
}
// batched (task = stream; params in device memory, one entry per task): the map
// counts units
template <class F>
__device__ __forceinline__ void each_task(const int* map, F f) {
    int2 u = unit_share(map[1 + map[0]], blockIdx.x, gridDim.x);
    while (u.x < u.y) {
        const TaskBlock t = task_block(map, u.x);
        const int n = min(u.y - u.x, map[map[0] + 2 + t.task] - t.x);
        f(t, n);
        u.x += n;
    }
}
template <int MODE, bool H16, bool NARROW>
__global__ void __launch_bounds__(SW_THREADS, fwd_res(MODE, true))
    k_dwt_fwd_multi(const FwdLevelParams* __restrict__ ps, const int* __restrict__ map) {
    extern __shared__ __align__(16) unsigned char fwd_smem[];
    StateRing* const states = reinterpret_cast<StateRing*>(fwd_smem) + (threadIdx.x >> 5);
    RowRing<MODE>& rows = reinterpret_cast<RowRing<MODE>*>(fwd_smem + SW_WARPS * sizeof(StateRing))[threadIdx.x >> 5];
    each_task(map, [&](const TaskBlock& t, int n) {
        fwd_segment<MODE, H16, NARROW>(ps[t.task], t.z, rows, states, t.y, t.x, n);
    });
}
template <int C, int OUT, bool H16, bool NARROW>
__global__ void __launch_bounds__(SW_THREADS, inv_res(C))
    k_dwt_inv_multi(const InvLevelParams* __restrict__ ps, const int* __restrict__ map) {
    each_task(map, [&](const TaskBlock& t, int n) {
        inv_segment<C, OUT, H16, NARROW>(ps[t.task], t.z, t.y, t.x, n);
    });
}

// ---- tuning of the batched sweeps, per device: variant v = 3 * i + k, at most
// kRes[inverse][i] CTAs per SM in units of kUnit[k] pairs of rows; the most is what
// fits of the one-channel kernels (the colour inverse fits 2 whatever is set)
constexpr int kDwtVariants = 9;
static const int kRes[2][3] = {{2, 3, 4}, {3, 4, 5}}, kUnit[3] = {1, 2, 4};
static std::atomic<int> g_dwt_var[64][2];     // [device][0 forward, 1 inverse], value + 1

static int dwt_dev_now() {
    int d = 0;
    cudaGetDevice(&d);
    return d;
}
int dwt_variant(int dev, int inverse) {
    const int v = (dev >= 0 && dev < 64) ? g_dwt_var[dev][inverse ? 1 : 0].load() : 0;
    return v > 0 ? v - 1 : 2 * 3 + 1;         // until tuned: the most CTAs per SM, 2 pairs of rows
}
bool dwt_set_variant(int dev, int inverse, int v) {
    if (dev < 0 || dev >= 64 || v < 0 || v >= kDwtVariants) return false;
    g_dwt_var[dev][inverse ? 1 : 0].store(v + 1);
    return true;
}
void dwt_variant_shape(int v, int inverse, int* res, int* unit) {
    *res = kRes[inverse ? 1 : 0][v / 3];
    *unit = kUnit[v % 3];
}

// CTAs of a sweep over `units` units of `unit` pairs of rows, an even share each:
// a segment of m units costs m unit + 4 steps (two pairs of rows of
// halo on either side), a step about 2 + k with k CTAs on the SM (0.5 us alone,
// 1.5 us with five).
static int sweep_ctas(int units, int unit, int res) {
    constexpr int kSm = 148;
    int best = units;
    long long least = -1;
    for (int k = 1; k <= res; k++) {
        const int most = kSm * k;
        const int m = std::max(1, (units + most - 1) / most);
        const int ctas = (units + m - 1) / m;
        const long long cost = ((long long)m * unit + 4) * (2 + (ctas + kSm - 1) / kSm);
        if (least < 0 || cost <= least) {
            least = cost;
            best = ctas;
        }
    }
    return best;
}
// more: CTAs per SM above the setting's (one stream's forward, without the filter's
// rings, fits one more than the batched)
static int ctas_for(int units, int inverse, int most, int more = 0) {
    int res, unit;
    dwt_variant_shape(dwt_variant(dwt_dev_now(), inverse), inverse, &res, &unit);
    return sweep_ctas(units, unit, std::min(res + more, most));
}

// ----------------------------------------------------------------- launch
static unsigned sweep_grid(int& unit, int sw, int sh, int channels_z, int inverse, bool narrow, unsigned& gx, unsigned& gy) {
    int res;
    dwt_variant_shape(dwt_variant(dwt_dev_now(), inverse), inverse, &res, &unit);
    if (narrow) unit *= SW_WARPS / sweep_across(sw, SQ);   // (a warp's rows stay the setting's)
    gx = (unsigned)((sh + unit - 1) / unit);
    gy = (unsigned)sweep_groups(sw, SQ);
    return gx * gy * (unsigned)channels_z;
}
bool dwt_narrow(int sw) { return sweep_across(sw, SQ) < SW_WARPS; }
// a task's units (gx per group of strips, gy groups), and sets p.unit; or its tiles
unsigned dwt_fwd_grid(FwdLevelParams& p, int channels_z, int form, unsigned& gx, unsigned& gy) {
    if (form >= kDwtTiles) return tiles_grid(p.sw, p.sh, channels_z, gx, gy);
    return sweep_grid(p.unit, p.sw, p.sh, channels_z, 0, true, gx, gy);
}
unsigned dwt_inv_grid(InvLevelParams& p, int channels_z, int form, unsigned& gx, unsigned& gy) {
    if (form >= kDwtTiles) return tiles_grid(p.sw, p.sh, channels_z, gx, gy);
    return sweep_grid(p.unit, p.sw, p.sh, channels_z, 1, true, gx, gy);
}

template <int MODE>
constexpr int ring_bytes() { return (int)(SW_WARPS * (sizeof(StateRing) + sizeof(RowRing<MODE>))); }

// the forward's rings: above the 48 KB default, and shared memory before
// first-level cache; call once per device
template <int MODE>
static cudaError_t prepare_fwd() {
    cudaError_t e = cudaSuccess;
    for (const void* k : {(const void*)k_dwt_fwd_multi<MODE, false, false>, (const void*)k_dwt_fwd_multi<MODE, true, false>,
                          (const void*)k_dwt_fwd_multi<MODE, false, true>, (const void*)k_dwt_fwd_multi<MODE, true, true>}) {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, ring_bytes<MODE>());
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    }
    return e;
}
cudaError_t dwt_prepare_device() {
    cudaError_t e = prepare_fwd<kSrcRgbU8>();
    if (e == cudaSuccess) e = prepare_fwd<kSrcPlanes>();
    return e == cudaSuccess ? tiles_prepare_device() : e;
}

template <int MODE, bool NARROW>
static void go_fwd_multi(bool h16, const FwdLevelParams* ps, const int* map, int ctas, cudaStream_t st) {
    if (h16) k_dwt_fwd_multi<MODE, true, NARROW><<<ctas, SW_THREADS, ring_bytes<MODE>(), st>>>(ps, map);
    else k_dwt_fwd_multi<MODE, false, NARROW><<<ctas, SW_THREADS, ring_bytes<MODE>(), st>>>(ps, map);
}
cudaError_t launch_dwt_fwd_multi(int mode, int channels, const FwdLevelParams* d_params, const int* d_map, unsigned blocks,
                                 int form, bool narrow, cudaStream_t st) {
    if (blocks == 0) return cudaSuccess;
    if (form >= kDwtTiles) return launch_tiles_fwd_multi(mode, channels, d_params, d_map, blocks, form == kDwtTiles16, st);
    const int n = ctas_for((int)blocks, 0, fwd_res(mode, true));
    const bool h16 = form == kDwtSweep16;
    if (mode == kSrcPlanes && narrow) go_fwd_multi<kSrcPlanes, true>(h16, d_params, d_map, n, st);
    else if (mode == kSrcPlanes) go_fwd_multi<kSrcPlanes, false>(h16, d_params, d_map, n, st);
    else if (mode == kSrcRgbU8 && narrow) go_fwd_multi<kSrcRgbU8, true>(h16, d_params, d_map, n, st);
    else if (mode == kSrcRgbU8) go_fwd_multi<kSrcRgbU8, false>(h16, d_params, d_map, n, st);
    else return cudaErrorInvalidValue;
    return cudaGetLastError();
}

template <int C, int OUT, bool NARROW>
static void go_inv_multi(bool h16, const InvLevelParams* ps, const int* map, int ctas, cudaStream_t st) {
    if (h16) k_dwt_inv_multi<C, OUT, true, NARROW><<<ctas, SW_THREADS, 0, st>>>(ps, map);
    else k_dwt_inv_multi<C, OUT, false, NARROW><<<ctas, SW_THREADS, 0, st>>>(ps, map);
}
cudaError_t launch_dwt_inv_multi(int channels, int out_mode, const InvLevelParams* d_params,
                                 const int* d_map, unsigned blocks, int form, bool narrow, cudaStream_t st) {
    if (blocks == 0) return cudaSuccess;
    if (form >= kDwtTiles) return launch_tiles_inv_multi(channels, out_mode, d_params, d_map, blocks, st);
    const int n = ctas_for((int)blocks, 1, inv_res(channels));
    const bool h16 = form == kDwtSweep16;
    if (out_mode == kOutRgb && channels == 3 && narrow) go_inv_multi<3, kOutRgb, true>(h16, d_params, d_map, n, st);
    else if (out_mode == kOutRgb && channels == 3) go_inv_multi<3, kOutRgb, false>(h16, d_params, d_map, n, st);
    else if (out_mode == kOutPlanes && narrow) go_inv_multi<1, kOutPlanes, true>(h16, d_params, d_map, n, st);
    else if (out_mode == kOutPlanes) go_inv_multi<1, kOutPlanes, false>(h16, d_params, d_map, n, st);
    else return cudaErrorInvalidValue;
    return cudaGetLastError();
}

// ---- one stream's level: by tiles (dwt_tiles.cu) or by sweeps.  A sweep's chain of
// steps (rows of a segment + 4) is longer than a tile's, so a level that does not
// fill the GPU several times over is a tile's; past the lines the sweeps' fewer
// instructions count, with frames of several sessions in flight above all.  Level
// alone, tiles / sweeps, us: forward from RGB24 1280x720 8.3 / 12.8, colour 17.0 /
// 21.8; 1920x1080 12.4 / 16.3, colour 27.1 / 33.4; 3840x2160 35.8 / 34.9, colour 77 /
// 92; 320x240 colour 13.6 / 10.8; planes of 640x360 5.0 / 7.0, 1920x1080 9.3 / 10.4,
// three of them 22.4 / 18.5.  Inverse 1280x720 6.2 / 6.6, 1920x1080 10.0 / 7.6, three
// planes of 960x540 7.8 / 8.7, of 1280x720 12.6 / 11.3; to RGB 1280x720 16.1 / 11.9,
// 1366x767 (rows that do not start at words) 14.5 / 16.9, 427x239 11.6 / 8.9.
// Three sessions side by side, us a frame, every level by sweeps / with these lines:
// 1366x767 48 / 41, colour 75 / 58, 1920x1080 63 / 59, colour 113 / 112, 2560x1440
// 98 / 94; on the far side of them 3840x2160 luma would go 198 -> 213 and colour
// 391 -> 407, 1920x1080 with its inverse by tiles 59 -> 60.  One session's frames in
// flight: 640x480 colour with FP16 planes 49 / 46, 1281x719 81 / 61, 853x479 colour
// 58 / 52.  (Float frames of one channel go over earlier: 1920x1080, one session,
// sweeps 110, tiles 118.)  A level at most two strips wide leaves half of a CTA's
// warps idle: 33x30000 colour 244 / 79.
static bool fwd_by_tiles(int mode, int channels, const FwdLevelParams& p) {
    const long long px = (long long)p.iw * p.ih;
    if (channels == 3 && mode != kSrcPlanes) return px >= 200000 && (px < 4000000 || dwt_narrow(p.sw));
    const long long line = channels == 3 ? 1000000 : mode == kSrcRgbU8 ? 5000000 : mode == kSrcPlanes ? 3000000 : 600000;
    return px < line || dwt_narrow(p.sw);
}
static bool inv_by_tiles(int channels, int out_mode, const InvLevelParams& p) {
    const long long px = (long long)p.ow * p.oh;
    if (out_mode == kOutRgb)
        return px >= 250000 && (dwt_narrow(p.sw) || ((p.ow & 3) && (p.out_f32 || px < 4000000)));
    return px < (channels == 1 ? 1200000 : 640000) || dwt_narrow(p.sw);
}

template <int MODE>
static void go_fwd(const FwdLevelParams& p, int units, cudaStream_t st) {
    const int n = ctas_for(units, 0, fwd_res(MODE, false), 1);
    if (p.h16) k_dwt_fwd<MODE, true><<<n, SW_THREADS, 0, st>>>(p, units);
    else k_dwt_fwd<MODE, false><<<n, SW_THREADS, 0, st>>>(p, units);
}
cudaError_t launch_dwt_fwd(int mode, int channels, const FwdLevelParams& p0, cudaStream_t st) {
    if (channels != 1 && channels != 3) return cudaErrorInvalidValue;
    if (fwd_by_tiles(mode, channels, p0)) return launch_tiles_fwd(mode, channels, p0, st);
    FwdLevelParams p = p0;
    unsigned gx, gy;
    const int units = (int)sweep_grid(p.unit, p.sw, p.sh, channels, 0, false, gx, gy);
    if (mode == kSrcPlanes) go_fwd<kSrcPlanes>(p, units, st);
    else if (mode == kSrcRgbU8) go_fwd<kSrcRgbU8>(p, units, st);
    else if (mode == kSrcRgbF32) go_fwd<kSrcRgbF32>(p, units, st);
    else return cudaErrorInvalidValue;
    return cudaGetLastError();
}

template <int C, int OUT>
static void go_inv(const InvLevelParams& p, int units, cudaStream_t st) {
    const int n = ctas_for(units, 1, inv_res(C));
    if (p.h16) k_dwt_inv<C, OUT, true><<<n, SW_THREADS, 0, st>>>(p, units);
    else k_dwt_inv<C, OUT, false><<<n, SW_THREADS, 0, st>>>(p, units);
}
cudaError_t launch_dwt_inv(int channels, int out_mode, const InvLevelParams& p0, cudaStream_t st) {
    if (inv_by_tiles(channels, out_mode, p0)) return launch_tiles_inv(channels, out_mode, p0, st);
    InvLevelParams p = p0;
    unsigned gx, gy;
    const int units = (int)sweep_grid(p.unit, p.sw, p.sh, out_mode == kOutPlanes ? channels : 1, 1, false, gx, gy);
    if (out_mode == kOutPlanes && (channels == 1 || channels == 3)) go_inv<1, kOutPlanes>(p, units, st);
    else if (out_mode == kOutRgb && channels == 3) go_inv<3, kOutRgb>(p, units, st);
    else return cudaErrorInvalidValue;
    return cudaGetLastError();
}

// Whether levels from one of sw x sh positions on run in a cluster: at most 6 rows
// of a strip per warp.  The cluster saves two launches of the host per direction and
// is the longer chain on the GPU (levels of 640x480 21 us, by tiles 14): the faster
// form where the host bounds the frames.  Three sessions side by side, us a frame, by
// tiles / in a cluster: luma 320x240 (1.2 rows) 38 / 30; colour 640x360 (2.8) 43.5 /
// 32, 640x480 (3.8) 43.5 / 32, 853x479 (5.0) 43.6 / 32; 1023x577 (7.6) 43 / 49.  One
// session's colour frames in flight, which the forward levels bound, pay for it: 640x480
// 42 / 47, 853x479 48 / 52.
constexpr int TAIL_ROWS = 6;
static bool tail_fits(int sw, int sh, int n) {
    const long long rows = (long long)((sw + SW_LANES * SQ - 1) / (SW_LANES * SQ)) * sh;
    return n >= 2 && n <= 3 && rows <= TAIL_ROWS * TAIL_CTAS * TAIL_WARPS;
}
cudaError_t launch_dwt_fwd_levels(int channels, const FwdLevelParams* p, int n, cudaStream_t st, int* launches) {
    if (n > 0 && tail_fits(p[0].sw, p[0].sh, n)) {
        LevelTail<FwdLevelParams> t{};
        for (int l = 0; l < n; l++) t.lv[l] = p[l];
        t.count = n;
        const dim3 grid(TAIL_CTAS, (unsigned)channels);
        if (p[0].h16) k_dwt_fwd_tail<true><<<grid, 32 * TAIL_WARPS, 0, st>>>(t);
        else k_dwt_fwd_tail<false><<<grid, 32 * TAIL_WARPS, 0, st>>>(t);
        *launches = 1;
        return cudaGetLastError();
    }
    *launches = n;
    cudaError_t e = cudaSuccess;
    for (int l = 0; l < n && e == cudaSuccess; l++) e = launch_dwt_fwd(kSrcPlanes, channels, p[l], st);
    return e;
}
cudaError_t launch_dwt_inv_levels(int channels, const InvLevelParams* p, int n, cudaStream_t st, int* launches) {
    if (n > 0 && tail_fits(p[n - 1].sw, p[n - 1].sh, n)) {
        LevelTail<InvLevelParams> t{};
        for (int l = 0; l < n; l++) t.lv[l] = p[l];
        t.count = n;
        const dim3 grid(TAIL_CTAS, (unsigned)channels);
        if (p[0].h16) k_dwt_inv_tail<true><<<grid, 32 * TAIL_WARPS, 0, st>>>(t);
        else k_dwt_inv_tail<false><<<grid, 32 * TAIL_WARPS, 0, st>>>(t);
        *launches = 1;
        return cudaGetLastError();
    }
    *launches = n;
    cudaError_t e = cudaSuccess;
    for (int l = 0; l < n && e == cudaSuccess; l++) e = launch_dwt_inv(channels, kOutPlanes, p[l], st);
    return e;
}

}  // namespace wema

namespace wema {

// ---- the autotuner's trial of the batched luma kernels' variants: the
// forward level-0 transform of a 3840 x 4320 RGB24 frame (two 2160-row frames'
// worth of tiles) and the inverse level-0 transform of its planes, each
// variant timed over five launches after one warm-up through the batched
// launch path (one task); the fastest of each is kept for the device.
cudaError_t dwt_autotune(int dev, float fwd_ms[9], float inv_ms[9], int* fwd_best, int* inv_best) {
    cudaError_t e = cudaSetDevice(dev);
    if (e != cudaSuccess) return e;
    const int W = 3840, H = 4320, SW = W / 2, SH = H / 2;   // level 0 of a 3840x4320 luma frame
    const size_t P = (size_t)W * H, N = (size_t)SW * SH;
    uint8_t* rgb = nullptr;
    float *coef = nullptr, *delta = nullptr, *ll = nullptr, *out = nullptr, *thr = nullptr;
    void *dp = nullptr, *dmap = nullptr, *state = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    cudaStream_t st = nullptr;
    const int keep_f = dwt_variant(dev, 0), keep_i = dwt_variant(dev, 1);
    auto done = [&](cudaError_t r) {
        for (void* p : {(void*)rgb, (void*)coef, (void*)delta, (void*)ll, (void*)out, (void*)thr, dp, dmap, state})
            if (p) cudaFree(p);
        if (e0) cudaEventDestroy(e0);
        if (e1) cudaEventDestroy(e1);
        if (st) cudaStreamDestroy(st);
        if (r != cudaSuccess) {                   // leave the device's choices as they were
            dwt_set_variant(dev, 0, keep_f);
            dwt_set_variant(dev, 1, keep_i);
        }
        return r;
    };
    if ((e = cudaMalloc(&rgb, 3 * P)) != cudaSuccess) return done(e);
    if ((e = cudaMalloc(&coef, 3 * N * sizeof(float))) != cudaSuccess) return done(e);
    if ((e = cudaMalloc(&delta, 3 * N * sizeof(float))) != cudaSuccess) return done(e);
    if ((e = cudaMalloc(&ll, N * sizeof(float))) != cudaSuccess) return done(e);
    if ((e = cudaMalloc(&out, P * sizeof(float))) != cudaSuccess) return done(e);
    if ((e = cudaMalloc(&thr, 8 * sizeof(float))) != cudaSuccess) return done(e);
    if ((e = cudaMalloc(&state, 3 * N * sizeof(float4))) != cudaSuccess) return done(e);
    if ((e = cudaMemset(state, 0, 3 * N * sizeof(float4))) != cudaSuccess) return done(e);
    if ((e = cudaMalloc(&dp, sizeof(FwdLevelParams) + sizeof(InvLevelParams))) != cudaSuccess) return done(e);
    if ((e = cudaMalloc(&dmap, 8 * sizeof(int))) != cudaSuccess) return done(e);
    if ((e = cudaMemset(rgb, 0x5a, 3 * P)) != cudaSuccess) return done(e);
    if ((e = cudaMemset(delta, 0, 3 * N * sizeof(float))) != cudaSuccess) return done(e);
    if ((e = cudaMemset(thr, 0, 8 * sizeof(float))) != cudaSuccess) return done(e);
    if ((e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking)) != cudaSuccess) return done(e);
    if ((e = cudaEventCreate(&e0)) != cudaSuccess || (e = cudaEventCreate(&e1)) != cudaSuccess) return done(e);
    if ((e = dwt_prepare_device()) != cudaSuccess) return done(e);
    FwdLevelParams fp{};
    fp.iw = W; fp.ih = H; fp.sw = SW; fp.sh = SH; fp.n = (long long)N;
    fp.vec_end = (long long)P;
    fp.src_u8 = rgb;
    fp.coef[0] = coef;
    fp.ll_out[0] = ll;
    // the steady batched forward runs the IIR step on each coefficient it
    // writes: time that kernel (a stable test biquad, poles at 0.9)
    fp.iir_state[0] = state;
    fp.iir_delta[0] = delta;
    const float bq[5] = {0.1f, 0.0f, -0.1f, -1.8f, 0.81f};
    for (int k = 0; k < 10; k++) fp.iir_c[k] = bq[k % 5];
    fp.iir_off6 = 0;
    fp.iir_simd_end = 6 * (long long)N;
    InvLevelParams ip{};
    ip.ow = W; ip.oh = H; ip.sw = SW; ip.sh = SH; ip.n = (long long)N;
    ip.ll[0] = ll;
    ip.coef[0] = coef;
    ip.delta[0] = delta;
    ip.thr = thr;
    ip.alpha[0] = 1.0f;
    ip.out_planes[0] = out;
    char* dpi = static_cast<char*>(dp) + sizeof(FwdLevelParams);
    int* map = static_cast<int*>(dmap);
    for (int inv = 0; inv < 2; inv++) {
        float* ms = inv ? inv_ms : fwd_ms;
        int best = 0;
        for (int v = 0; v < kDwtVariants; v++) {
            dwt_set_variant(dev, inv, v);
            unsigned gx, gy;
            const unsigned units = inv ? dwt_inv_grid(ip, 1, kDwtSweep, gx, gy) : dwt_fwd_grid(fp, 1, kDwtSweep, gx, gy);
            const int m[5] = {1, 0, (int)units, (int)gx, (int)gy};
            if ((e = cudaMemcpy(map, m, sizeof m, cudaMemcpyHostToDevice)) != cudaSuccess) return done(e);
            e = inv ? cudaMemcpy(dpi, &ip, sizeof ip, cudaMemcpyHostToDevice)
                    : cudaMemcpy(dp, &fp, sizeof fp, cudaMemcpyHostToDevice);
            if (e != cudaSuccess) return done(e);
            for (int rep = 0; rep < 6; rep++) {
                if (rep == 1 && (e = cudaEventRecord(e0, st)) != cudaSuccess) return done(e);
                e = inv ? launch_dwt_inv_multi(1, kOutPlanes, (const InvLevelParams*)dpi, map, units, kDwtSweep, false, st)
                        : launch_dwt_fwd_multi(kSrcRgbU8, 1, (const FwdLevelParams*)dp, map, units, kDwtSweep, false, st);
                if (e != cudaSuccess) return done(e);
            }
            if ((e = cudaEventRecord(e1, st)) != cudaSuccess) return done(e);
            if ((e = cudaEventSynchronize(e1)) != cudaSuccess) return done(e);
            float t = 0.f;
            if ((e = cudaEventElapsedTime(&t, e0, e1)) != cudaSuccess) return done(e);
            ms[v] = t / 5.f;
            if (ms[v] < ms[best]) best = v;
        }
        dwt_set_variant(dev, inv, best);
        (inv ? *inv_best : *fwd_best) = best;
    }
    return done(cudaSuccess);
}

}  // namespace wema
