// Refinement and final-selection kernels of the ASTC encoder (sm_100a).
//
//   k_refine       passes 13-17 (shaders/pass13..pass17), six iterations as
//                  driven by compression_pipeline.cpp:473-484: least-squares
//                  endpoints, colour endpoint packing (every LDR encoding the
//                  reference tries), unpacking, weight realignment, final
//                  error with a best-so-far snapshot.  One thread runs one
//                  candidate's iteration (in launches of one wave with the
//                  help of two or four lanes in passes 13-15); the 8
//                  candidates of a partitioned block share a CTA and its
//                  staged texels.
//   k_select_pack  pass18 plus the host argmin over candidates and partition
//                  counts (compression_pipeline.cpp:500-519), then the ASTC
//                  physical block layout (code/physical_compression.cpp:843)
//                  written straight to the 16-byte output block.
#include <cuda_fp16.h>

#include <algorithm>
#include <mutex>
#include <type_traits>

#include "decode_fast.cuh"
#include "device_math.cuh"
#include "kernels.h"

namespace astcb200 {

using namespace dev;

namespace {

constexpr float ERR_DEFAULT = 1e37f;
__constant__ int c_levels_r[21] = {2, 3, 4, 5, 6, 8, 10, 12, 16, 20, 24, 32, 40, 48, 64, 80, 96, 128, 160, 192, 256};

enum {
    FMT_LUMINANCE = 0, FMT_LUMINANCE_DELTA = 1, FMT_LUMINANCE_ALPHA = 4, FMT_LUMINANCE_ALPHA_DELTA = 5,
    FMT_RGB_SCALE = 6, FMT_RGB = 8, FMT_RGB_DELTA = 9, FMT_RGB_SCALE_ALPHA = 10, FMT_RGBA = 12, FMT_RGBA_DELTA = 13
};

struct I4 { int32_t x, y, z, w; };
__device__ __forceinline__ int32_t ic(const I4& v, int c) { return c == 0 ? v.x : c == 1 ? v.y : c == 2 ? v.z : v.w; }
__device__ __forceinline__ int32_t shl1(int32_t v) { return (int32_t)((uint32_t)v << 1); }

// x / 257 for an endpoint clamped to [0, 65535], rounded to nearest: the product with the
// reciprocal split in two (Brisebarre, Muller and Raina, "Accelerating correctly rounded
// floating-point division when the divisor is known in advance", 2004), equal to the division
// for every float of the range at or above 1e-33 (checked exhaustively).
__device__ __forceinline__ float over257(float color) {
    const float x = fminf(fmaxf(color, 0.0f), 65535.0f);
    float r = __fmaf_rn(x, 0x1.fe01fep-9f, x * 0x1.fe01fep-41f);
    if (x > 0.0f && x < 1e-30f) r = x / 257.0f;
    return r;
}
__device__ __forceinline__ float4 over257(float4 c) { return make_float4(over257(c.x), over257(c.y), over257(c.z), over257(c.w)); }

// ------------------------------------------------------------ pass14 colour endpoint packing
// The endpoints it packs are clamped to 0..255, so every value converted to an integer here is
// finite and small.  The refinement kernels stalled on instruction fetch first (4.7 of 13 warps
// per issue), so this code and the iteration are written for size: one
// copy of each encoding's body and of the final error, loops left rolled.
// Measured with f2i / f2u as one conversion: full search of 1024x1024 at 4x4 47.5 -> 39.3 ms, of
// 1021x765 at 10x8 72.5 -> 69.6 ms; proposal search of 2048x2048 at 4x4 10.2 -> 8.8 ms.
__device__ __forceinline__ int32_t rni(float v) { return __float2int_rn(v); }
struct Packer {
    const uint8_t* t;  // quantise-unquantise row of the quant level (cu2u, [512])
    __device__ __forceinline__ int32_t tab(int32_t idx) const { return t[idx]; }
    __device__ __forceinline__ int32_t qf1(int32_t v, float vf) const { return tab(v * 2 + ((vf - (float)v) >= -0.1f ? 1 : 0)); }
    __device__ __forceinline__ int32_t qint(int32_t v) const { return tab(v * 2 + 1); }
    __device__ __forceinline__ int32_t qrn(float v) const { return qf1(rni(v), v); }
    __device__ static float enc_err(float4 u0, float4 u1, I4 q0, I4 q1) {
        const float4 e0 = u0 - make_float4((float)q0.x, (float)q0.y, (float)q0.z, (float)q0.w);
        const float4 e1 = u1 - make_float4((float)q1.x, (float)q1.y, (float)q1.z, (float)q1.w);
        const float4 e = e0 * e0 + e1 * e1;
        return ((e.x + e.y) + e.z) + e.w;
    }

    // bit_transfer_signed(&a, &b) (pass14:355-369)
    __device__ static void bts1(int32_t& a, int32_t& b) {
        const uint32_t a0 = (uint32_t)a, b0 = (uint32_t)b;
        int32_t na = (int32_t)((a0 >> 1) & 0x3F);
        if (na & 0x20) na -= 0x40;
        b = (int32_t)((b0 >> 1) | (a0 & 0x80));
        a = na;
    }
    __device__ static void bts(I4& a, I4& b) { bts1(a.x, b.x); bts1(a.y, b.y); bts1(a.z, b.z); bts1(a.w, b.w); }
    __device__ static I4 uncontract(I4 v) { return {(v.x + v.z) >> 1, (v.y + v.z) >> 1, v.z, v.w}; }
    __device__ static int32_t clamp255(int32_t v) { return min(max(v, 0), 255); }
    __device__ static void delta_unpack(I4 i0, I4 i1, I4& o0, I4& o1) {
        bts(i1, i0);
        const int32_t s = i1.x + i1.y + i1.z;
        i1 = {i1.x + i0.x, i1.y + i0.y, i1.z + i0.z, i1.w + i0.w};
        if (s < 0) { I4 t = uncontract(i0); i0 = uncontract(i1); i1 = t; }
        o0 = {clamp255(i0.x), clamp255(i0.y), clamp255(i0.z), clamp255(i0.w)};
        o1 = {clamp255(i1.x), clamp255(i1.y), clamp255(i1.z), clamp255(i1.w)};
    }
    __device__ static void rgba_unpack(I4 i0, I4 i1, I4& o0, I4& o1) {
        if ((i0.x + i0.y + i0.z) > (i1.x + i1.y + i1.z)) { I4 t = uncontract(i0); i0 = uncontract(i1); i1 = t; }
        o0 = i0; o1 = i1;
    }
    __device__ static bool out_of_range(float4 c) {
        return c.x < 0.0f || c.x > 255.0f || c.y < 0.0f || c.y > 255.0f || c.z < 0.0f || c.z > 255.0f || c.w < 0.0f || c.w > 255.0f;
    }
    __device__ static float4 inv_bc(float4 c) { return make_float4((c.x + c.x) - c.z, (c.y + c.y) - c.z, (c.z + c.z) - c.z, (c.w + c.w) - c.w); }

    // One channel of a delta encoding: the low endpoint v0 and the difference to the high one
    // v1 (8-bit units), quantised to q0 and q1; false when the difference does not fit.
    __device__ __forceinline__ bool delta1(float v0, float v1, int32_t& q0, int32_t& q1, int32_t& base9) const {
        const int32_t a = shl1(rni(v0));
        q0 = qint(a & 0xFF);
        base9 = q0 | (a & 0x100);
        const int32_t d = shl1(rni(v1)) - base9;
        const bool fits = d <= 63 && d >= -64;
        const int32_t d8 = (d & 0x7F) | ((base9 & 0x100) >> 1);
        q1 = qint(d8);
        return fits && ((d8 ^ q1) & 0xC0) == 0;
    }
    // try_quantize_rgb_delta(_blue_contract) body after the optional inverse contraction (w is
    // left to the alpha)
    __device__ __forceinline__ bool rgb_delta(float4 c0, float4 c1, I4& o0, I4& o1, bool want_bc) const {
        int32_t b9;
        bool ok = delta1(c0.x, c1.x, o0.x, o1.x, b9);
        ok = delta1(c0.y, c1.y, o0.y, o1.y, b9) && ok;
        ok = delta1(c0.z, c1.z, o0.z, o1.z, b9) && ok;
        I4 e0 = {o0.x, o0.y, o0.z, 0}, e1 = {o1.x, o1.y, o1.z, 0};
        bts(e1, e0);
        const int32_t s = e1.x + e1.y + e1.z;
        ok = ok && (want_bc ? (s < 0) : (s >= 0));
        e0 = {e0.x + e1.x, e0.y + e1.y, e0.z + e1.z, 0};
        return ok && (uint32_t)e0.x <= 0xFFu && (uint32_t)e0.y <= 0xFFu && (uint32_t)e0.z <= 0xFFu;
    }
    __device__ __forceinline__ bool alpha_delta(float v0, float v1, int32_t& q0, int32_t& q1) const {
        int32_t b9;
        if (!delta1(v0, v1, q0, q1, b9)) return false;
        int32_t du = q1 & 0x7F;
        if (du & 0x40) du -= 0x80;
        du += b9;
        return du >= 0 && du <= 0x1FF;
    }
    __device__ __forceinline__ I4 q3flt(float4 c) const { return {qrn(c.x), qrn(c.y), qrn(c.z), 0}; }
    // Quantised channel sums of the endpoints at one step of the loop below: true when the
    // step ends it (the low endpoint's sum no longer above the high one's).
    __device__ __forceinline__ bool qrgb_probe(float x0, float y0, float z0, float x1, float y1, float z1, I4& c0i, I4& c1i) const {
        c0i = {qf1(max(rni(x0), 0), x0), qf1(max(rni(y0), 0), y0), qf1(max(rni(z0), 0), z0), 0};
        c1i = {qf1(min(rni(x1), 255), x1), qf1(min(rni(y1), 255), y1), qf1(min(rni(z1), 255), z1), 0};
        return (c0i.x + c0i.y + c0i.z) <= (c1i.x + c1i.y + c1i.z);
    }
    // The reference's loop nudges the endpoints 0.2 apart per step (at most 4096 steps) and
    // stops at the first step whose quantised channel sums no longer cross.  A rounded
    // channel and its half-step bit move monotonically with its endpoint and the table is
    // monotonic, so the low sum never rises and the high one never falls from step to step:
    // the stopping test is monotonic in the step.  The stop is found by probing steps 0, 1,
    // 3, 7, ... and bisecting the last bracket; the endpoints are always brought to a probed
    // step by the loop's own float subtractions and additions from an earlier probed step,
    // so each probe sees the values the loop would.
    __device__ __forceinline__ void quant_rgb(float4 c0, float4 c1, I4& o0, I4& o1) const {
        float x0 = c0.x, y0 = c0.y, z0 = c0.z, x1 = c1.x, y1 = c1.y, z1 = c1.z;  // at step lo
        int lo = 0, hi = 0, at = 0, step = 1;  // at: the step to probe
        bool bracketed = false;                // the stop is in (lo, hi] (hi = 4095: the last step)
        for (;;) {
            float a = x0, b = y0, c = z0, d = x1, e = y1, f = z1;
#pragma unroll 1
            for (int i = lo; i < at; i++) { a = a - 0.2f; b = b - 0.2f; c = c - 0.2f; d = d + 0.2f; e = e + 0.2f; f = f + 0.2f; }
            const bool stop = qrgb_probe(a, b, c, d, e, f, o0, o1);
            if (bracketed ? at == hi : (stop && at <= 1)) return;
            if (stop || at == 4095) {
                hi = at;
                bracketed = true;
            } else {
                x0 = a; y0 = b; z0 = c; x1 = d; y1 = e; z1 = f;
                lo = at;
            }
            if (bracketed) {
                at = hi - lo > 1 ? lo + (hi - lo) / 2 : hi;
            } else {
                at = min(lo + step, 4095);
                step *= 2;
            }
        }
    }
    __device__ __forceinline__ void quant_rgbs(float4 color, uint32_t* out) const {
        const float scale = 1.0f / 257.0f;
        const float r = clampf(color.x * scale, 0.0f, 255.0f), g = clampf(color.y * scale, 0.0f, 255.0f), b = clampf(color.z * scale, 0.0f, 255.0f);
        const uint32_t ri = (uint32_t)qrn(r), gi = (uint32_t)qrn(g), bi = (uint32_t)qrn(b);
        const float oldsum = ((color.x + color.y) + color.z) * scale;
        const float newsum = (float)(ri + gi + bi);
        const float sa = clampf((color.w * (oldsum + 1e-10f)) / (newsum + 1e-10f), 0.0f, 1.0f);
        const int32_t si = min(max(rni(sa * 256.0f), 0), 255);
        out[0] = ri; out[1] = gi; out[2] = bi; out[3] = (uint32_t)qint(si);
    }
    // pack_color_endpoints_helper (pass14:917-1224) at quant level q.  Returns the format (x)
    // and the up to eight packed values, one byte each (y, then z).
    __device__ static __noinline__ uint4 pack(const uint8_t* cu2u, float4 color0, float4 color1, float4 rgbs, uint32_t fmt, uint32_t q) {
        const Packer k{cu2u + (q - 4) * 512};
        const float4 c0 = over257(color0), c1 = over257(color1);
        uint32_t out[8];
#pragma unroll
        for (int i = 0; i < 8; i++) out[i] = 0;
        uint32_t bf = FMT_LUMINANCE;
        if (fmt == FMT_RGB || fmt == FMT_RGBA) {
            const bool rgba = fmt == FMT_RGBA;
            float best = ERR_DEFAULT;
            I4 o0 = {0, 0, 0, 0}, o1 = {0, 0, 0, 0};
            // the four encodings in the order the reference tries them: delta with blue
            // contraction, delta, blue contraction, plain; the first of the smallest error wins
#pragma unroll 1
            for (int v = q <= 18 ? 0 : q < 20 ? 2 : 3; v < 4; v++) {
                const bool contract = v == 0 || v == 2;
                float4 a0 = c0, a1 = c1;
                if (contract) {
                    a0 = inv_bc(c1); a1 = inv_bc(c0);
                    if (out_of_range(a0) || out_of_range(a1)) continue;
                }
                I4 p0, p1, u0, u1;
                p0.w = p1.w = 0;
                if (v < 2) {
                    if (!k.rgb_delta(a0, a1, p0, p1, contract)) continue;
                    if (rgba && !k.alpha_delta(contract ? c1.w : c0.w, contract ? c0.w : c1.w, p0.w, p1.w)) continue;
                    delta_unpack(p0, p1, u0, u1);
                } else {
                    if (contract) {
                        p0 = k.q3flt(a0); p1 = k.q3flt(a1);
                        if ((p0.x + p0.y + p0.z) <= (p1.x + p1.y + p1.z)) continue;
                    } else {
                        k.quant_rgb(c0, c1, p0, p1);
                    }
                    if (rgba) { p0.w = k.qrn(contract ? c1.w : c0.w); p1.w = k.qrn(contract ? c0.w : c1.w); }
                    rgba_unpack(p0, p1, u0, u1);
                }
                const float e = enc_err(c0, c1, u0, u1);
                if (e < best) { best = e; bf = v < 2 ? fmt + 1 : fmt; o0 = p0; o1 = p1; }
            }
            out[0] = (uint32_t)o0.x; out[1] = (uint32_t)o1.x; out[2] = (uint32_t)o0.y;
            out[3] = (uint32_t)o1.y; out[4] = (uint32_t)o0.z; out[5] = (uint32_t)o1.z;
            if (rgba) { out[6] = (uint32_t)o0.w; out[7] = (uint32_t)o1.w; }
        } else if (fmt == FMT_RGB_SCALE || fmt == FMT_RGB_SCALE_ALPHA) {
            if (fmt == FMT_RGB_SCALE_ALPHA) { out[4] = (uint32_t)k.qrn(c0.w); out[5] = (uint32_t)k.qrn(c1.w); }
            k.quant_rgbs(rgbs, out);
            bf = fmt;
        } else {  // FMT_LUMINANCE_ALPHA, FMT_LUMINANCE and any other format
            const bool la = fmt == FMT_LUMINANCE_ALPHA;
            float l0 = ((c0.x + c0.y) + c0.z) / 3.0f, l1 = ((c1.x + c1.y) + c1.z) / 3.0f;
            int32_t q0, q1, a0, a1;
            if (la && q <= 18 && k.alpha_delta(l0, l1, q0, q1) && k.alpha_delta(c0.w, c1.w, a0, a1)) {
                bf = FMT_LUMINANCE_ALPHA_DELTA;
            } else {
                if (!la && l0 > l1) { const float av = (l0 + l1) * 0.5f; l0 = av; l1 = av; }
                q0 = k.qrn(l0); q1 = k.qrn(l1);
                a0 = la ? k.qrn(c0.w) : 0; a1 = la ? k.qrn(c1.w) : 0;
                bf = la ? FMT_LUMINANCE_ALPHA : FMT_LUMINANCE;
            }
            out[0] = (uint32_t)q0; out[1] = (uint32_t)q1; out[2] = (uint32_t)a0; out[3] = (uint32_t)a1;
        }
        return make_uint4(bf, out[0] | out[1] << 8 | out[2] << 16 | out[3] << 24, out[4] | out[5] << 8 | out[6] << 16 | out[7] << 24, 0u);
    }
};

// pass15: decode the packed endpoints (bytes of lo, then hi) of one partition to 0..255.
__device__ __forceinline__ void unpack_endpoints(uint32_t fmt, uint32_t lo, uint32_t hi, I4& o0, I4& o1) {
    auto I = [&](int k) { return (int32_t)(((k < 4 ? lo : hi) >> (8 * (k & 3))) & 0xFF); };
    switch (fmt) {
        case FMT_LUMINANCE_DELTA: {
            const int32_t l0 = (I(0) >> 2) | (I(1) & 0xC0), l1 = min(l0 + (I(1) & 0x3F), 255);
            o0 = {l0, l0, l0, 255}; o1 = {l1, l1, l1, 255}; break;
        }
        case FMT_LUMINANCE_ALPHA: o0 = {I(0), I(0), I(0), I(2)}; o1 = {I(1), I(1), I(1), I(3)}; break;
        case FMT_LUMINANCE_ALPHA_DELTA: {
            int32_t l0 = I(0), l1 = I(1), a0 = I(2), a1 = I(3);
            l0 |= (l1 & 0x80) << 1; a0 |= (a1 & 0x80) << 1;
            l1 &= 0x7F; a1 &= 0x7F;
            if (l1 & 0x40) l1 -= 0x80;
            if (a1 & 0x40) a1 -= 0x80;
            l0 >>= 1; l1 >>= 1; a0 >>= 1; a1 >>= 1;
            l1 = min(max(l0 + l1, 0), 255); a1 = min(max(a0 + a1, 0), 255);
            o0 = {l0, l0, l0, a0}; o1 = {l1, l1, l1, a1}; break;
        }
        case FMT_RGB_SCALE: {
            const int32_t s = I(3);
            o1 = {I(0), I(1), I(2), 255};
            o0 = {(I(0) * s) >> 8, (I(1) * s) >> 8, (I(2) * s) >> 8, 255}; break;
        }
        case FMT_RGB_SCALE_ALPHA: {
            const int32_t s = I(3);
            o1 = {I(0), I(1), I(2), I(5)};
            o0 = {(I(0) * s) >> 8, (I(1) * s) >> 8, (I(2) * s) >> 8, I(4)}; break;
        }
        case FMT_RGB: Packer::rgba_unpack({I(0), I(2), I(4), 0}, {I(1), I(3), I(5), 0}, o0, o1); o0.w = 255; o1.w = 255; break;
        case FMT_RGB_DELTA: Packer::delta_unpack({I(0), I(2), I(4), 0}, {I(1), I(3), I(5), 0}, o0, o1); o0.w = 255; o1.w = 255; break;
        case FMT_RGBA: Packer::rgba_unpack({I(0), I(2), I(4), I(6)}, {I(1), I(3), I(5), I(7)}, o0, o1); break;
        case FMT_RGBA_DELTA: Packer::delta_unpack({I(0), I(2), I(4), I(6)}, {I(1), I(3), I(5), I(7)}, o0, o1); break;
        default: o0 = {I(0), I(0), I(0), 255}; o1 = {I(1), I(1), I(1), 255}; break;
    }
}

// ------------------------------------------------------------ k_refine
constexpr int kRefineThreads = 128;
constexpr int kRefineCtas = 5;
constexpr int kOneWaveGroups = 148 * kRefineCtas;

// Candidate threads per partitioned block (the refinement top-N rounded up to a power of
// two) and partitioned blocks per CTA: 16 x 8 for the full search; more, narrower ones when
// the proposal search keeps fewer candidates, capped so the staged texels stay <= 40 KB.
__host__ __device__ inline int refine_cpb(int topn) { return topn <= 1 ? 1 : topn <= 2 ? 2 : topn <= 4 ? 4 : 8; }
__host__ __device__ inline int refine_pbs(int T, int topn) {
    const int by_threads = kRefineThreads / refine_cpb(topn);
    const int by_smem = 40960 / (T * (T > 16 ? 4 : 16));
    return by_threads < by_smem ? by_threads : (by_smem > 16 ? by_smem : 16);
}

// Candidates a warp runs at a time in a launch of npb partitioned blocks.  A launch of one wave is as long as
// its slowest warp, and a warp of 32 different candidates runs the union of their paths and
// the longest of their loops: with 8 or 16 a warp it is shorter, while the waves still hold every
// group, and a candidate's 4 or 2 lanes (8 or 16 apart) share its partitions in passes 13 to 15,
// of which packing is most of an iteration.  Measured (B200), k_refine of a full search of 64x64 at 4x4 (3,328
// partitioned blocks) 519 us with 32, 494 with 16, 394 to 421 with 16 and their second lanes; both
// launches of the proposal search of 200x120 at 4x4 454 us with 8, 365 with 8 and their other lanes.
// With twice the limits: full search of 256 blocks at 4x4 0.42 -> 0.53 ms, of 1,400 1.12 -> 1.21.
__host__ __device__ inline int refine_spread(int npb) {
    return npb <= kOneWaveGroups * 4 ? 8 : npb <= kOneWaveGroups * 8 ? 16 : 32;
}
// Live candidates at or below which a CTA hands them to the tail (T > 16: u8).  At 4x4, where the sorted
// warps of a full group are the denser ones, late: proposal search of 900x700 1.90 ms at 64, 2.05 at
// 96; full search of 436x292 4.14 ms at 32, 4.23 at 64.  Above 16 texels the proposal pass hands over
// most after the first iteration, which the tail's refilled slots run as densely without holding
// the groups that wait: 3000x2000 at 6x6 8.54 ms at 64, 7.92 at 96; 1024x1024 mip chain 6.68, 5.83.
// So does a full search of few waves, whose last one is partly empty, with room in the tail for every
// candidate: at 6x6 228x156 (1.1 waves) 2.06 ms at 32, 1.81 at 128; 300x180 (1.6) 2.69 and 2.43; 420x240
// (3.1) 4.17 and 4.01; 540x300 (4.9) 6.23 and 6.15; 600x360 (6.6) 7.97 and 7.97; 660x480 (9.7) 11.27 and
// 11.41.  (With room for 16 a block, which most CTAs find full, 2.09, 2.74, 4.34 and 6.48 for the first four.)
__host__ __device__ inline bool refine_few_waves(bool u8, int ngroups) { return u8 && ngroups <= 5 * kOneWaveGroups; }
__device__ inline int refine_spill_live(bool u8, bool prop, int ngroups) {
    if (!u8) return prop ? 64 : 32;
    return prop ? 96 : refine_few_waves(u8, ngroups) ? kRefineThreads : 32;
}
__host__ __device__ inline int refine_group(int T, int cpb, int spread) {  // partitioned blocks per CTA
    const int pbs = refine_pbs(T, cpb), n = kRefineThreads / 32 * spread / cpb;
    return n < 1 ? 1 : n < pbs ? n : pbs;
}
__host__ __device__ inline int refine_groups(int npb, int pbs) { return (npb + pbs - 1) / pbs; }
__host__ __device__ inline bool refine_one_wave(int ngroups) { return ngroups <= kOneWaveGroups; }

// Candidate state in shared memory, one slot per candidate a CTA runs, arrays of [row][slot]:
// lanes on consecutive slots hit consecutive banks whatever rows they read.  A slot is the
// candidate's rank in its group's initial order, so the first iteration's lanes are on
// consecutive slots and the gathered ones of later iterations on increasing ones.
//   ep   [8]      least-squares endpoints (float4): ep0 and ep1 of partition q in rows 2q, 2q + 1
//   u    [4]      unpacked endpoints of partition q, eight bytes: ep0 xyzw, ep1 xyzw (used times 257)
//   s    [T]      infilled weight of each texel times 16, 0..1024, exact in half precision
//   qw   [max_w]  grid weights 0..64
// The best error so far is in the candidate's snapshot.
// 328 bytes a candidate at 80 texels, with its share of the staged ones 447, so that four CTAs fit on an
// SM instead of three: k_refine of 1021x765 at 10x8 15.3 -> 13.2 ms.  (Six CTAs of 80 registers
// instead of five at 4x4: 10.2 and 10.3 ms for 1024x1024.)
// The infilled weights are kept as sums of grid weight x (contribution x 16), small integers
// that pass16 updates when it moves a weight; every use of one (pass13's weight s / 1024,
// pass16's s / 16, pass17's rounded s / 16) is the exact value the passes' own sums of
// products give, since those sums are exact too.  Before, each texel's four table entries
// and weights were read again at every use (two to three uses per
// texel and iteration in pass13 and pass17 and one per texel of each weight in pass16).
// Measured with pass13's walk in partition order (B200): full search of 1024x1024 at 4x4 50.2 -> 47.5 ms,
// of 64x64 1.08 -> 0.90 ms; proposal search of 2047x2050 at 6x6 8.98 -> 8.13 ms.
constexpr int kSlotRow16 = kRefineThreads * 16;  // bytes of a row of 16-byte elements
constexpr int kSlotRow8 = kRefineThreads * 8;    // of 8-byte elements
constexpr int kSlotRow4 = kRefineThreads * 4;    // of two s or four qw
struct RefineLayout {
    int ep, u, s, qw, pos, map, px, part, staged, total;  // both kernels
    int item, next_it;                                    // k_refine_tail
    int keys;                                             // k_refine: over u, which only an iteration holds
};
// Texel rows of the staged partitioned blocks, an odd number of banks (or 16-byte bank groups)
// apart: a warp's candidates, sorted by path, belong to different partitioned blocks.
__host__ __device__ inline int px_row_bytes(int T, bool u8) { return u8 ? (T | 1) * 4 : (T + 1) * 16; }
__host__ __device__ inline int part_row_bytes(int T, int width) { return ((T * width + 3) / 4 | 1) * 4; }
// rows: staged partitioned blocks (the tail stages one per slot, with partition bytes).
__host__ __device__ inline RefineLayout refine_layout(int T, int max_w, int rows, bool u8, bool tail) {
    RefineLayout f;
    int o = 0;
    auto take = [&](int bytes) { const int r = o; o += (bytes + 15) & ~15; return r; };
    f.ep = take(8 * kSlotRow16);
    f.keys = f.u = take(4 * kSlotRow8);
    f.s = take((T + 1) / 2 * kSlotRow4);
    f.qw = take((max_w + 3) / 4 * kSlotRow4);
    f.pos = take(kRefineThreads);
    f.map = take(kRefineThreads);
    f.px = take(rows * px_row_bytes(T, u8));
    f.part = take(rows * part_row_bytes(T, u8 && !tail ? 2 : 1));
    f.staged = take(tail ? 0 : rows * 4);
    f.item = take(tail ? kRefineThreads * 4 : 0);
    f.next_it = take(tail ? kRefineThreads : 0);
    f.total = o;
    return f;
}
struct Cand {  // one slot of the arrays above
    uint8_t *epb, *ub, *sb, *qb;
    __device__ Cand(uint8_t* sm, const RefineLayout& f, int slot)
        : epb(sm + f.ep + slot * 16), ub(sm + f.u + slot * 8), sb(sm + f.s + slot * 4), qb(sm + f.qw + slot * 4) {}
    __device__ __forceinline__ float4& ep(int i) const { return *reinterpret_cast<float4*>(epb + i * kSlotRow16); }
    __device__ __forceinline__ uint2& u(int q) const { return *reinterpret_cast<uint2*>(ub + q * kSlotRow8); }
    __device__ __forceinline__ __half& s(int t) const { return *reinterpret_cast<__half*>(sb + (t >> 1) * kSlotRow4 + (t & 1) * 2); }
    __device__ __forceinline__ uint8_t& qw(int w) const { return qb[(w >> 2) * kSlotRow4 + (w & 3)]; }
    __device__ __forceinline__ uint32_t& qw4(int i) const { return *reinterpret_cast<uint32_t*>(qb + i * kSlotRow4); }
};
// The four bytes of v times 257, as floats: 2^23 + n has n as its low bits, and a byte times 257 is the
// byte twice.
__device__ __forceinline__ float4 x257(uint32_t v) {
    return make_float4(__uint_as_float(__byte_perm(v, 0x4B000000u, 0x7600)) - 8388608.0f, __uint_as_float(__byte_perm(v, 0x4B000000u, 0x7611)) - 8388608.0f,
                       __uint_as_float(__byte_perm(v, 0x4B000000u, 0x7622)) - 8388608.0f, __uint_as_float(__byte_perm(v, 0x4B000000u, 0x7633)) - 8388608.0f);
}
// Round to the nearest integer, ties to even, for 0 <= v < 2^22 (rintf on the FP32 adders).
__device__ __forceinline__ float rn_small(float v) { return (v + 8388608.0f) - 8388608.0f; }

struct RTabs {
    const uint8_t* b;
    const TableLayout* L;
    __device__ const DevDm& dm(int m) const { return reinterpret_cast<const DevDm*>(b + L->off_dm)[m]; }
    __device__ const DevBm& bm(int i) const { return reinterpret_cast<const DevBm*>(b + L->off_bm)[i]; }
    __device__ int wt_count(int m, int w) const { return b[L->off_wt_count + m * 64 + w]; }
    __device__ int wt_start(int m, int w) const { return reinterpret_cast<const uint16_t*>(b + L->off_wt_start)[m * 64 + w]; }
    __device__ uint32_t w2t(int i) const { return reinterpret_cast<const uint16_t*>(b + L->off_w2t)[i]; }
    __device__ uint64_t tw4(int m, int t) const { return reinterpret_cast<const uint64_t*>(b + L->off_tw4)[m * L->T + t]; }
    __device__ int part_count(int P, int e, int q) const { return b[L->off_part_counts + ((P - 2) * 1024 + e) * 4 + q]; }
    __device__ uint32_t prev_next(int q, int v) const { return reinterpret_cast<const uint16_t*>(b + L->off_prev_next)[q * 65 + v]; }
};

// Sets the candidate's infilled weights from its grid weights (pass13:165-184, pass17:127-146).
// Padding entries of the dense list contribute 0.
__device__ __forceinline__ void infill(const RTabs& tb, const Cand& c, int dm, int T, bool direct) {
#pragma unroll 1
    for (int t = 0; t < T; t++) {
        uint32_t v;
        if (direct) {
            v = (uint32_t)c.qw(t) * 16u;
        } else {
            const uint64_t e4 = tb.tw4(dm, t);
            v = 0;
#pragma unroll
            for (int j = 0; j < 4; j++) { const uint32_t e = (uint32_t)(e4 >> (16 * j)) & 0xFFFF; v += (e >> 8) * (uint32_t)c.qw(e & 0xFF); }
        }
        c.s(t) = __ushort2half_rn((unsigned short)v);
    }
}

// A partitioned block's staged texels.  Up to 16 texels they are floats; larger blocks
// stage RGBA8 (4 bytes a texel, so more CTAs fit on an SM), converted where read.
__host__ __device__ inline bool refine_u8(int T) { return T > 16; }
template <bool U8> struct TexelRow;
template <> struct TexelRow<true> {
    const uchar4* c;
    __device__ __forceinline__ float4 operator[](int t) const { return texel_float(c[t]); }
};
template <> struct TexelRow<false> {
    const float4* c;
    __device__ __forceinline__ float4 operator[](int t) const { return c[t]; }
};
// Its partitioning: entry i holds texel i's partition and, in the low bits, the i-th texel in
// (partition, texel) order, which pass13 walks one partition after another.
template <class E> struct PartRow {
    static constexpr int kShift = sizeof(E) == 1 ? 6 : 8;  // bytes for blocks of up to 64 texels
    E* v;
    __device__ __forceinline__ int part(int t) const { return v[t] >> kShift; }
    __device__ __forceinline__ int order(int i) const { return v[i] & ((1 << kShift) - 1); }
    // prow: the partitioning's row of texel partitions (null: one partition); one thread
    __device__ __forceinline__ void set(const uint32_t* prow, const uint8_t* counts, int T) const {
        uint32_t next = 0;  // next position of each partition, a byte each
        if (prow) next = (uint32_t)counts[0] << 8 | ((uint32_t)counts[0] + counts[1]) << 16 | ((uint32_t)counts[0] + counts[1] + counts[2]) << 24;
#pragma unroll 1
        for (int t = 0; t < T; t++) v[t] = prow ? (E)(((prow[t >> 4] >> (2 * (t & 15))) & 3u) << kShift) : (E)0;
#pragma unroll 1
        for (int t = 0; t < T; t++) {
            const int sh = 8 * part(t);
            const int i = (next >> sh) & 0xFF;
            v[i] = (E)(v[i] | t);
            next += 1u << sh;
        }
    }
};
// Row of a partitioning's texel partitions, two bits a texel.
__device__ __forceinline__ const uint32_t* part2_row(const KernelArgs& a, int P, int entry) {
    return reinterpret_cast<const uint32_t*>(a.tables + a.L.off_part2) + ((size_t)(P - 2) * 1024 + entry) * ((a.L.T + 15) >> 4);
}
// Direction of the partition's average colour (pass13's scale direction), the same for every
// candidate and iteration of a partitioned block.
__device__ __forceinline__ float4 scale_dir(float4 avg, float ps) {
    const float4 cw = chan_w();
    const float4 rsum = (avg * ps) * cw;
    const float4 rws = vmax(cw * ps, mk(1e-17f));
    float4 sv = rsum / rws; sv.w = 0.0f;
    return normalize4(sv);
}

// One refinement iteration (passes 13-17) of candidate k of a partitioned block, its
// state in cs; iteration 0 first loads the front's initial state.  Returns whether pass16
// moved a weight: a pass16 that moved none leaves a fixed point, where the next iteration's
// pass13 recomputes the same endpoints from the same weights (channels whose system is
// degenerate keep the previous values, which are these), so packing, unpacking, realignment
// and the final error repeat exactly and can never lower the error: stopping there gives
// the result of running the remaining iterations.
// HELP: `lanes` candidates a warp (refine_spread), each run by the 32 / lanes lanes that hold its
// slot, which must enter together; the first has the result.
template <bool HELP, class Row, class Part>
__device__ bool refine_step(const KernelArgs& a, const PBRec& rec, const int P, int k, const Row px, const Part pt,
                            const Cand cs, Snap* snap, const int it, const int lanes) {
    const RTabs tb{a.tables, &a.L};
    const int T = a.L.T;
    const CandInit& ci = rec.c[k];
    const DevBm bm = tb.bm(ci.bm);
    const DevDm dmi = tb.dm(bm.dm);
    const int W = dmi.W;
    const bool direct = W == T;
    const float4 cw = chan_w();
    const float lsw = (cw.x + cw.y) + cw.z;
    const uint8_t* cu2u = a.tables + a.L.off_cu2u;
    float4 rgbs[4];
    uint2 packed[4], packed_mod[4];
    // this lane's partitions: every qstep-th from q0
    const int spread = HELP ? lanes : 32, q0 = HELP ? (threadIdx.x & 31) / spread : 0, qstep = 32 / spread, first = threadIdx.x & (spread - 1);
    const unsigned group = (spread == 32 ? 1u : spread == 16 ? 0x10001u : 0x1010101u) << first;
    if (it == 0 && q0 == 0) {
#pragma unroll
        for (int q = 0; q < 4; q++) { cs.ep(2 * q) = rec.ep0[q]; cs.ep(2 * q + 1) = rec.ep1[q]; }
        const uint32_t* src = reinterpret_cast<const uint32_t*>(ci.qw);  // 8-byte aligned in PBRec
#pragma unroll 1
        for (int w = 0; w < (W + 3) / 4; w++) cs.qw4(w) = src[w];
        infill(tb, cs, bm.dm, T, direct);
    }
    if (qstep > 1) __syncwarp(group);
    uint32_t formats = 0, matched = 0, final_q = ci.ql;  // formats: a byte per partition

    // The texel's partition endpoints change only with the partition, so they are read again
    // only when it does (never, for one partition).  A decoded channel is floor(v + 1/2) of
    // v = u0 + (u1 - u0) w1 / 64, the integer (u0 w0 + u1 w1 + 32) >> 6: v is a multiple of 1/64
    // below 2^16, so v + 1/128 is exact and rounds to that integer.
    auto final_error = [&]() {
        float total = 0.0f;
        float4 base = mk(0.0f), offs = mk(0.0f);
        int pc = -1;
#pragma unroll 1
        for (int t = 0; t < T; t++) {
            const int p = pt.part(t);
            if (p != pc) {
                const uint2 u = cs.u(p);
                base = x257(u.x);
                offs = (x257(u.y) - base) * (1.0f / 64.0f);
                base = base + mk(1.0f / 128.0f);
                pc = p;
            }
            const float w1 = rn_small(__half2float(cs.s(t)) * (1.0f / 16.0f));
            const float4 x = px[t];
            float4 d;
            d.x = x.x - rn_small(base.x + offs.x * w1);
            d.y = x.y - rn_small(base.y + offs.y * w1);
            d.z = x.z - rn_small(base.z + offs.z * w1);
            d.w = x.w - rn_small(base.w + offs.w * w1);
            total = total + dot4(d * d, cw);
        }
        if (total < snap->err) {  // the best so far (ERR_DEFAULT at first)
            uint4* d = reinterpret_cast<uint4*>(snap);  // 16-byte aligned: 112-byte records
            d[0] = make_uint4(__float_as_uint(total), (uint32_t)ci.bm | final_q << 16 | matched << 24,
                              formats, 0u);
            d[1] = make_uint4(packed[0].x, packed[0].y, packed[1].x, packed[1].y);
            d[2] = make_uint4(packed[2].x, packed[2].y, packed[3].x, packed[3].y);
            const int nw = (W + 3) / 4;
#pragma unroll 1
            for (int i = 0; i < 4; i++) {
                uint4 v = make_uint4(0u, 0u, 0u, 0u);
                if (4 * i < nw) v.x = cs.qw4(4 * i);
                if (4 * i + 1 < nw) v.y = cs.qw4(4 * i + 1);
                if (4 * i + 2 < nw) v.z = cs.qw4(4 * i + 2);
                if (4 * i + 3 < nw) v.w = cs.qw4(4 * i + 3);
                d[3 + i] = v;
            }
        }
    };

    // ---------------- pass13: least-squares endpoints from the current weights
    int i0 = 0, counted = 0;  // the partition's first texel in partition order
#pragma unroll 1
    for (int q = q0; q < P; q += qstep) {
        if (HELP)
#pragma unroll 1
            for (; counted < q; counted++) i0 += tb.part_count(P, rec.entry, counted);
        const int n = P == 1 ? T : tb.part_count(P, rec.entry, q);
        const float ps = (float)n;
        // the scale direction and its sums are only read by the formats with a scale
        const bool scale = ci.fmt[q] == FMT_RGB_SCALE || ci.fmt[q] == FMT_RGB_SCALE_ALPHA;
        const float4 sdir = scale ? scale_dir(rec.avg[q], ps) : mk(0.0f);
        float wmin = 1.0f, wmax = 0.0f, ls = 0.0f, ms = 0.0f, rs = 0.0f, smin = 1e10f, smax = 0.0f, sv0 = 0.0f, sv1 = 0.0f;
        float4 cx = mk(0.0f), cy = mk(0.0f);
#pragma unroll 1
        for (int i = i0; i < i0 + n; i++) {
            const int t = pt.order(i);
            const float4 rgba = px[t];
            const float w = __half2float(cs.s(t)) * (1.0f / 1024.0f);
            wmin = fminf(wmin, w);
            wmax = fmaxf(wmax, w);
            const float om = 1.0f - w;
            ls = ls + om * om; ms = ms + om * w; rs = rs + w * w;
            const float4 cyc = rgba * w;
            cy = cy + cyc;
            cx = cx + (rgba - cyc);
            if (scale) {
                const float sc = dot3(rgba, sdir);
                if (sc < smin) smin = sc;
                if (sc > smax) smax = sc;
                sv0 = sv0 + (om * sc) * lsw;
                sv1 = sv1 + (w * sc) * lsw;
            }
        }
        i0 += n;
        counted = q + 1;
        const float4 colx = cx * cw, coly = cy * cw;
        const float4 lv = mk(ls) * cw, mv = mk(ms) * cw, rv = mk(rs) * cw;
        float4 rg = mk(0.0f);
        if (scale) {
            const float scalediv = clampf(smin / fmaxf(smax, 1e-10f), 0.0f, 1.0f);
            const float4 sds = sdir * smax;
            rg = make_float4(sds.x, sds.y, sds.z, scalediv);
        }
        float4 e0 = cs.ep(2 * q), e1 = cs.ep(2 * q + 1);
        if (wmin >= wmax * 0.999f) {
            const float4 ac = (colx + coly) / vmax(cw * ps, mk(1e-17f));
            if (ac.x == ac.x) { e0.x = ac.x; e1.x = ac.x; }
            if (ac.y == ac.y) { e0.y = ac.y; e1.y = ac.y; }
            if (ac.z == ac.z) { e0.z = ac.z; e1.z = ac.z; }
            if (ac.w == ac.w) { e0.w = ac.w; e1.w = ac.w; }
            rg.w = 1.0f;
        } else {
            const float4 det = (lv * rv) - (mv * mv);
            const float4 rdet = mk(1.0f) / det;
            const float4 mss = ((lv * lv) + mk(2.0f) * (mv * mv)) + (rv * rv);
            const float4 ne0 = ((rv * colx) - (mv * coly)) * rdet;
            const float4 ne1 = ((lv * coly) - (mv * colx)) * rdet;
            if (fabsf(det.x) > (mss.x * 1e-4f) && ne0.x == ne0.x && ne1.x == ne1.x) { e0.x = ne0.x; e1.x = ne1.x; }
            if (fabsf(det.y) > (mss.y * 1e-4f) && ne0.y == ne0.y && ne1.y == ne1.y) { e0.y = ne0.y; e1.y = ne1.y; }
            if (fabsf(det.z) > (mss.z * 1e-4f) && ne0.z == ne0.z && ne1.z == ne1.z) { e0.z = ne0.z; e1.z = ne1.z; }
            if (fabsf(det.w) > (mss.w * 1e-4f) && ne0.w == ne0.w && ne1.w == ne1.w) { e0.w = ne0.w; e1.w = ne1.w; }
            if (scale) {
                const float lx = ls * lsw, my = ms * lsw, rz = rs * lsw;
                const float lsdet = (lx * rz) - (my * my), lsrdet = 1.0f / lsdet;
                const float lsmss = ((lx * lx) + 2.0f * (my * my)) + (rz * rz);
                const float se0 = ((rz * sv0) - (my * sv1)) * lsrdet;
                const float se1 = ((lx * sv1) - (my * sv0)) * lsrdet;
                if ((fabsf(lsdet) > (lsmss * 1e-4f)) && se0 == se0 && se1 == se1 && se0 < se1) {
                    const float4 sdsm = sdir * se1;
                    rg = make_float4(sdsm.x, sdsm.y, sdsm.z, se0 / se1);
                }
            }
        }
        rgbs[q] = rg;
        cs.ep(2 * q) = e0; cs.ep(2 * q + 1) = e1;
    }
    // ---------------- pass14: pack at the trial quant level, then the "mod" level
    {
        const uint32_t used = 0xFFFFFFFFu >> (8 * (4 - P));
        auto joined = [&](uint32_t f) {  // of the candidate's lanes
            for (int o = spread; o < 32; o <<= 1) f |= __shfl_xor_sync(group, f, o);
            return f;
        };
#pragma unroll
        for (int q = 0; q < 4; q++) packed[q] = make_uint2(0u, 0u);
#pragma unroll 1
        for (int q = q0; q < P; q += qstep) {
            const uint4 v = Packer::pack(cu2u, cs.ep(2 * q), cs.ep(2 * q + 1), rgbs[q], ci.fmt[q], ci.ql);
            formats |= v.x << (8 * q);
            packed[q] = make_uint2(v.y, v.z);
        }
        formats = joined(formats);
        if (P >= 2 && ci.ql != ci.qlm && formats == ((formats & 0xFF) * 0x01010101u & used)) {
            uint32_t fm = 0;
#pragma unroll 1
            for (int q = q0; q < P; q += qstep) {
                const uint4 v = Packer::pack(cu2u, cs.ep(2 * q), cs.ep(2 * q + 1), rgbs[q], ci.fmt[q], ci.qlm);
                fm |= v.x << (8 * q);
                packed_mod[q] = make_uint2(v.y, v.z);
                if (qstep == 1 && v.x != (fm & 0xFF)) break;
            }
            fm = joined(fm);
            if (fm == ((fm & 0xFF) * 0x01010101u & used)) {
                matched = 1;
                final_q = ci.qlm;
                formats = fm;
#pragma unroll 1
                for (int q = q0; q < P; q += qstep) packed[q] = packed_mod[q];
            }
        }
    }
    // ---------------- pass15
#pragma unroll 1
    for (int q = q0; q < P; q += qstep) {
        I4 o0, o1;
        unpack_endpoints(formats >> (8 * q) & 0xFF, packed[q].x, packed[q].y, o0, o1);
        cs.u(q) = make_uint2((uint32_t)o0.x | (uint32_t)o0.y << 8 | (uint32_t)o0.z << 16 | (uint32_t)o0.w << 24,
                             (uint32_t)o1.x | (uint32_t)o1.y << 8 | (uint32_t)o1.z << 16 | (uint32_t)o1.w << 24);
    }
    if (qstep > 1) {  // the rest is the first lane's
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int lane = first + (q & (qstep - 1)) * spread;
            packed[q].x = __shfl_sync(group, packed[q].x, lane);
            packed[q].y = __shfl_sync(group, packed[q].y, lane);
        }
        __syncwarp(group);
        if (q0 != 0) return false;
    }
    // ---------------- pass16: move each weight one quant step if that lowers the error
    bool moved = false;
#pragma unroll 1
    for (int turn = it == 0 ? 0 : 1; turn < 2; turn++) {
    if (turn == 1) {
    float4 base = mk(0.0f), offs = mk(0.0f);
    int pc = -1;
    auto endpoints = [&](int p) {  // of texel partition p, read again when it changes
        if (p == pc) return;
        const uint2 u = cs.u(p);
        base = x257(u.x);
        offs = (x257(u.y) - base) * (1.0f / 64.0f);
        pc = p;
    };
    if (direct) {
#pragma unroll 1
        for (int t = 0; t < T; t++) {
            const int32_t uqw = cs.qw(t);
            const uint32_t pn = tb.prev_next(bm.quant, uqw);
            const int32_t dn = pn & 0xFF, up = (pn >> 8) & 0xFF;
            endpoints(pt.part(t));
            const float4 cd = (base + offs * (float)uqw) - px[t];
            const float4 cdd = cd + offs * (float)(dn - uqw), cdu = cd + offs * (float)(up - uqw);
            const float eb = dot4(cd * cd, cw), ed = dot4(cdd * cdd, cw), eu = dot4(cdu * cdu, cw);
            int32_t nw = uqw;
            if ((eu < eb) && (eu < ed) && (uqw < 64)) nw = up;
            else if ((ed < eb) && (uqw > 0)) nw = dn;
            if (nw != uqw) {
                moved = true;
                cs.qw(t) = (uint8_t)nw;
                cs.s(t) = __ushort2half_rn((unsigned short)(nw * 16));
            }
        }
    } else {
#pragma unroll 1
        for (int we = 0; we < W; we++) {
            const int32_t uqw = cs.qw(we);
            const uint32_t pn = tb.prev_next(bm.quant, uqw);
            const float dn = (float)(pn & 0xFF), up = (float)((pn >> 8) & 0xFF), ub = (float)uqw;
            const float ddn = dn - ub, dup = up - ub;
            float4 ebv = mk(0.0f), edv = mk(0.0f), euv = mk(0.0f);
            const int nt = tb.wt_count(bm.dm, we), wbase = dmi.wt_base + tb.wt_start(bm.dm, we);
#pragma unroll 1
            for (int te = 0; te < nt; te++) {
                // the weight's own contribution to texel t is the w2t entry's
                // (each (texel, weight) pair appears once in both maps)
                const uint32_t we2 = tb.w2t(wbase + te);
                const int t = we2 & 0xFF;
                const float twb = (float)(we2 >> 8) * (1.0f / 16.0f);
                const float wb = __half2float(cs.s(t)) * (1.0f / 16.0f);
                endpoints(pt.part(t));
                const float4 cd = (base + offs * wb) - px[t];
                const float4 cdd = cd + offs * (ddn * twb), cdu = cd + offs * (dup * twb);
                ebv = ebv + cd * cd; edv = edv + cdd * cdd; euv = euv + cdu * cdu;
            }
            const float eb = dot4(ebv, cw), ed = dot4(edv, cw), eu = dot4(euv, cw);
            float dw = 0.0f;
            if ((eu < eb) && (eu < ed) && (uqw < 64)) dw = dup;
            else if ((ed < eb) && (uqw > 0)) dw = ddn;
            if (dw != 0.0f) {
                moved = true;
                cs.qw(we) = (uint8_t)(uqw + (int)dw);
#pragma unroll 1
                for (int te = 0; te < nt; te++) {
                    const uint32_t we2 = tb.w2t(wbase + te);
                    __half& sv = cs.s(we2 & 0xFF);
                    sv = __float2half_rn(__half2float(sv) + dw * (float)(we2 >> 8));
                }
            }
        }
    }
    // In iteration 0 a pass16 that moved no weight leaves the weights and endpoints of the
    // error taken before it: the same total, which cannot improve the snapshot.
    if (it == 0 && !moved) break;
    }
    final_error();
    }
    return moved;
}

// A refinement-tail entry: the partitioned block (lb * slots + slot), the candidate and the
// next iteration, then the state an iteration carries over (endpoints, weights; the best
// result so far is in the candidate's snapshot already).
__device__ __forceinline__ void write_tail(const KernelArgs& a, const Cand& c, uint32_t pbi, int k, int it, int pos) {
    uint4* e = a.tail + (size_t)pos * kTailWords;
    e[0] = make_uint4(pbi, (uint32_t)k | (uint32_t)it << 8, 0u, 0u);
    float4* ep = reinterpret_cast<float4*>(e + 1);
#pragma unroll
    for (int i = 0; i < 8; i++) ep[i] = c.ep(i);
    const int n4 = (a.L.max_w + 3) / 4;
    uint32_t* w = reinterpret_cast<uint32_t*>(e + 9);
#pragma unroll 1
    for (int i = 0; i < n4; i++) w[i] = c.qw4(i);
}

// CPB: candidate threads per partitioned block (refine_cpb of the launch's top-N), a
// template parameter so that the full search's instance (8) keeps constant indexing.
// U8: texels staged as RGBA8 (refine_u8).  HELP: launches of few candidates (refine_spread below
// 32), an instance of its own: with both in one, 1024x1024 at 4x4 took 10.5 ms instead of 10.0.
template <int CPB, bool U8, bool HELP>
__global__ void __launch_bounds__(kRefineThreads, kRefineCtas) k_refine(const __grid_constant__ KernelArgs a) {
    extern __shared__ __align__(16) uint8_t smem[];
    const int T = a.L.T;
    constexpr int cpb = CPB;
    const RefineLayout fl = refine_layout(T, a.L.max_w, refine_pbs(T, CPB), U8, false);
    using Px = typename std::conditional<U8, uchar4, float4>::type;
    using Pe = typename std::conditional<U8, uint16_t, uint8_t>::type;
    const int px_row = px_row_bytes(T, U8), part_row = part_row_bytes(T, sizeof(Pe));
    uint8_t* pos_of = smem + fl.pos;                                   // by slot: staging position
    uint8_t* map = smem + fl.map;                                      // by rank: the candidate's slot
    uint32_t* staged = reinterpret_cast<uint32_t*>(smem + fl.staged);  // by staged partitioned block: lb + 1 | slot << 27, 0 if none
    int* keys = reinterpret_cast<int*>(smem + fl.keys);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // Items: every slot of every block in slot-major order (consecutive CTAs hold
    // partitioned blocks of the same slot, hence the same partition count, so
    // co-resident warps run the same code), or the proposal pass's work list.
    const int nb = list_blocks(a);
    const int npb = a.pb_list ? pb_total(a) : nb * a.slots;
    if ((refine_spread(npb) < 32) != HELP) return;  // the other instance's launch
    const int spread = HELP ? refine_spread(npb) : 32, pbs = refine_group(T, CPB, spread);
    const int ngroups = refine_groups(npb, pbs);
    // this thread's place among those that run candidates, the first `spread` lanes of each warp
    const int place = lane < spread ? warp * spread + lane : kRefineThreads;
    const int iters = a.refine_iters > 0 ? a.refine_iters : 6;
    __shared__ unsigned int refined[4];  // candidates refined by this CTA, by P (work counters)
    __shared__ int live_in_warp[kRefineThreads / 32];
    __shared__ int spill_base;
    if (tid < 4) refined[tid] = 0;
    // Hand the last candidates to the tail (until it is found full).  A launch of one wave is as long
    // as its longest chain of iterations, which a second kernel would lengthen: the full search
    // keeps its candidates then, the proposal pass hands them over for the last iteration only.
    const bool one_wave = refine_one_wave(ngroups);
    bool spill = a.tail != nullptr && T <= kTailMaxTexels && !(one_wave && !a.prop);
    const int spill_live = refine_spill_live(U8, a.prop != nullptr, ngroups);
    // (the first group's barrier below orders these writes before any read)
    for (int grp = blockIdx.x; grp < ngroups; grp += gridDim.x) {
        {
            const int pbl = tid / cpb, k = tid % cpb;
            const int li = grp * pbs + pbl;
            int key = 0x3FFFFF;  // empty slots sort last
            uint32_t item = 0;
            if (pbl < pbs && li < npb) {
                int slot, lb;
                if (a.pb_list) pb_item(a, li, lb, slot);
                else { slot = li / nb; lb = li % nb; }
                item = (uint32_t)(lb + 1) | ((uint32_t)slot << 27);
                const PBRec& r = a.pbrec[(size_t)lb * a.slots + slot];
                if (k < (int)r.ncand) {
                    const int dm = reinterpret_cast<const DevBm*>(a.tables + a.L.off_bm)[r.c[k].bm].dm;
                    int fk = 0;
#pragma unroll 1
                    for (int q = 0; q < 4; q++) { const int f = r.c[k].fmt[q]; fk = fk * 8 + (f == 0 ? 0 : f == 4 ? 1 : f == 6 ? 2 : f == 8 ? 3 : f == 10 ? 4 : f == 12 ? 5 : 6); }
                    if constexpr (U8) {
                        // weight count, decimation mode, partition count, first format: pass16's loops are most of an iteration
                        const int W = reinterpret_cast<const DevDm*>(a.tables + a.L.off_dm)[dm].W;
                        key = (((W - 1) << 7 | dm) << 2 | ((int)r.P - 1)) << 3 | fk >> 9;
                    } else {
                        key = ((((int)r.P - 1) << 12 | fk) << 7) | dm;  // partition count, formats, decimation mode
                    }
                }
                if (r.ncand > 0) {
                    const int P = r.P;
                    const uint32_t* prow = P > 1 ? part2_row(a, P, (int)r.entry) : nullptr;
                    const uint8_t* counts = P > 1 ? a.tables + a.L.off_part_counts + ((size_t)(P - 2) * 1024 + r.entry) * 4 : nullptr;
                    const BlockSrc src = block_src(a, chunk_block(a, lb));
                    Px* row = reinterpret_cast<Px*>(smem + fl.px + pbl * px_row);
#pragma unroll 1
                    for (int t = k; t < T; t += cpb) {
                        if constexpr (U8) row[t] = src_rgba8(src, a.L.bx, t);
                        else row[t] = src_texel(src, a.L.bx, t);
                    }
                    if (k == 0) PartRow<Pe>{reinterpret_cast<Pe*>(smem + fl.part + pbl * part_row)}.set(prow, counts, T);
                }
            }
            keys[tid] = key * kRefineThreads + tid;  // unique keys: P, formats, decimation mode, then position
            if (k == 0 && pbl < pbs) staged[pbl] = item;
        }
        __syncthreads();
        // The thread of place i takes the candidate of rank i in (partition count, endpoint formats,
        // decimation mode) order, so a warp's candidates mostly take the same packing path
        // and share loop bounds and table rows; the rank is also its slot.
        int cand = -1;  // slot of the candidate this thread runs
        {
            const int kk = keys[tid];
            int rank = 0;
            const int4* k4 = reinterpret_cast<const int4*>(keys);
#pragma unroll 2
            for (int j = 0; j < kRefineThreads / 4; j++) {
                const int4 o = k4[j];
                rank += (o.x < kk) + (o.y < kk) + (o.z < kk) + (o.w < kk);
            }
            map[rank] = (uint8_t)tid;
            __syncthreads();  // also: every thread has read the keys, which the first iteration overwrites
            const int mine = place < kRefineThreads ? map[place] : kRefineThreads * cpb;
            const int pbl = mine / cpb, k = mine % cpb;
            const uint32_t item = pbl < pbs ? staged[pbl] : 0u;
            if (item != 0) {
                const int lb = (int)(item & 0x07FFFFFFu) - 1, slot = (int)(item >> 27);
                const size_t pbi = (size_t)lb * a.slots + slot;
                a.snaps[pbi * kNumCand + k].err = ERR_DEFAULT;  // inert slot unless refined below
                if (k < (int)a.pbrec[pbi].ncand) {
                    cand = place;
                    pos_of[place] = (uint8_t)mine;
                    if (a.work) atomicAdd(&refined[a.pbrec[pbi].P - 1], 1u);
                }
            }
        }
        // Iterations.  Candidates stop at different iterations (at a fixed point of pass16),
        // so after every iteration the live candidates are gathered onto the lowest threads,
        // in the same order: warps stay full while any work is left, and warps with none
        // wait at the barrier without issuing.  The staged texels and each candidate's state
        // stay where they are; only the candidate-to-thread map changes.
        for (int it = 0; ; it++) {
            const bool live = cand >= 0;
            const unsigned bal = __ballot_sync(0xFFFFFFFFu, live);
            if (lane == 0) live_in_warp[warp] = __popc(bal);
            __syncthreads();  // also: every thread has read map[] before it is rewritten
            int nlive = 0, before = 0;
#pragma unroll
            for (int w = 0; w < kRefineThreads / 32; w++) {
                const int n = live_in_warp[w];
                nlive += n;
                before += w < warp ? n : 0;
            }
            if (nlive == 0) break;
            const int rank = before + __popc(bal & ((1u << lane) - 1u));
            if (spill && it > 0 && nlive <= spill_live && (!one_wave || it + 1 >= iters)) {
                // Few candidates left: hand them to the tail pass, which runs them densely, and
                // take the next group instead of holding the CTA for them.
                if (tid == 0) {
                    spill_base = atomicAdd(a.tail_count, nlive);
                    if (a.work) atomicAdd(a.work + 13, (unsigned long long)nlive);
                }
                __syncthreads();
                const int sb = spill_base, pos = sb + rank;
                if (sb + nlive <= a.tail_cap) {
                    // (the next group's staging writes no slot state: it is first written after
                    // its staging barriers)
                    if (live) {
                        const uint32_t item = staged[pos_of[cand] / cpb];
                        const uint32_t pbi = ((item & 0x07FFFFFFu) - 1) * (uint32_t)a.slots + (item >> 27);
                        write_tail(a, Cand(smem, fl, cand), pbi, pos_of[cand] % cpb, it, pos);
                    }
                    if (a.work && tid == 0) atomicAdd(a.work + 14, (unsigned long long)nlive);
                    __syncthreads();  // staged[] is rewritten next
                    break;
                }
                if (live && pos < a.tail_cap) a.tail[(size_t)pos * kTailWords].x = 0xFFFFFFFFu;  // reserved, left empty
                spill = false;  // the tail is full: finish here
            }
            if (live) map[rank] = (uint8_t)cand;
            __syncthreads();
            cand = place < nlive ? map[place] : -1;
            const int shared_cand = HELP ? __shfl_sync(0xFFFFFFFFu, cand, lane & (spread - 1)) : cand;
            if (shared_cand >= 0) {
                const int pbl = pos_of[shared_cand] / cpb, k = pos_of[shared_cand] % cpb;
                const uint32_t item = staged[pbl];
                const size_t pbi = (size_t)((item & 0x07FFFFFFu) - 1) * a.slots + (item >> 27);
                const PBRec& rec = a.pbrec[pbi];
                Snap* snap = &a.snaps[pbi * kNumCand + k];
                const TexelRow<U8> row{reinterpret_cast<const Px*>(smem + fl.px + pbl * px_row)};
                const PartRow<Pe> part{reinterpret_cast<Pe*>(smem + fl.part + pbl * part_row)};
                const bool moved = refine_step<HELP>(a, rec, (int)rec.P, k, row, part, Cand(smem, fl, shared_cand), snap, it, spread);
                if (!moved || it + 1 >= iters) cand = -1;
            }
            // (the next pass's first barrier orders this iteration's state writes before
            // other threads read them; the counts and the map were read before its second)
        }
    }
    if (a.work && tid < 4 && refined[tid]) atomicAdd(a.work + 6 + tid, (unsigned long long)refined[tid]);
}

// The candidates k_refine handed over, one per thread with its own staged texels (RGBA8),
// iterated with the same gathering of live candidates onto the lowest threads.  The CTAs stay
// resident: a CTA's 128 slots are refilled whenever at most kTailRefillAt of them hold a
// live candidate, each warp claiming list entries for its own free slots from
// tail_count[1], and the new candidates join the live list behind the running ones.  (Fixed
// batches of 128 entries would hold each CTA until the slowest candidate of its batch ended.)
constexpr int kTailCtas = 4;
constexpr int kTailRefillAt = 64;
__global__ void __launch_bounds__(kRefineThreads, kTailCtas) k_refine_tail(const __grid_constant__ KernelArgs a) {
    extern __shared__ __align__(16) uint8_t smem[];
    const int T = a.L.T;
    const RefineLayout fl = refine_layout(T, a.L.max_w, kRefineThreads, true, true);
    const int px_row = px_row_bytes(T, true), part_row = part_row_bytes(T, 1);
    uint8_t* map = smem + fl.map;                                     // by rank: the candidate's slot
    uint8_t* next_it = smem + fl.next_it;                             // by slot
    uint32_t* pbi_of = reinterpret_cast<uint32_t*>(smem + fl.item);   // by slot
    uint8_t* k_of = smem + fl.pos;                                    // by slot: the candidate
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned below = (1u << lane) - 1u;
    __shared__ int live_in_warp[kRefineThreads / 32], new_in_warp[kRefineThreads / 32];
    __shared__ uint8_t busy[kRefineThreads];  // slot holds a candidate that has not ended
    __shared__ int dry_flag;                  // the list has no unclaimed entry left
    busy[tid] = 0;
    if (tid == 0) dry_flag = 0;
    const int total = min(*a.tail_count, a.tail_cap);
    int* claim = a.tail_count + 1;
    const int iters = a.refine_iters > 0 ? a.refine_iters : 6;
    // Few entries are spread over more warps, as in k_refine: only the first `spread` lanes of a
    // warp take any.
    const int warps = (int)gridDim.x * (kRefineThreads / 32);
    const int spread = total <= warps * 8 ? 8 : total <= warps * 16 ? 16 : 32;
    const int place = lane < spread ? warp * spread + lane : kRefineThreads;
    int cand = -1;     // the slot whose candidate this thread runs
    bool dry = false;  // CTA-uniform
    for (;;) {
        const bool live = cand >= 0;
        const unsigned bal = __ballot_sync(0xFFFFFFFFu, live);
        if (lane == 0) live_in_warp[warp] = __popc(bal);
        __syncthreads();  // also orders the last step's state writes and slot releases
        int nlive = 0, before = 0;
#pragma unroll
        for (int w = 0; w < kRefineThreads / 32; w++) {
            const int n = live_in_warp[w];
            nlive += n;
            before += w < warp ? n : 0;
        }
        int nnew = 0, new_before = 0, filled = -1;
        unsigned bnew = 0;
        if (!dry && nlive * 32 <= kTailRefillAt * spread) {
            // Thread tid stages into slot tid when that slot is free and its warp's claim
            // reached an entry for it.
            const bool fr = busy[tid] == 0 && lane < spread;
            const unsigned fb = __ballot_sync(0xFFFFFFFFu, fr);
            const int nfree = __popc(fb);
            int base = 0;
            if (lane == 0 && nfree > 0) base = atomicAdd(claim, nfree);
            base = __shfl_sync(0xFFFFFFFFu, base, 0);
            if (lane == 0 && nfree > 0 && base + nfree >= total) dry_flag = 1;
            const int idx = base + __popc(fb & below);
            if (fr && idx < total) {
                const uint4* e = a.tail + (size_t)idx * kTailWords;
                const uint4 h = e[0];
                if (h.x != 0xFFFFFFFFu) {
                    const int lb = (int)(h.x / (uint32_t)a.slots);
                    const PBRec& r = a.pbrec[h.x];
                    const int P = (int)r.P, k = (int)(h.y & 0xFF);
                    const uint32_t* prow = P > 1 ? part2_row(a, P, (int)r.entry) : nullptr;
                    const uint8_t* counts = P > 1 ? a.tables + a.L.off_part_counts + ((size_t)(P - 2) * 1024 + r.entry) * 4 : nullptr;
                    const BlockSrc src = block_src(a, chunk_block(a, lb));
                    uchar4* row = reinterpret_cast<uchar4*>(smem + fl.px + tid * px_row);
#pragma unroll 1
                    for (int t = 0; t < T; t++) row[t] = src_rgba8(src, a.L.bx, t);
                    PartRow<uint8_t>{smem + fl.part + tid * part_row}.set(prow, counts, T);
                    const Cand c(smem, fl, tid);
#pragma unroll 1
                    for (int i = 0; i < 8; i++) c.ep(i) = reinterpret_cast<const float4*>(e + 1)[i];
                    const int n4 = (a.L.max_w + 3) / 4;
                    const uint32_t* w = reinterpret_cast<const uint32_t*>(e + 9);
#pragma unroll 1
                    for (int i = 0; i < n4; i++) c.qw4(i) = w[i];
                    const RTabs tb{a.tables, &a.L};
                    const int dm = tb.bm(r.c[k].bm).dm;
                    infill(tb, c, dm, T, tb.dm(dm).W == T);
                    k_of[tid] = (uint8_t)k;
                    next_it[tid] = (uint8_t)(h.y >> 8);
                    pbi_of[tid] = h.x;
                    busy[tid] = 1;
                    filled = tid;
                }
            }
            bnew = __ballot_sync(0xFFFFFFFFu, filled >= 0);
            if (lane == 0) new_in_warp[warp] = __popc(bnew);
            __syncthreads();  // the staged slots, the new counts and the flag
#pragma unroll
            for (int w = 0; w < kRefineThreads / 32; w++) {
                const int n = new_in_warp[w];
                nnew += n;
                new_before += w < warp ? n : 0;
            }
            dry = dry_flag != 0;
        }
        const int n = nlive + nnew;
        if (n == 0) {
            if (dry) break;
            continue;  // every claimed entry was a reservation left empty: claim again
        }
        if (live) map[before + __popc(bal & below)] = (uint8_t)cand;
        if (filled >= 0) map[nlive + new_before + __popc(bnew & below)] = (uint8_t)filled;
        __syncthreads();
        cand = place < n ? map[place] : -1;
        const int shared_cand = __shfl_sync(0xFFFFFFFFu, cand, lane & (spread - 1));
        if (shared_cand >= 0) {
            const uint32_t pbi = pbi_of[shared_cand];
            const int k = (int)k_of[shared_cand], it = next_it[shared_cand];
            const PBRec& rec = a.pbrec[pbi];
            Snap* snap = &a.snaps[(size_t)pbi * kNumCand + k];
            const TexelRow<true> row{reinterpret_cast<const uchar4*>(smem + fl.px + shared_cand * px_row)};
            const PartRow<uint8_t> part{smem + fl.part + shared_cand * part_row};
            const bool moved = spread == 32 ? refine_step<false>(a, rec, (int)rec.P, k, row, part, Cand(smem, fl, shared_cand), snap, it, 32)
                                                : refine_step<true>(a, rec, (int)rec.P, k, row, part, Cand(smem, fl, shared_cand), snap, it, spread);
            if (cand >= 0) next_it[cand] = (uint8_t)(it + 1);
            if (cand >= 0 && (!moved || it + 1 >= iters)) {
                busy[cand] = 0;  // released: read by the next refill, after the next barrier
                cand = -1;
            }
        }
    }
}

size_t refine_tail_smem_bytes(int T, int max_w) { return (size_t)refine_layout(T, max_w, kRefineThreads, true, true).total; }

// ------------------------------------------------------------ k_select_pack
// bits | trits << 4 | quints << 5 of the quantisation methods
__constant__ uint8_t c_method[21] = {1, 16, 2, 32, 17, 3, 33, 18, 4, 34, 19, 5, 35, 20, 6, 36, 21, 7, 37, 22, 8};
__device__ __forceinline__ void method_of(int q, int& bits, int& trits, int& quints) {
    const int m = c_method[q];
    bits = m & 15; trits = m & 16; quints = m & 32;
}
__device__ __forceinline__ int ise_bits(int n, int q) {
    int b, t, qu;
    method_of(q, b, t, qu);
    if (t) return (n * (8 + 5 * b) + 4) / 5;
    if (qu) return (n * (7 + 3 * b) + 2) / 3;
    return n * b;
}
// ORs the low `width` bits (at most 32) of v into a 128-bit value at bit `off`.
__device__ __forceinline__ void or_bits(uint32_t (&acc)[4], uint32_t v, int off, int width) {
    const int word = off >> 5, sh = off & 31;
    const uint32_t lo = v << sh, hi = sh + width > 32 ? v >> (32 - sh) : 0u;
#pragma unroll
    for (int j = 0; j < 4; j++) acc[j] |= (j == word ? lo : 0u) | (j == word + 1 ? hi : 0u);
}
// Value i of an integer sequence (code/physical_compression.cpp:672-826) of n codes in v (zeros
// after them): its bits, with its share of the group's packed trits or quints, at their place.
__device__ __forceinline__ void or_ise(uint32_t (&acc)[4], const TableLayout& L, const uint8_t* tabs, int q, const uint8_t* v, int i, int off) {
    int bits, trits, quints;
    method_of(q, bits, trits, quints);
    const uint32_t m = v[i] & ((1u << bits) - 1u);
    if (trits) {
        const int g = i / 5, e = i - 5 * g;
        const uint8_t* d = v + 5 * g;
        const uint32_t T = (tabs + L.off_trits)[((((d[4] >> bits) * 3 + (d[3] >> bits)) * 3 + (d[2] >> bits)) * 3 + (d[1] >> bits)) * 3 + (d[0] >> bits)];
        const int at = (0x75420 >> (4 * e)) & 15, tb = (e == 2 || e == 4) ? 1 : 2;
        or_bits(acc, m | ((T >> at) & ((1u << tb) - 1u)) << bits, off + g * (8 + 5 * bits) + e * bits + at, bits + tb);
    } else if (quints) {
        const int g = i / 3, e = i - 3 * g;
        const uint8_t* d = v + 3 * g;
        const uint32_t Q = (tabs + L.off_quints)[((d[2] >> bits) * 5 + (d[1] >> bits)) * 5 + (d[0] >> bits)];
        const int at = (0x530 >> (4 * e)) & 15, qb = e == 0 ? 3 : 2;
        or_bits(acc, m | ((Q >> at) & ((1u << qb) - 1u)) << bits, off + g * (7 + 3 * bits) + e * bits + at, bits + qb);
    } else {
        or_bits(acc, m, off + i * bits, bits);
    }
}

// A block's codes while a warp packs it: weights and colour values, zeros after them.
struct PackWarp {
    uint8_t w[72], c[32];
};

// The block of nw weight codes of method wq, nc colour codes of method cq at bit coff, and the bits
// in acc of this lane, packed by a warp: lane i takes weights i and i + 32 and colour value i.  The
// weights fill the block from its last bit down.
__device__ __forceinline__ uint4 pack_block(const KernelArgs& a, const PackWarp& s, int nw, int wq, int nc, int cq, int coff, uint32_t (&acc)[4], int lane) {
    uint32_t ws[4] = {0u, 0u, 0u, 0u};
#pragma unroll 1
    for (int i = lane; i < nw; i += 32) or_ise(ws, a.L, a.tables, wq, s.w, i, 0);
    if (lane < nc) or_ise(acc, a.L, a.tables, cq, s.c, lane, coff);
#pragma unroll
    for (int j = 0; j < 4; j++) acc[j] = __reduce_or_sync(0xFFFFFFFFu, acc[j] | __brev(ws[3 - j]));
    return make_uint4(acc[0], acc[1], acc[2], acc[3]);
}

// pass18, the host argmin and the physical block of one block, by a warp: the candidates' errors
// a lane each, then pack_block.  One thread a block, which this replaces, took 62 us for 256
// blocks or fewer (a chain of dependent loads and byte writes); this takes 10 us.  For the 262,144
// blocks of a proposal pass it takes 178 us instead of 134, which its fallback pass's 10 instead of 54
// gives back.
__device__ __forceinline__ void select_pack_one(const KernelArgs& a, int lb, int blk, PackWarp& s, int lane) {
    constexpr unsigned FULL = 0xFFFFFFFFu;
    // slots the front filled: all of them, or P=1 (unless skipped) plus the proposed partitionings
    const int nslots = a.prop ? 1 + (int)a.prop[lb].n : a.slots;
    const int s0 = a.prop && (a.prop[lb].flags & 1) ? 1 : 0;
    const size_t pb0 = (size_t)lb * a.slots;
    uint32_t key = FULL;  // errors are never negative: their bits order like them
    int at = 0x7FFFFFFF;
#pragma unroll 1
    for (int i = s0 * kNumCand + lane; i < nslots * kNumCand; i += 32) {
        if ((i & (kNumCand - 1)) >= (int)a.pbrec[pb0 + i / kNumCand].ncand) continue;
        const float e = a.snaps[pb0 * kNumCand + i].err;
        if (e < 1e30f && __float_as_uint(e) < key) { key = __float_as_uint(e); at = i; }
    }
    const uint32_t best_bits = __reduce_min_sync(FULL, key);
    const int win = __reduce_min_sync(FULL, key == best_bits ? at : 0x7FFFFFFF);
    const bool found = best_bits != FULL;
    const float best = found ? __uint_as_float(best_bits) : 1e30f;
    if (!found && a.reroute_list) {  // proposal search found nothing: hand the block to the full search
        if (lane == 0) {
            const int pos = atomicAdd(a.reroute_count, 1);
            a.reroute_list[pos] = blk;
            a.reroute_err[pos] = 3e38f;
        }
        return;
    }
    if (a.prev_err && !(best < a.prev_err[lb])) return;  // the proposal search's result stands
    if (a.reroute_list && a.reroute_above > 0.0f && best > a.reroute_above && lane == 0) {
        // a poor proposal-search result: write it, and let the full search try to beat it
        const int pos = atomicAdd(a.reroute_count, 1);
        a.reroute_list[pos] = blk;
        a.reroute_err[pos] = best;
    }
    uint32_t acc[4] = {0u, 0u, 0u, 0u};
    uint4 out = make_uint4(0u, 0u, 0u, 0u);
    uint32_t* sym = a.symbolic ? a.symbolic + (size_t)blk * 108 : nullptr;
    if (sym) {
        for (int i = lane; i < 108; i += 32) sym[i] = i == 0 ? __float_as_uint(best) : 0u;
        __syncwarp();
    }
    if (found) {
        const PBRec& rec = a.pbrec[pb0 + win / kNumCand];
        const Snap& sn = a.snaps[pb0 * kNumCand + win];
        const DevBm bm = reinterpret_cast<const DevBm*>(a.tables + a.L.off_bm)[sn.bm];
        const int W = reinterpret_cast<const DevDm*>(a.tables + a.L.off_dm)[bm.dm].W;
        const int pc = (int)rec.P, q = bm.quant, cq = sn.final_q;
        const uint32_t fmts = *reinterpret_cast<const uint32_t*>(sn.ffmt), seed = rec.seed;
        auto fmt = [&](int i) { return (int)((fmts >> (8 * i)) & 0xFF); };
        // weights: requantise 0..64 to the ISE alphabet and scramble
        const uint8_t* wscr = a.tables + a.L.off_wscr + q * 32;
        const float top = (float)c_levels_r[q] - 1.0f;
        __syncwarp();
#pragma unroll 1
        for (int i = lane; i < W + 4; i += 32) s.w[i] = i < W ? wscr[(int)(((float)sn.qw[i] / 64.0f) * top + 0.5f)] : 0;
        s.c[lane] = 0;  // (at most 18 values)
        __syncwarp();
        // colour values of partition lane / 8, one partition after another
        int nc = 0, first = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int n = i < pc ? 2 * (fmt(i) >> 2) + 2 : 0;
            if (i < lane / 8) first += n;
            nc += n;
        }
        if (lane / 8 < pc && (lane & 7) < 2 * (fmt(lane / 8) >> 2) + 2)
            s.c[first + (lane & 7)] = (a.tables + a.L.off_cscr + (cq - 4) * 256)[sn.packed[lane]];
        __syncwarp();
        if (lane == 0) {
            or_bits(acc, bm.mode_index, 0, 11);
            or_bits(acc, (uint32_t)pc - 1u, 11, 2);
            if (pc > 1) {
                or_bits(acc, seed & 1023u, 13, 10);
                if (sn.matched) {
                    or_bits(acc, ((uint32_t)fmt(0) << 2) & 63u, 23, 6);
                } else {
                    int low = 4;
                    for (int i = 0; i < pc; i++) low = min(fmt(i) >> 2, low);
                    if (low == 3) low = 2;
                    int et = low + 1, bp = 2;
                    for (int i = 0; i < pc; i++) { et |= ((fmt(i) >> 2) - low) << bp; bp++; }
                    for (int i = 0; i < pc; i++) { et |= (fmt(i) & 3) << bp; bp += 2; }
                    const int hs = 3 * pc - 4;
                    or_bits(acc, et & 0x3F, 23, 6);
                    or_bits(acc, ((uint32_t)et >> 6) & ((1u << hs) - 1u), 128 - ise_bits(W, q) - hs, hs);
                }
            } else {
                or_bits(acc, fmt(0) & 15, 13, 4);
            }
        }
        out = pack_block(a, s, W, q, nc, cq, pc == 1 ? 17 : 29, acc, lane);
        if (sym) {
            if (lane == 0) { sym[1] = bm.mode_index; sym[2] = (uint32_t)pc; sym[3] = seed; sym[4] = sn.matched; sym[5] = (uint32_t)cq; }
            if (lane < 4) sym[8 + lane] = (uint32_t)fmt(lane);
            sym[12 + lane] = sn.packed[lane];
            sym[44 + lane] = sn.qw[lane];
            sym[76 + lane] = sn.qw[32 + lane];
        }
        __syncwarp();  // the codes are read
    }
    if (lane == 0) *block_dst(a, blk) = out;
}

constexpr int kPackWarps = 4;
__global__ void __launch_bounds__(kPackWarps * 32) k_select_pack(const __grid_constant__ KernelArgs a) {
    __shared__ PackWarp ws[kPackWarps];
    const int nb = list_blocks(a), warp = threadIdx.x >> 5;
    for (int lb = blockIdx.x * kPackWarps + warp; lb < nb; lb += gridDim.x * kPackWarps)
        select_pack_one(a, lb, chunk_block(a, lb), ws[warp], threadIdx.x & 31);
}

// ------------------------------------------------------------ optional encodings
// Encodings the reference never emits, enabled by ASTCB200_FLAG_VOID_EXTENT and
// ASTCB200_FLAG_DUAL_PLANE, applied to a chunk's blocks after the search has written them:
// a block whose texels are all equal becomes an LDR void-extent block; otherwise single-
// partition dual-plane encodings are tried (plane-2 component 0..3, every dual-plane block
// mode on a trial decimation mode) and the best replaces the search's block when its exact
// decoded error is lower.  The search's block is decoded; the
// candidates' texels are computed the way a decoder produces them (integer weight infill,
// endpoints x257, integer interpolation, 16-bit to 8-bit rounding); errors are integer
// weighted squared differences (channel weights x 10^4).  One warp per block; the CPU
// oracle (orc_set_extensions) computes the same choices bit for bit.
//
// A lane tries a block mode.  What its siblings share is made once per plane-2 component (the
// ideal weights of every grid), the infilled weights are kept as 16-bit sums between the endpoints and
// the error, squared differences are summed per channel before they are weighted, the best
// candidate's weights and endpoints are kept by its lane, and the winner is packed by the warp.
// Measured (B200, 65,536 4x4 blocks): 7.0 -> 1.9 ms against decimating per mode, infilling twice and parsing
// the search's block on one lane.
constexpr int kExtWarps = 4;
constexpr int kExtCacheTexels = 64;  // blocks of more texels infill again instead of keeping the sums
__constant__ int c_cwi[4] = {6750, 13275, 2475, 10000};

struct ExtLayout { int c8, w1, w2, sdir, dw, qw, save, sums, total; };  // bytes, per warp
__host__ __device__ inline ExtLayout ext_layout(int T, int ndual_w) {
    ExtLayout f;
    int o = 0;
    auto take = [&](int bytes) { const int r = o; o += (bytes + 15) & ~15; return r; };
    f.c8 = take(T * 4);
    f.w1 = take(T * 4);
    f.w2 = take(T * 4);
    f.sdir = take(16 * 4);
    f.dw = take(2 * ndual_w * 4);
    f.qw = take(32 * 64);    // per lane: two planes of up to 32 grid weights, interleaved by lane
    f.save = take(32 * 64);  // the same of its best candidate
    f.sums = take(T <= kExtCacheTexels ? T * 32 * 4 : 0);
    f.total = o;
    return f;
}

__device__ __forceinline__ int ext_dec8(int v16) { return (int)((((uint32_t)v16 + 128u) * 65281u) >> 24); }  // (v 255 + 32767) / 65535

// Weight i of plane pl of a lane, in the lane-interleaved arrays: words of a plane's four
// consecutive weights, 32 lanes side by side.
__device__ __forceinline__ uint8_t& ext_weight(uint8_t* base, int lane, int pl, int i) { return base[((pl * 8 + (i >> 2)) * 32 + lane) * 4 + (i & 3)]; }

// Sums (weight x contribution x 16) of texel t from both planes' grid weights, the first in the low half.
__device__ __forceinline__ uint32_t ext_sums(const uint8_t* tabs, const TableLayout& L, bool direct, int dmi, uint8_t* qw, int lane, int t) {
    if (direct) return (uint32_t)ext_weight(qw, lane, 0, t) * 16u | (uint32_t)ext_weight(qw, lane, 1, t) * 16u << 16;
    const uint64_t e4 = reinterpret_cast<const uint64_t*>(tabs + L.off_tw4)[(size_t)dmi * L.T + t];
    uint32_t s1 = 0, s2 = 0;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const uint32_t e = (uint32_t)(e4 >> (16 * j)) & 0xFFFF, c = e >> 8;
        const int i = (int)(e & 0xFF);
        s1 += c * ext_weight(qw, lane, 0, i);
        s2 += c * ext_weight(qw, lane, 1, i);
    }
    return s1 | s2 << 16;
}

__global__ void __launch_bounds__(kExtWarps * 32) k_extend(const __grid_constant__ KernelArgs a, int flags) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ dec::fast::Stage<kExtWarps> stage;
    __shared__ PackWarp packs[kExtWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const TableLayout& L = a.L;
    const uint8_t* tabs = a.tables;
    const int T = L.T, bx = L.bx, by = L.by;
    const ExtLayout fl = ext_layout(T, L.ndual_w);
    uint8_t* ws = smem + warp * fl.total;
    uchar4* c8 = reinterpret_cast<uchar4*>(ws + fl.c8);
    float* w1 = reinterpret_cast<float*>(ws + fl.w1);
    float* w2 = reinterpret_cast<float*>(ws + fl.w2);
    float (*S)[4] = reinterpret_cast<float (*)[4]>(ws + fl.sdir);
    float* dw = reinterpret_cast<float*>(ws + fl.dw);  // [2][ndual_w]
    uint8_t* qw = ws + fl.qw;
    uint8_t* save = ws + fl.save;
    uint32_t* sums = reinterpret_cast<uint32_t*>(ws + fl.sums);  // [T][32]
    const bool cached = T <= kExtCacheTexels;
    constexpr unsigned FULL = 0xffffffffu;
    for (int lb = blockIdx.x * kExtWarps + warp; lb < a.nblocks; lb += gridDim.x * kExtWarps) {
        const int blk = chunk_block(a, lb);
        if (blk < 0) continue;
        const BlockSrc src = block_src(a, blk);
        for (int t = lane; t < T; t += 32) c8[t] = src_rgba8(src, bx, t);
        __syncwarp();
        const uchar4 c0 = c8[0];
        bool same = true, opaque = true, const_a = true;
        int sum[4] = {0, 0, 0, 0};
        for (int t = lane; t < T; t += 32) {
            const uchar4 x = c8[t];
            same = same && x.x == c0.x && x.y == c0.y && x.z == c0.z && x.w == c0.w;
            opaque = opaque && x.w == 255;
            const_a = const_a && x.w == c0.w;
            sum[0] += x.x; sum[1] += x.y; sum[2] += x.z; sum[3] += x.w;
        }
        same = __all_sync(FULL, same);
        opaque = __all_sync(FULL, opaque);
        const_a = __all_sync(FULL, const_a);
#pragma unroll
        for (int ch = 0; ch < 4; ch++) sum[ch] = __reduce_add_sync(FULL, sum[ch]);
        uint4* dst = block_dst(a, blk);
        if (same && (flags & 1)) {  // LDR void-extent block of the colour x 257, no extent
            if (lane == 0) {
                *dst = make_uint4(0xFFFFFDFCu, 0xFFFFFFFFu, (uint32_t)c0.x * 0x101u | ((uint32_t)c0.y * 0x101u) << 16,
                                  (uint32_t)c0.z * 0x101u | ((uint32_t)c0.w * 0x101u) << 16);
                if (a.symbolic) {
                    uint32_t* s = a.symbolic + (size_t)blk * 108;
                    for (int i = 0; i < 108; i++) s[i] = 0;
                    s[2] = 1; s[7] = 1; s[12] = c0.x; s[13] = c0.y; s[14] = c0.z; s[15] = c0.w;
                }
            }
            __syncwarp();
            continue;
        }
        if (!(flags & 2)) { __syncwarp(); continue; }
        // exact error of the search's block, decoded
        if (lane == 0) {
            const uint4 v = *dst;
            uint32_t* w = stage.words[warp];
            w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w; w[4] = 0u;
        }
        __syncwarp();
        if (lane < 2) dec::fast::parse_part(stage, dec::fast::g_tables.values, warp, bx, by, lane == 1);
        __syncwarp();
        long long es;
        {
            const uint32_t h = stage.head[warp];
            const int xw = h & 15, yw = (h >> 4) & 15, pc = (h >> 8) & 15, ccs = (h & (1u << 12)) ? (int)(h >> 13) : -1;
            const int ds = (1024 + bx / 2) / (bx - 1), dt = (1024 + by / 2) / (by - 1);
            const int small = T < 31 ? 1 : 0;
            int sq[4] = {0, 0, 0, 0};
            for (int t = lane; t < T; t += 32) {
                const int x = t % bx, y = t / bx;
                const int gs = (ds * x * (xw - 1) + 32) >> 6, gt = (dt * y * (yw - 1) + 32) >> 6, fs = gs & 15, ft = gt & 15;
                const int w11 = (fs * ft + 8) >> 4, w10 = ft - w11, w01 = fs - w11, w00 = 16 - fs - ft + w11;
                const uint8_t* g = stage.w[warp] + (gs >> 4) + (gt >> 4) * xw;
                int wt[2];
#pragma unroll
                for (int p = 0; p < 2; p++) {
                    const uint8_t* gp = g + (ccs >= 0 ? p * dec::fast::kPlane2 : 0);
                    wt[p] = (gp[0] * w00 + gp[1] * w01 + gp[xw] * w10 + gp[xw + 1] * w11 + 8) >> 4;
                }
                const int part = pc > 1 ? dec::fast::texel_partition(stage.seed[warp], stage.offs[warp], pc, (uint32_t)x << small, (uint32_t)y << small) : 0;
                const int4 b = stage.ep[warp][part][0], d = stage.ep[warp][part][1];
                const uchar4 c = c8[t];
                const int d0 = (int)c.x - (int)dec::fast::unorm8((b.x + d.x * wt[ccs == 0]) >> 6), d1 = (int)c.y - (int)dec::fast::unorm8((b.y + d.y * wt[ccs == 1]) >> 6);
                const int d2 = (int)c.z - (int)dec::fast::unorm8((b.z + d.z * wt[ccs == 2]) >> 6), d3 = (int)c.w - (int)dec::fast::unorm8((b.w + d.w * wt[ccs == 3]) >> 6);
                sq[0] += d0 * d0; sq[1] += d1 * d1; sq[2] += d2 * d2; sq[3] += d3 * d3;
            }
            es = 0;
#pragma unroll
            for (int ch = 0; ch < 4; ch++) es += (long long)c_cwi[ch] * __reduce_add_sync(FULL, sq[ch]);
        }
        // dual-plane candidates: plane-2 component outer, block modes inner
        long long best = LLONG_MAX;
        int best_idx = 0x7FFFFFFF;
        uint32_t best_e0 = 0, best_e1 = 0;  // its endpoint bytes
        const int nd = L.ndual;
#pragma unroll 1
        for (int ccs = 0; ccs < 4; ccs++) {
            if (ccs == 3 && const_a) continue;
            float mu[4];
#pragma unroll
            for (int ch = 0; ch < 4; ch++) mu[ch] = (float)sum[ch] / (float)T;
            if (lane < 4 && lane != ccs) {  // positive-deviation sums along axis `lane`, in texel order
                float Sx = 0.0f, Sy = 0.0f, Sz = 0.0f, Sw = 0.0f;
#pragma unroll 1
                for (int t = 0; t < T; t++) {
                    const uchar4 x = c8[t];
                    const float d0 = ccs == 0 ? 0.0f : (float)x.x - mu[0], d1 = ccs == 1 ? 0.0f : (float)x.y - mu[1];
                    const float d2 = ccs == 2 ? 0.0f : (float)x.z - mu[2], d3 = ccs == 3 ? 0.0f : (float)x.w - mu[3];
                    const float dl = lane == 0 ? d0 : lane == 1 ? d1 : lane == 2 ? d2 : d3;
                    if (dl > 0.0f) { Sx = Sx + d0; Sy = Sy + d1; Sz = Sz + d2; Sw = Sw + d3; }
                }
                S[lane][0] = Sx; S[lane][1] = Sy; S[lane][2] = Sz; S[lane][3] = Sw;
            }
            __syncwarp();
            int bax = -1;
            float bl = 0.0f;
            for (int ax = 0; ax < 4; ax++) {
                if (ax == ccs) continue;
                float l = S[ax][0] * S[ax][0];
                l = l + S[ax][1] * S[ax][1];
                l = l + S[ax][2] * S[ax][2];
                l = l + S[ax][3] * S[ax][3];
                if (l > bl) { bl = l; bax = ax; }
            }
            float dir[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            if (bax >= 0) {
                const float len = sqrtf(bl);
#pragma unroll
                for (int ch = 0; ch < 4; ch++) dir[ch] = S[bax][ch] / len;
            }
            float pmin = 1e30f, pmax = -1e30f;
            int vmin = 255, vmax = 0;
            for (int t = lane; t < T; t += 32) {
                const uchar4 x = c8[t];
                const float d0 = ccs == 0 ? 0.0f : (float)x.x - mu[0], d1 = ccs == 1 ? 0.0f : (float)x.y - mu[1];
                const float d2 = ccs == 2 ? 0.0f : (float)x.z - mu[2], d3 = ccs == 3 ? 0.0f : (float)x.w - mu[3];
                float v = d0 * dir[0];
                v = v + d1 * dir[1];
                v = v + d2 * dir[2];
                v = v + d3 * dir[3];
                w1[t] = v;
                pmin = fminf(pmin, v); pmax = fmaxf(pmax, v);
                const int c = ccs == 0 ? x.x : ccs == 1 ? x.y : ccs == 2 ? x.z : x.w;
                vmin = min(vmin, c); vmax = max(vmax, c);
            }
            for (int o = 16; o > 0; o >>= 1) {
                pmin = fminf(pmin, __shfl_xor_sync(FULL, pmin, o)); pmax = fmaxf(pmax, __shfl_xor_sync(FULL, pmax, o));
            }
            vmin = __reduce_min_sync(FULL, vmin); vmax = __reduce_max_sync(FULL, vmax);
            for (int t = lane; t < T; t += 32) {
                const uchar4 x = c8[t];
                const int c = ccs == 0 ? x.x : ccs == 1 ? x.y : ccs == 2 ? x.z : x.w;
                w1[t] = pmax > pmin ? (w1[t] - pmin) / (pmax - pmin) : 0.0f;
                w2[t] = vmax > vmin ? (float)(c - vmin) / (float)(vmax - vmin) : 0.0f;
            }
            __syncwarp();
            // the ideal weights of every dual-plane grid, both planes
#pragma unroll 1
            for (int it = lane; it < L.ndual_w; it += 32) {
                const int e = reinterpret_cast<const uint16_t*>(tabs + L.off_dual_w)[it], m = e >> 6, w = e & 63;
                float v1, v2;
                if (reinterpret_cast<const DevDm*>(tabs + L.off_dm)[m].W == T) {
                    v1 = w1[w]; v2 = w2[w];
                } else {
                    // (the entries' padding adds 0 to sums that are never -0)
                    const uint32_t info = reinterpret_cast<const uint32_t*>(tabs + L.off_wt_info)[m * 64 + w];
                    const uint4* ent = reinterpret_cast<const uint4*>(tabs + L.off_w2tf) + (info & 0xFFFF);
                    float n1 = 0.0f, n2 = 0.0f, den = 0.0f;
#pragma unroll 1
                    for (int n4 = info >> 16; n4 > 0; n4--) {
                        const uint4 q4 = *ent++;
                        const uint32_t q[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
                        for (int k = 0; k < 4; k++) {
                            const float c = __uint_as_float(q[k] & 0xFFFF0000u);
                            const int t = (int)(q[k] & 0xFFFF);
                            n1 = n1 + c * w1[t];
                            n2 = n2 + c * w2[t];
                            den = den + c;
                        }
                    }
                    v1 = n1 / den; v2 = n2 / den;
                }
                dw[it] = fminf(fmaxf(v1, 0.0f), 1.0f);
                dw[L.ndual_w + it] = fminf(fmaxf(v2, 0.0f), 1.0f);
            }
            __syncwarp();
            const bool rgb_only = opaque && ccs != 3;
#pragma unroll 1
            for (int j = lane; j < nd; j += 32) {
                const DevBm bm = reinterpret_cast<const DevBm*>(tabs + L.off_dual)[j];
                const int qc = rgb_only ? bm.colour6 : bm.colour8;
                if (qc == 0) continue;
                const int W = reinterpret_cast<const DevDm*>(tabs + L.off_dm)[bm.dm].W;
                const bool direct = W == T;
                // quantise both planes (pass07's rule over [0, 1])
                {
                    const float* d = dw + reinterpret_cast<const uint16_t*>(tabs + L.off_dual_first)[bm.dm];
                    const uint32_t top = (uint32_t)(c_levels_r[bm.quant] - 1);
                    const float qlm1 = (float)top;
                    const uint8_t* q2u = tabs + L.off_q2u + tabs[L.off_q2u_start + bm.quant];
#pragma unroll 1
                    for (int i = 0; i < W; i++) {
#pragma unroll
                        for (int pl = 0; pl < 2; pl++) {
                            const float ix = d[pl * L.ndual_w + i];
                            const uint32_t wl = __float_as_uint(__fadd_rz(ix * qlm1, 8388608.0f)) - 0x4B000000u, wh = min(wl + 1, top);
                            const uint32_t li = q2u[wl], hi = q2u[wh];
                            ext_weight(qw, lane, pl, i) = (uint8_t)(((float)li + (float)hi) < (128.0f * ix) ? hi : li);
                        }
                    }
                }
                // endpoints per channel: least squares on the channel's plane
                float a1 = 0.0f, b1 = 0.0f, k1 = 0.0f, a2 = 0.0f, b2 = 0.0f, k2 = 0.0f;
                float s0[4] = {0.0f, 0.0f, 0.0f, 0.0f}, s1[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 1
                for (int t = 0; t < T; t++) {
                    const uint32_t ss = ext_sums(tabs, L, direct, bm.dm, qw, lane, t);
                    if (cached) sums[t * 32 + lane] = ss;
                    const float f1 = (float)(((ss & 0xFFFF) + 8) >> 4) / 64.0f;
                    const float f2 = (float)(((ss >> 16) + 8) >> 4) / 64.0f;
                    const float o1 = 1.0f - f1, o2 = 1.0f - f2;
                    a1 = a1 + o1 * o1; b1 = b1 + o1 * f1; k1 = k1 + f1 * f1;
                    a2 = a2 + o2 * o2; b2 = b2 + o2 * f2; k2 = k2 + f2 * f2;
                    const uchar4 x = c8[t];
                    const float xv[4] = {(float)x.x, (float)x.y, (float)x.z, (float)x.w};
#pragma unroll
                    for (int ch = 0; ch < 4; ch++) {
                        const float w = ch == ccs ? f2 : f1, o = ch == ccs ? o2 : o1;
                        s0[ch] = s0[ch] + o * xv[ch];
                        s1[ch] = s1[ch] + w * xv[ch];
                    }
                }
                const uint8_t* cu2u = tabs + L.off_cu2u + (qc - 4) * 512;
                int ue[2][4];
#pragma unroll
                for (int ch = 0; ch < 4; ch++) {
                    const float aa = ch == ccs ? a2 : a1, bb = ch == ccs ? b2 : b1, cc = ch == ccs ? k2 : k1;
                    const float det = aa * cc - bb * bb;
                    float e0, e1;
                    if (det > 0.0001f * (aa * cc)) { e0 = (cc * s0[ch] - bb * s1[ch]) / det; e1 = (aa * s1[ch] - bb * s0[ch]) / det; }
                    else { e0 = e1 = mu[ch]; }
                    e0 = fminf(fmaxf(e0, 0.0f), 255.0f);
                    e1 = fminf(fmaxf(e1, 0.0f), 255.0f);
                    ue[0][ch] = cu2u[(int)rintf(e0) * 2 + 1];
                    ue[1][ch] = cu2u[(int)rintf(e1) * 2 + 1];
                }
                if (rgb_only) { ue[0][3] = 255; ue[1][3] = 255; }
                const bool swapped = ue[1][0] + ue[1][1] + ue[1][2] < ue[0][0] + ue[0][1] + ue[0][2];  // the decoder would swap
                if (swapped) {
#pragma unroll
                    for (int ch = 0; ch < 4; ch++) { const int t = ue[0][ch]; ue[0][ch] = ue[1][ch]; ue[1][ch] = t; }
                }
                int base[4], diff[4], sq[4] = {0, 0, 0, 0};
#pragma unroll
                for (int ch = 0; ch < 4; ch++) { base[ch] = ue[0][ch] * (257 * 64) + 32; diff[ch] = (ue[1][ch] - ue[0][ch]) * 257; }
#pragma unroll 1
                for (int t = 0; t < T; t++) {
                    uint32_t ss = cached ? sums[t * 32 + lane] : ext_sums(tabs, L, direct, bm.dm, qw, lane, t);
                    if (swapped) ss = 0x04000400u - ss;  // of 64 - weight: contributions sum to 16
                    const int v1 = (int)(((ss & 0xFFFF) + 8) >> 4), v2 = (int)(((ss >> 16) + 8) >> 4);
                    const uchar4 x = c8[t];
                    const int xv[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                    for (int ch = 0; ch < 4; ch++) {
                        const int d = xv[ch] - ext_dec8((base[ch] + diff[ch] * (ch == ccs ? v2 : v1)) >> 6);
                        sq[ch] += d * d;
                    }
                }
                long long err = 0;
#pragma unroll
                for (int ch = 0; ch < 4; ch++) err += (long long)c_cwi[ch] * (long long)sq[ch];
                if (err < best) {
                    best = err;
                    best_idx = ccs * nd + j;
                    best_e0 = (uint32_t)ue[0][0] | (uint32_t)ue[0][1] << 8 | (uint32_t)ue[0][2] << 16 | (uint32_t)ue[0][3] << 24;
                    best_e1 = (uint32_t)ue[1][0] | (uint32_t)ue[1][1] << 8 | (uint32_t)ue[1][2] << 16 | (uint32_t)ue[1][3] << 24;
#pragma unroll 1
                    for (int i = 0; i < W; i++)
#pragma unroll
                        for (int pl = 0; pl < 2; pl++) {
                            const int v = ext_weight(qw, lane, pl, i);
                            ext_weight(save, lane, pl, i) = (uint8_t)(swapped ? 64 - v : v);
                        }
                }
            }
            __syncwarp();  // the next plane-2 component overwrites the plane weights
        }
        // the best candidate, the first of equal ones in component and mode order
        long long b = best;
        int bi = best_idx;
        for (int o = 16; o > 0; o >>= 1) {
            const long long ob = __shfl_xor_sync(FULL, b, o);
            const int oi = __shfl_xor_sync(FULL, bi, o);
            if (ob < b || (ob == b && oi < bi)) { b = ob; bi = oi; }
        }
        if (b < es) {  // else the search's block stays
            const int src_lane = __ffs(__ballot_sync(FULL, best == b && best_idx == bi)) - 1;
            const uint32_t e0 = __shfl_sync(FULL, best_e0, src_lane), e1 = __shfl_sync(FULL, best_e1, src_lane);
            const int ccs = bi / nd, j = bi % nd;
            const DevBm bm = reinterpret_cast<const DevBm*>(tabs + L.off_dual)[j];
            const int W = reinterpret_cast<const DevDm*>(tabs + L.off_dm)[bm.dm].W, q = bm.quant;
            const bool rgb_only = opaque && ccs != 3;
            const int nint = rgb_only ? 6 : 8, cem = rgb_only ? 8 : 12, qc = rgb_only ? bm.colour6 : bm.colour8;
            // physical block: interleaved plane weights, mode, partition count, format, plane-2
            // component below the weights, colour values (single partition)
            PackWarp& ps = packs[warp];
            const uint8_t* wscr = tabs + L.off_wscr + q * 32;
            const float top = (float)c_levels_r[q] - 1.0f;
            for (int i = lane; i < 2 * W + 4; i += 32)
                ps.w[i] = i < 2 * W ? wscr[(int)((((float)ext_weight(save, src_lane, i & 1, i >> 1)) / 64.0f) * top + 0.5f)] : 0;
            auto endpoint = [&](int k) { return (((k & 1) ? e1 : e0) >> (8 * (k >> 1))) & 0xFFu; };
            ps.c[lane] = lane < nint ? (tabs + L.off_cscr + (qc - 4) * 256)[endpoint(lane)] : 0;
            __syncwarp();
            uint32_t acc[4] = {0u, 0u, 0u, 0u};
            if (lane == 0) {
                or_bits(acc, bm.mode_index, 0, 11);
                or_bits(acc, (uint32_t)cem, 13, 4);
                or_bits(acc, (uint32_t)ccs, 128 - ise_bits(2 * W, q) - 2, 2);
            }
            const uint4 out = pack_block(a, ps, 2 * W, q, nint, qc, 17, acc, lane);
            if (lane == 0) *dst = out;
            if (a.symbolic) {
                uint32_t* sym = a.symbolic + (size_t)blk * 108;
                for (int i = lane; i < 108; i += 32) {
                    uint32_t v = 0;
                    if (i == 0) v = __float_as_uint((float)b * 1e-4f);
                    else if (i == 1) v = bm.mode_index;
                    else if (i == 2) v = 1;
                    else if (i == 5) v = (uint32_t)qc;
                    else if (i == 6) v = 1u + (uint32_t)ccs;
                    else if (i == 8) v = (uint32_t)cem;
                    else if (i >= 12 && i < 12 + nint) v = endpoint(i - 12);
                    else if (i >= 44 && i < 44 + W) v = ext_weight(save, src_lane, 0, i - 44);
                    else if (i >= 76 && i < 76 + W) v = ext_weight(save, src_lane, 1, i - 76);
                    sym[i] = v;
                }
            }
        }
        __syncwarp();
    }
}

}  // namespace

static size_t extend_smem_bytes(const TableLayout& L) { return (size_t)kExtWarps * ext_layout(L.T, L.ndual_w).total; }

cudaError_t launch_extend(const KernelArgs& a, int flags, cudaStream_t s) {
    if (!(flags & 3)) return cudaSuccess;
    int grid = (a.nblocks + kExtWarps - 1) / kExtWarps;
    if (a.block_list) grid = std::min(grid, kListGridPack);
    if (grid <= 0) return cudaSuccess;
    k_extend<<<grid, kExtWarps * 32, extend_smem_bytes(a.L), s>>>(a, flags);
    return cudaGetLastError();
}

size_t refine_smem_bytes(const TableLayout& L, int topn) {
    return (size_t)refine_layout(L.T, L.max_w, refine_pbs(L.T, topn), refine_u8(L.T), false).total;
}

template <bool U8, bool HELP>
static auto refine_kernel(int cpb) {
    return cpb == 1 ? k_refine<1, U8, HELP> : cpb == 2 ? k_refine<2, U8, HELP> : cpb == 4 ? k_refine<4, U8, HELP> : k_refine<8, U8, HELP>;
}
static auto refine_kernel(int cpb, bool u8, bool help) {
    return u8 ? help ? refine_kernel<true, true>(cpb) : refine_kernel<true, false>(cpb)
              : help ? refine_kernel<false, true>(cpb) : refine_kernel<false, false>(cpb);
}

size_t refine_smem_bytes(const TableLayout& L) {  // the largest over the refinement top-N
    size_t m = 0;
    for (int topn : {1, 2, 4, 8}) m = std::max(m, refine_smem_bytes(L, topn));
    return m;
}

cudaError_t configure_search_kernels(size_t search_bytes, size_t front_bytes);
constexpr int kMaxConfigDevices = 64;

// The dynamic shared-memory limit is a per-function attribute shared by every
// context and thread of the process; it only ever grows (per device), so
// launches for different footprints may be queued concurrently.
cudaError_t configure_kernels(const TableLayout& L) {
    static std::mutex mu;
    static size_t limit[kMaxConfigDevices][4];
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxConfigDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> g(mu);
    size_t* m = limit[dev];
    const size_t need[4] = {search_smem_bytes(L), front_smem_bytes(L), refine_smem_bytes(L), extend_smem_bytes(L)};
    if (need[0] <= m[0] && need[1] <= m[1] && need[2] <= m[2] && need[3] <= m[3]) return cudaSuccess;
    for (int i = 0; i < 4; i++) m[i] = std::max(m[i], need[i]);
    e = configure_search_kernels(m[0], m[1]);
    if (e != cudaSuccess) return e;
    using Kernel = void (*)(KernelArgs);
    Kernel refine[16];
    for (int i = 0; i < 16; i++) refine[i] = refine_kernel(1 << (i & 3), i & 4, i & 8);
    for (Kernel f : refine)
        if ((e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)m[2])) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(k_extend, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)m[3])) != cudaSuccess) return e;
    return cudaFuncSetAttribute(k_refine_tail, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)refine_tail_smem_bytes(kTailMaxTexels, kTailMaxTexels));
}

// A launch over a list, whose length the device knows, queues both instances where it may be either's;
// the one it isn't returns at once (2 us).
cudaError_t launch_refine(const KernelArgs& a, cudaStream_t s, int* launched) {
    const int cpb = refine_cpb(a.topn);
    const int npb = a.nblocks * a.slots;  // of a list: at most
    const size_t smem = refine_smem_bytes(a.L, cpb);
    const bool list = a.block_list || a.pb_list;
    for (int help = 0; help < 2; help++) {
        if ((refine_spread(npb) < 32) != (help != 0) && !(list && help)) continue;
        if (launched) ++*launched;
        const int spread = help ? std::min(refine_spread(npb), 16) : 32, pbs = refine_group(a.L.T, cpb, spread);
        int grid = refine_groups(npb, pbs);
        if (list) grid = std::min(grid, help ? kOneWaveGroups : kListGridRefine);
        refine_kernel(cpb, refine_u8(a.L.T), help != 0)<<<grid, kRefineThreads, smem, s>>>(a);
    }
    return cudaGetLastError();
}

size_t refine_tail_entries(const TableLayout& L, int nblocks) {
    const int npb = nblocks * kSlotsPerBlock, ngroups = refine_groups(npb, refine_group(L.T, refine_cpb(kNumCand), refine_spread(npb)));
    if (L.T > kTailMaxTexels || refine_one_wave(ngroups)) return 0;
    return (size_t)nblocks * (refine_few_waves(refine_u8(L.T), ngroups) ? kTailPerBlockAll : kTailPerBlockFull);
}
size_t refine_tail_entries_up_to(const TableLayout& L, int nblocks) {  // the most blocks of few waves, or all of them
    const int few = 5 * kOneWaveGroups * refine_group(L.T, refine_cpb(kNumCand), 32) / kSlotsPerBlock;
    return std::max(refine_tail_entries(L, nblocks), refine_tail_entries(L, std::min(nblocks, few)));
}

cudaError_t launch_refine_tail(const KernelArgs& a, cudaStream_t s) {
    if (!a.tail || a.L.T > kTailMaxTexels) return cudaSuccess;
    const int grid = std::min((a.tail_cap + kRefineThreads / 4 - 1) / (kRefineThreads / 4), 148 * kTailCtas);
    k_refine_tail<<<std::max(grid, 1), kRefineThreads, refine_tail_smem_bytes(a.L.T, a.L.max_w), s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_select_pack(const KernelArgs& a, cudaStream_t s) {
    int grid = (a.nblocks + kPackWarps - 1) / kPackWarps;
    if (a.block_list) grid = std::min(grid, kListGridPack);
    k_select_pack<<<grid, kPackWarps * 32, 0, s>>>(a);
    return cudaGetLastError();
}

}  // namespace astcb200
