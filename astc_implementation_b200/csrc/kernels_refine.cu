// Refinement and final-selection kernels of the ASTC encoder (sm_100a).
//
//   k_refine       passes 13-17 (shaders/pass13..pass17), six iterations as
//                  driven by compression_pipeline.cpp:473-484: least-squares
//                  endpoints, colour endpoint packing (every LDR encoding the
//                  reference tries), unpacking, weight realignment, final
//                  error with a best-so-far snapshot.  One thread owns one
//                  candidate for all six iterations; the 8 candidates of a
//                  partitioned block share a CTA and its staged texels.
//   k_select_pack  pass18 plus the host argmin over candidates and partition
//                  counts (compression_pipeline.cpp:500-519), then the ASTC
//                  physical block layout (code/physical_compression.cpp:843)
//                  written straight to the 16-byte output block.
#include <cuda_fp16.h>

#include <algorithm>
#include <mutex>
#include <type_traits>

#include "decode_block.cuh"
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
__device__ __forceinline__ I4 ivec(float4 v) { return {f2i(v.x), f2i(v.y), f2i(v.z), f2i(v.w)}; }
__device__ __forceinline__ float4 rnev(float4 v) { return make_float4(rintf(v.x), rintf(v.y), rintf(v.z), rintf(v.w)); }
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
// per issue at 7,500 instructions), so this code and the iteration are written for size: one
// copy of each encoding's body and of the final error, loops left rolled; 4,200 instructions.
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

// Candidate threads per partitioned block (the refinement top-N rounded up to a power of
// two) and partitioned blocks per CTA: 16 x 8 for the full search; more, narrower ones when
// the proposal search keeps fewer candidates, capped so the staged texels stay <= 40 KB.
__host__ __device__ inline int refine_cpb(int topn) { return topn <= 1 ? 1 : topn <= 2 ? 2 : topn <= 4 ? 4 : 8; }
__host__ __device__ inline int refine_pbs(int T, int topn) {
    const int by_threads = kRefineThreads / refine_cpb(topn);
    const int by_smem = 40960 / (T * (T > 16 ? 4 : 16));
    return by_threads < by_smem ? by_threads : (by_smem > 16 ? by_smem : 16);
}

// Candidate state in shared memory, one slot per candidate a CTA runs, arrays of [row][slot]:
// lanes on consecutive slots hit consecutive banks whatever rows they read.  A slot is the
// candidate's rank in its group's initial order, so the first iteration's lanes are on
// consecutive slots and the gathered ones of later iterations on increasing ones.
//   ep   [8]      least-squares endpoints (float4): ep0 and ep1 of partition q in rows 2q, 2q + 1
//   u    [4]      unpacked endpoints of partition q, 0..255 x 257, eight u16: ep0 xyzw, ep1 xyzw
//   s    [T]      infilled weight of each texel times 16, 0..1024, exact in half precision
//   qw   [max_w]  grid weights 0..64
//   err           best error so far
// The infilled weights are kept as sums of grid weight x (contribution x 16), small integers
// that pass16 updates when it moves a weight; every use of one (pass13's weight s / 1024,
// pass16's s / 16, pass17's rounded s / 16) is the exact value the passes' own sums of
// products give, since those sums are exact too.  Before, each texel's four table entries
// and weights were read again at every use (about 45 instructions, two to three uses per
// texel and iteration in pass13 and pass17 and one per texel of each weight in pass16).
// Measured with pass13's walk in partition order (B200): full search of 1024x1024 at 4x4 50.2 -> 47.5 ms,
// of 64x64 1.08 -> 0.90 ms; proposal search of 2047x2050 at 6x6 8.98 -> 8.13 ms.
constexpr int kSlotRow16 = kRefineThreads * 16;  // bytes of a row of 16-byte elements
constexpr int kSlotRow4 = kRefineThreads * 4;    // of two s or four qw
struct RefineLayout {
    int ep, u, s, qw, err, item, pos, px, part, sdir, keys, aux, total;
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
    f.u = take(4 * kSlotRow16);
    f.s = take((T + 1) / 2 * kSlotRow4);
    f.qw = take((max_w + 3) / 4 * kSlotRow4);
    f.err = take(kRefineThreads * 4);
    f.item = take(kRefineThreads * 4);
    f.pos = take(kRefineThreads);
    f.px = take(rows * px_row_bytes(T, u8));
    f.part = take(rows * part_row_bytes(T, u8 && !tail ? 2 : 1));
    f.sdir = take(tail ? 0 : rows * 64);
    f.keys = take(kRefineThreads * 4);
    f.aux = take(tail ? kRefineThreads * 4 : rows * 4);
    f.total = o;
    return f;
}
struct Cand {  // one slot of the arrays above
    uint8_t *epb, *ub, *sb, *qb;
    float* err;
    __device__ Cand(uint8_t* sm, const RefineLayout& f, int slot)
        : epb(sm + f.ep + slot * 16), ub(sm + f.u + slot * 16), sb(sm + f.s + slot * 4), qb(sm + f.qw + slot * 4),
          err(reinterpret_cast<float*>(sm + f.err) + slot) {}
    __device__ __forceinline__ float4& ep(int i) const { return *reinterpret_cast<float4*>(epb + i * kSlotRow16); }
    __device__ __forceinline__ uint4& u(int q) const { return *reinterpret_cast<uint4*>(ub + q * kSlotRow16); }
    __device__ __forceinline__ __half& s(int t) const { return *reinterpret_cast<__half*>(sb + (t >> 1) * kSlotRow4 + (t & 1) * 2); }
    __device__ __forceinline__ uint8_t& qw(int w) const { return qb[(w >> 2) * kSlotRow4 + (w & 3)]; }
    __device__ __forceinline__ uint32_t& qw4(int i) const { return *reinterpret_cast<uint32_t*>(qb + i * kSlotRow4); }
};
// The u16 in the low (hi = false) or high half of v as a float: 2^23 + v has v as its low bits.
__device__ __forceinline__ float u16f(uint32_t v, bool hi) { return __uint_as_float(__byte_perm(v, 0x4B000000u, hi ? 0x7632 : 0x7610)) - 8388608.0f; }
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
template <class Row, class Part, class SDir>
__device__ bool refine_step(const KernelArgs& a, const PBRec& rec, const int P, int k, const Row px, const Part pt, const SDir sdir_of,
                            const Cand cs, Snap* snap, const int it) {
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
    if (it == 0) {
#pragma unroll
        for (int q = 0; q < 4; q++) { cs.ep(2 * q) = rec.ep0[q]; cs.ep(2 * q + 1) = rec.ep1[q]; }
        const uint32_t* src = reinterpret_cast<const uint32_t*>(ci.qw);  // 8-byte aligned in PBRec
#pragma unroll 1
        for (int w = 0; w < (W + 3) / 4; w++) cs.qw4(w) = src[w];
        *cs.err = ERR_DEFAULT;
        infill(tb, cs, bm.dm, T, direct);
    }
    uint32_t ffmt[4] = {0, 0, 0, 0}, matched = 0, final_q = ci.ql;

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
                const uint4 u = cs.u(p);
                base = make_float4(u16f(u.x, false), u16f(u.x, true), u16f(u.y, false), u16f(u.y, true));
                offs = (make_float4(u16f(u.z, false), u16f(u.z, true), u16f(u.w, false), u16f(u.w, true)) - base) * (1.0f / 64.0f);
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
        if (total < *cs.err) {  // the best so far (ERR_DEFAULT at first)
            *cs.err = total;
            uint4* d = reinterpret_cast<uint4*>(snap);  // 16-byte aligned: 112-byte records
            d[0] = make_uint4(__float_as_uint(total), (uint32_t)ci.bm | final_q << 16 | matched << 24,
                              ffmt[0] | ffmt[1] << 8 | ffmt[2] << 16 | ffmt[3] << 24, 0u);
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
    int i0 = 0;  // the partition's first texel in partition order
#pragma unroll 1
    for (int q = 0; q < P; q++) {
        const int n = P == 1 ? T : tb.part_count(P, rec.entry, q);
        const float ps = (float)n;
        // the scale direction and its sums are only read by the formats with a scale
        const bool scale = ci.fmt[q] == FMT_RGB_SCALE || ci.fmt[q] == FMT_RGB_SCALE_ALPHA;
        const float4 sdir = scale ? sdir_of(q, ps) : mk(0.0f);
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
        bool all_same = ci.ql != ci.qlm;
        uint32_t fn[4] = {0, 0, 0, 0};
#pragma unroll
        for (int q = 0; q < 4; q++) packed[q] = make_uint2(0u, 0u);
#pragma unroll 1
        for (int q = 0; q < P; q++) {
            const uint4 v = Packer::pack(cu2u, cs.ep(2 * q), cs.ep(2 * q + 1), rgbs[q], ci.fmt[q], ci.ql);
            const uint32_t f = v.x;
            fn[0] = q == 0 ? f : fn[0]; fn[1] = q == 1 ? f : fn[1]; fn[2] = q == 2 ? f : fn[2]; fn[3] = q == 3 ? f : fn[3];
            packed[q] = make_uint2(v.y, v.z);
            if (q > 0) all_same = all_same && f == fn[0];
        }
        bool m = false;
        if (P >= 2 && all_same) {
            uint32_t fm[4] = {0, 0, 0, 0};
            bool same_mod = true;
#pragma unroll 1
            for (int q = 0; q < P; q++) {
                const uint4 v = Packer::pack(cu2u, cs.ep(2 * q), cs.ep(2 * q + 1), rgbs[q], ci.fmt[q], ci.qlm);
                const uint32_t f = v.x;
                fm[0] = q == 0 ? f : fm[0]; fm[1] = q == 1 ? f : fm[1]; fm[2] = q == 2 ? f : fm[2]; fm[3] = q == 3 ? f : fm[3];
                packed_mod[q] = make_uint2(v.y, v.z);
                if (q > 0 && f != fm[0]) { same_mod = false; break; }
            }
            if (same_mod) {
                m = true;
#pragma unroll
                for (int q = 0; q < 4; q++) fn[q] = fm[q];
#pragma unroll 1
                for (int q = 0; q < P; q++) packed[q] = packed_mod[q];
            }
        }
        matched = m ? 1 : 0;
        final_q = m ? ci.qlm : ci.ql;
#pragma unroll
        for (int q = 0; q < 4; q++) ffmt[q] = fn[q];
    }
    // ---------------- pass15
#pragma unroll 1
    for (int q = 0; q < P; q++) {
        I4 o0, o1;
        unpack_endpoints(q == 0 ? ffmt[0] : q == 1 ? ffmt[1] : q == 2 ? ffmt[2] : ffmt[3], packed[q].x, packed[q].y, o0, o1);
        cs.u(q) = make_uint4((uint32_t)(o0.x * 257) | (uint32_t)(o0.y * 257) << 16, (uint32_t)(o0.z * 257) | (uint32_t)(o0.w * 257) << 16,
                             (uint32_t)(o1.x * 257) | (uint32_t)(o1.y * 257) << 16, (uint32_t)(o1.z * 257) | (uint32_t)(o1.w * 257) << 16);
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
        const uint4 u = cs.u(p);
        base = make_float4(u16f(u.x, false), u16f(u.x, true), u16f(u.y, false), u16f(u.y, true));
        offs = (make_float4(u16f(u.z, false), u16f(u.z, true), u16f(u.w, false), u16f(u.w, true)) - base) * (1.0f / 64.0f);
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
// next iteration, the best error so far, then the state an iteration carries over (endpoints,
// weights; the best result so far is in the candidate's snapshot already).
__device__ __forceinline__ void write_tail(const KernelArgs& a, const Cand& c, uint32_t pbi, int k, int it, int pos) {
    uint4* e = a.tail + (size_t)pos * kTailWords;
    e[0] = make_uint4(pbi, (uint32_t)k | (uint32_t)it << 8, __float_as_uint(*c.err), 0u);
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
// U8: texels staged as RGBA8 (refine_u8).
template <int CPB, bool U8>
__global__ void __launch_bounds__(kRefineThreads, kRefineCtas) k_refine(const __grid_constant__ KernelArgs a) {
    extern __shared__ __align__(16) uint8_t smem[];
    const int T = a.L.T;
    constexpr int cpb = CPB;
    const int pbs = CPB == 8 ? kRefineThreads / 8 : refine_pbs(T, CPB);
    const RefineLayout fl = refine_layout(T, a.L.max_w, pbs, U8, false);
    using Px = typename std::conditional<U8, uchar4, float4>::type;
    using Pe = typename std::conditional<U8, uint16_t, uint8_t>::type;
    const int px_row = px_row_bytes(T, U8), part_row = part_row_bytes(T, sizeof(Pe));
    uint32_t* item_of = reinterpret_cast<uint32_t*>(smem + fl.item);  // by slot: lb * slots + slot
    uint8_t* pos_of = smem + fl.pos;                                  // by slot: staging position
    uint32_t* staged = reinterpret_cast<uint32_t*>(smem + fl.aux);    // by staged partitioned block: lb + 1 | slot << 27, 0 if none
    float4* sdirs = reinterpret_cast<float4*>(smem + fl.sdir);
    int* keys = reinterpret_cast<int*>(smem + fl.keys);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // Items: every slot of every block in slot-major order (consecutive CTAs hold
    // partitioned blocks of the same slot, hence the same partition count, so
    // co-resident warps run the same code), or the proposal pass's work list.
    const int nb = list_blocks(a);
    const int npb = a.pb_list ? pb_total(a) : nb * a.slots;
    const int ngroups = (npb + pbs - 1) / pbs;
    const int iters = a.refine_iters > 0 ? a.refine_iters : 6;
    __shared__ unsigned int refined[4];  // candidates refined by this CTA, by P (work counters)
    __shared__ int live_in_warp[kRefineThreads / 32];
    __shared__ int spill_base;
    if (tid < 4) refined[tid] = 0;
    bool spill = a.tail != nullptr && T <= kTailMaxTexels;  // until the tail is found full
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
                    key = ((((int)r.P - 1) << 12 | fk) << 7) | dm;  // partition count, formats, decimation mode
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
#pragma unroll 1
                    for (int q = k; q < P; q += cpb) sdirs[pbl * 4 + q] = scale_dir(r.avg[q], (float)(P == 1 ? T : (int)counts[q]));
                }
            }
            keys[tid] = key * kRefineThreads + tid;  // unique keys: P, formats, decimation mode, then position
            if (k == 0 && pbl < pbs) staged[pbl] = item;
        }
        __syncthreads();
        // Thread tid takes the candidate of rank tid in (partition count, endpoint formats,
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
            __syncthreads();
            keys[rank] = tid;
            __syncthreads();
            const int mine = keys[tid];
            const int pbl = mine / cpb, k = mine % cpb;
            const uint32_t item = pbl < pbs ? staged[pbl] : 0u;
            if (item != 0) {
                const int lb = (int)(item & 0x07FFFFFFu) - 1, slot = (int)(item >> 27);
                const size_t pbi = (size_t)lb * a.slots + slot;
                a.snaps[pbi * kNumCand + k].err = ERR_DEFAULT;  // inert slot unless refined below
                if (k < (int)a.pbrec[pbi].ncand) {
                    cand = tid;
                    item_of[tid] = (uint32_t)pbi;
                    pos_of[tid] = (uint8_t)mine;
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
            __syncthreads();  // also: every thread has read keys[] before it is rewritten
            int nlive = 0, before = 0;
#pragma unroll
            for (int w = 0; w < kRefineThreads / 32; w++) {
                const int n = live_in_warp[w];
                nlive += n;
                before += w < warp ? n : 0;
            }
            if (nlive == 0) break;
            const int rank = before + __popc(bal & ((1u << lane) - 1u));
            if (spill && it > 0 && nlive <= a.spill_live) {
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
                    if (live) write_tail(a, Cand(smem, fl, cand), item_of[cand], pos_of[cand] % cpb, it, pos);
                    break;
                }
                if (live && pos < a.tail_cap) a.tail[(size_t)pos * kTailWords].x = 0xFFFFFFFFu;  // reserved, left empty
                spill = false;  // the tail is full: finish here
            }
            if (live) keys[rank] = cand;
            __syncthreads();
            cand = tid < nlive ? keys[tid] : -1;
            if (cand >= 0) {
                const int pbl = pos_of[cand] / cpb, k = pos_of[cand] % cpb;
                const size_t pbi = item_of[cand];
                const PBRec& rec = a.pbrec[pbi];
                Snap* snap = &a.snaps[pbi * kNumCand + k];
                const TexelRow<U8> row{reinterpret_cast<const Px*>(smem + fl.px + pbl * px_row)};
                const PartRow<Pe> part{reinterpret_cast<Pe*>(smem + fl.part + pbl * part_row)};
                const float4* sd = sdirs + pbl * 4;
                const bool moved = refine_step(a, rec, (int)rec.P, k, row, part, [&](int q, float) { return sd[q]; }, Cand(smem, fl, cand), snap, it);
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
    int* keys = reinterpret_cast<int*>(smem + fl.keys);
    int* next_it = reinterpret_cast<int*>(smem + fl.aux);             // by slot
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
        if (!dry && nlive <= kTailRefillAt) {
            // Thread tid stages into slot tid when that slot is free and its warp's claim
            // reached an entry for it.
            const bool fr = busy[tid] == 0;
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
                    *c.err = __uint_as_float(h.z);
                    const RTabs tb{a.tables, &a.L};
                    const int dm = tb.bm(r.c[k].bm).dm;
                    infill(tb, c, dm, T, tb.dm(dm).W == T);
                    k_of[tid] = (uint8_t)k;
                    next_it[tid] = (int)((h.y >> 8) & 0xFF);
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
        if (live) keys[before + __popc(bal & below)] = cand;
        if (filled >= 0) keys[nlive + new_before + __popc(bnew & below)] = filled;
        __syncthreads();
        cand = tid < n ? keys[tid] : -1;
        if (cand >= 0) {
            const uint32_t pbi = pbi_of[cand];
            const int k = (int)k_of[cand], it = next_it[cand];
            const PBRec& rec = a.pbrec[pbi];
            Snap* snap = &a.snaps[(size_t)pbi * kNumCand + k];
            const TexelRow<true> row{reinterpret_cast<const uchar4*>(smem + fl.px + cand * px_row)};
            const PartRow<uint8_t> part{smem + fl.part + cand * part_row};
            const bool moved = refine_step(a, rec, (int)rec.P, k, row, part, [&](int q, float ps) { return scale_dir(rec.avg[q], ps); },
                                           Cand(smem, fl, cand), snap, it);
            next_it[cand] = it + 1;
            if (!moved || it + 1 >= iters) {
                busy[cand] = 0;  // released: read by the next refill, after the next barrier
                cand = -1;
            }
        }
    }
}

size_t refine_tail_smem_bytes(int T, int max_w) { return (size_t)refine_layout(T, max_w, kRefineThreads, true, true).total; }

// ------------------------------------------------------------ k_select_pack
__device__ __forceinline__ void write_bits(uint32_t value, uint32_t count, uint32_t off, uint8_t* p) {
    uint32_t mask = (1u << count) - 1;
    value &= mask;
    p += off >> 3;
    off &= 7;
    value <<= off; mask <<= off; mask = ~mask;
    p[0] &= mask; p[0] |= value;
    p[1] &= mask >> 8; p[1] |= value >> 8;
}

__device__ void btq(int q, int& bits, int& trits, int& quints) {
    int L = c_levels_r[q];
    trits = quints = 0;
    if (L % 3 == 0) { trits = 1; L /= 3; } else if (L % 5 == 0) { quints = 1; L /= 5; }
    bits = 0;
    while ((1 << bits) < L) bits++;
}
__device__ uint32_t ise_bits(uint32_t n, int q) {
    int b, t, qu; btq(q, b, t, qu);
    if (t) return (n * (8 + 5 * b) + 4) / 5;
    if (qu) return (n * (7 + 3 * b) + 2) / 3;
    return n * b;
}

// encode_ise (code/physical_compression.cpp:672-826); out has 2 spare bytes.
__device__ void encode_ise(const TableLayout& L, const uint8_t* tabs, int q, uint32_t n, const uint8_t* in, uint8_t* out, uint32_t off) {
    int bits, trits, quints; btq(q, bits, trits, quints);
    const uint32_t mask = (1u << bits) - 1;
    const uint8_t* tt = tabs + L.off_trits;
    const uint8_t* qt = tabs + L.off_quints;
    if (trits) {
        const uint8_t tb[5] = {2, 2, 1, 2, 1}, ts[5] = {0, 2, 4, 5, 7};
        for (uint32_t i = 0; i < n; i += 5) {
            uint32_t d[5];
            for (int e = 0; e < 5; e++) d[e] = i + e < n ? (uint32_t)(in[i + e] >> bits) : 0;
            const uint32_t T = tt[(((d[4] * 3 + d[3]) * 3 + d[2]) * 3 + d[1]) * 3 + d[0]];
            for (int e = 0; e < 5 && i + e < n; e++) {
                const uint32_t pack = (in[i + e] & mask) | (((T >> ts[e]) & ((1u << tb[e]) - 1)) << bits);
                write_bits(pack, bits + tb[e], off, out);
                off += bits + tb[e];
            }
        }
    } else if (quints) {
        const uint8_t qb[3] = {3, 2, 2}, qs[3] = {0, 3, 5};
        for (uint32_t i = 0; i < n; i += 3) {
            uint32_t d[3];
            for (int e = 0; e < 3; e++) d[e] = i + e < n ? (uint32_t)(in[i + e] >> bits) : 0;
            const uint32_t Q = qt[(d[2] * 5 + d[1]) * 5 + d[0]];
            for (int e = 0; e < 3 && i + e < n; e++) {
                const uint32_t pack = (in[i + e] & mask) | (((Q >> qs[e]) & ((1u << qb[e]) - 1)) << bits);
                write_bits(pack, bits + qb[e], off, out);
                off += bits + qb[e];
            }
        }
    } else {
        for (uint32_t i = 0; i < n; i++) { write_bits(in[i], bits, off, out); off += bits; }
    }
}

__device__ __forceinline__ int bitrev8(int p) {
    p = ((p & 0x0F) << 4) | ((p >> 4) & 0x0F);
    p = ((p & 0x33) << 2) | ((p >> 2) & 0x33);
    p = ((p & 0x55) << 1) | ((p >> 1) & 0x55);
    return p;
}

__device__ __noinline__ void select_pack_one(const KernelArgs& a, int lb, int blk) {
    float best = 1e30f;
    int win_slot = -1, win_k = 0;
    // slots the front filled: all of them, or P=1 (unless skipped) plus the proposed partitionings
    const int nslots = a.prop ? 1 + (int)a.prop[lb].n : a.slots;
    const int s0 = a.prop && (a.prop[lb].flags & 1) ? 1 : 0;
    for (int s = s0; s < nslots; s++) {
        const PBRec& r = a.pbrec[(size_t)lb * a.slots + s];
        const int n = r.ncand;
        for (int k = 0; k < n; k++) {
            const float e = a.snaps[((size_t)lb * a.slots + s) * kNumCand + k].err;
            if (e < best) { best = e; win_slot = s; win_k = k; }
        }
    }
    if (win_slot < 0 && a.reroute_list) {  // proposal search found nothing: hand the block to the full search
        const int pos = atomicAdd(a.reroute_count, 1);
        a.reroute_list[pos] = blk;
        a.reroute_err[pos] = 3e38f;
        return;
    }
    if (a.prev_err && !(best < a.prev_err[lb])) return;  // the proposal search's result stands
    if (a.reroute_list && a.reroute_above > 0.0f && best > a.reroute_above) {
        // a poor proposal-search result: write it, and let the full search try to beat it
        const int pos = atomicAdd(a.reroute_count, 1);
        a.reroute_list[pos] = blk;
        a.reroute_err[pos] = best;
    }
    uint8_t blockbytes[18];
    uint32_t sym[8 + 4 + 32];  // header words of the SymbolicBlock record
    for (int i = 0; i < 18; i++) blockbytes[i] = 0;
    for (int i = 0; i < 44; i++) sym[i] = 0;
    const Snap* sn = nullptr;
    const PBRec* rec = nullptr;
    if (win_slot >= 0) {
        rec = &a.pbrec[(size_t)lb * a.slots + win_slot];
        sn = &a.snaps[((size_t)lb * a.slots + win_slot) * kNumCand + win_k];
        const DevBm bm = reinterpret_cast<const DevBm*>(a.tables + a.L.off_bm)[sn->bm];
        const DevDm dm = reinterpret_cast<const DevDm*>(a.tables + a.L.off_dm)[bm.dm];
        const uint32_t pc = rec->P, q = bm.quant;
        sym[0] = __float_as_uint(best); sym[1] = bm.mode_index; sym[2] = pc; sym[3] = rec->seed;
        sym[4] = sn->matched; sym[5] = sn->final_q;
        for (int i = 0; i < 4; i++) sym[8 + i] = sn->ffmt[i];
        for (int i = 0; i < 32; i++) sym[12 + i] = sn->packed[i];
        // weights: requantise 0..64 to the ISE alphabet, scramble, encode, bit-reverse
        const uint8_t* wscr = a.tables + a.L.off_wscr + q * 32;
        const float levels = (float)c_levels_r[q];
        uint8_t wv[64], wbuf[18];
        for (int i = 0; i < 18; i++) wbuf[i] = 0;
        for (int i = 0; i < dm.W; i++) {
            const float uqw = (float)sn->qw[i];
            const float qw = (uqw / 64.0f) * (levels - 1.0f);
            wv[i] = wscr[(int)(qw + 0.5f)];
        }
        const uint32_t wbits = ise_bits(dm.W, (int)q);
        encode_ise(a.L, a.tables, (int)q, dm.W, wv, wbuf, 0);
        for (int i = 0; i < 16; i++) blockbytes[i] = (uint8_t)bitrev8(wbuf[15 - i]);
        write_bits(bm.mode_index, 11, 0, blockbytes);
        write_bits(pc - 1, 2, 11, blockbytes);
        if (pc > 1) {
            write_bits(rec->seed, 6, 13, blockbytes);
            write_bits(rec->seed >> 6, 4, 19, blockbytes);
            if (sn->matched) {
                write_bits((uint32_t)sn->ffmt[0] << 2, 6, 23, blockbytes);
            } else {
                int low = 4;
                for (uint32_t i = 0; i < pc; i++) low = min((int)(sn->ffmt[i] >> 2), low);
                if (low == 3) low = 2;
                int et = low + 1, bp = 2;
                for (uint32_t i = 0; i < pc; i++) { et |= ((int)(sn->ffmt[i] >> 2) - low) << bp; bp++; }
                for (uint32_t i = 0; i < pc; i++) { et |= (int)(sn->ffmt[i] & 3) << bp; bp += 2; }
                const int hs = 3 * (int)pc - 4;
                write_bits(et & 0x3F, 6, 23, blockbytes);
                write_bits((uint32_t)et >> 6, hs, 128 - wbits - hs, blockbytes);
            }
        } else {
            write_bits(sn->ffmt[0], 4, 13, blockbytes);
        }
        const uint8_t* cscr = a.tables + a.L.off_cscr + (sn->final_q - 4) * 256;
        uint8_t vals[32];
        int nv = 0;
        for (uint32_t i = 0; i < pc; i++) {
            const int n = 2 * (sn->ffmt[i] >> 2) + 2;
            for (int j = 0; j < n; j++) vals[nv + j] = cscr[sn->packed[i * 8 + j]];
            nv += n;
        }
        encode_ise(a.L, a.tables, sn->final_q, nv, vals, blockbytes, pc == 1 ? 17 : 29);
    }
    uint4 o;
    o.x = blockbytes[0] | (blockbytes[1] << 8) | (blockbytes[2] << 16) | ((uint32_t)blockbytes[3] << 24);
    o.y = blockbytes[4] | (blockbytes[5] << 8) | (blockbytes[6] << 16) | ((uint32_t)blockbytes[7] << 24);
    o.z = blockbytes[8] | (blockbytes[9] << 8) | (blockbytes[10] << 16) | ((uint32_t)blockbytes[11] << 24);
    o.w = blockbytes[12] | (blockbytes[13] << 8) | (blockbytes[14] << 16) | ((uint32_t)blockbytes[15] << 24);
    *block_dst(a, blk) = o;
    if (a.symbolic) {
        uint32_t* s = a.symbolic + (size_t)blk * 108;
        if (win_slot < 0) sym[0] = __float_as_uint(1e30f);
        for (int i = 0; i < 44; i++) s[i] = sym[i];
        for (int i = 0; i < 64; i++) s[44 + i] = sn ? sn->qw[i] : 0;
    }
}

__global__ void __launch_bounds__(128) k_select_pack(const __grid_constant__ KernelArgs a) {
    const int nb = list_blocks(a);
    for (int lb = blockIdx.x * blockDim.x + threadIdx.x; lb < nb; lb += gridDim.x * blockDim.x)
        select_pack_one(a, lb, chunk_block(a, lb));
}

}  // namespace

namespace {

// ------------------------------------------------------------ optional encodings
// Encodings the reference never emits, enabled by ASTCB200_FLAG_VOID_EXTENT and
// ASTCB200_FLAG_DUAL_PLANE, applied to a chunk's blocks after the search has written them:
// a block whose texels are all equal becomes an LDR void-extent block; otherwise single-
// partition dual-plane encodings are tried (plane-2 component 0..3, every dual-plane block
// mode on a trial decimation mode) and the best replaces the search's block when its exact
// decoded error is lower.  The search's block is decoded with the library's decoder; the
// candidates' texels are computed the way a decoder produces them (integer weight infill,
// endpoints x257, integer interpolation, 16-bit to 8-bit rounding); errors are integer
// weighted squared differences (channel weights x 10^4).  One warp per block; the CPU
// oracle (orc_set_extensions) computes the same choices bit for bit.
constexpr int kExtWarps = 4;
__constant__ int c_cwi[4] = {6750, 13275, 2475, 10000};

struct ExtWarp {
    uchar4 c8[kMaxTexels];
    float w1[kMaxTexels], w2[kMaxTexels];
    float S[4][4];
    dec::Block kb;
    uint8_t qw[32][2][32];  // per lane: two planes of up to 32 grid weights
};

__device__ __forceinline__ int ext_dec8(int v16) { return (int)(((uint32_t)v16 * 255u + 32767u) / 65535u); }
__device__ __forceinline__ int ext_lerp(int e0, int e1, int w) { return (e0 * (64 - w) + e1 * w + 32) >> 6; }

// Integer infill of texel t from 0..64 grid weights (the specification's weights / 16).
__device__ __forceinline__ int ext_infill(const uint8_t* tabs, const TableLayout& L, int W, int dmi, const uint8_t* qw, int t) {
    if (W == L.T) return qw[t];
    const uint64_t e4 = reinterpret_cast<const uint64_t*>(tabs + L.off_tw4)[(size_t)dmi * L.T + t];
    int s = 0;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const uint32_t e = (uint32_t)(e4 >> (16 * j)) & 0xFFFF;
        s += (int)(e >> 8) * (int)qw[e & 0xFF];
    }
    return (s + 8) >> 4;
}

// Dual-plane candidate (ccs, dual mode j) from the warp's plane weights: its exact error
// (LLONG_MAX when no colour quant fits), and with phys != nullptr its block and symbolic words.
__device__ __noinline__ long long dual_candidate(const KernelArgs& a, const ExtWarp& ws, int ccs, int j, bool calpha,
                                                 const int* sum, uint8_t (*qw)[32], uint8_t* phys, uint32_t* sym) {
    const uint8_t* tabs = a.tables;
    const TableLayout& L = a.L;
    const int T = L.T;
    const DevBm bm = reinterpret_cast<const DevBm*>(tabs + L.off_dual)[j];
    const DevDm dm = reinterpret_cast<const DevDm*>(tabs + L.off_dm)[bm.dm];
    const int W = dm.W;
    const bool rgb_only = calpha && ccs != 3;
    const int nint = rgb_only ? 6 : 8, cem = rgb_only ? 8 : 12;
    const int avail = 109 - (int)bm.weight_bits;
    int qc = -1;
    for (int q = 20; q >= 4; q--)
        if ((int)ise_bits(nint, q) <= avail) { qc = q; break; }
    if (qc < 0) return LLONG_MAX;
    // decimate and quantise both planes (pass07's rule over [0, 1])
    const float qlm1 = (float)(c_levels_r[bm.quant] - 1);
    const uint8_t* q2u = tabs + L.off_q2u;
    const int qoff = tabs[L.off_q2u_start + bm.quant];
    for (int pl = 0; pl < 2; pl++) {
        const float* wv = pl ? ws.w2 : ws.w1;
        for (int i = 0; i < W; i++) {
            float dw;
            if (W == T) dw = wv[i];
            else {
                float num = 0.0f, den = 0.0f;
                const int n = tabs[L.off_wt_count + bm.dm * 64 + i];
                const int base = dm.wt_base + reinterpret_cast<const uint16_t*>(tabs + L.off_wt_start)[bm.dm * 64 + i];
                for (int k = 0; k < n; k++) {
                    const uint32_t e = reinterpret_cast<const uint16_t*>(tabs + L.off_w2t)[base + k];
                    const float c = (float)(e >> 8) * (1.0f / 16.0f);
                    num = num + c * wv[e & 0xFF];
                    den = den + c;
                }
                dw = num / den;
            }
            const float ix = fminf(fmaxf(dw, 0.0f), 1.0f), ix1 = ix * qlm1;
            const uint32_t wl = f2u(ix1), wh = min(wl + 1, f2u(qlm1));
            const uint32_t li = q2u[qoff + wl], hi = q2u[qoff + wh];
            qw[pl][i] = (uint8_t)(((float)li + (float)hi) < (128.0f * ix) ? hi : li);
        }
    }
    // endpoints per channel: least squares on the channel's plane
    float a1 = 0.0f, b1 = 0.0f, k1 = 0.0f, a2 = 0.0f, b2 = 0.0f, k2 = 0.0f;
    float s0[4] = {0.0f, 0.0f, 0.0f, 0.0f}, s1[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    for (int t = 0; t < T; t++) {
        const float w1 = (float)ext_infill(tabs, L, W, bm.dm, qw[0], t) / 64.0f;
        const float w2 = (float)ext_infill(tabs, L, W, bm.dm, qw[1], t) / 64.0f;
        const float o1 = 1.0f - w1, o2 = 1.0f - w2;
        a1 = a1 + o1 * o1; b1 = b1 + o1 * w1; k1 = k1 + w1 * w1;
        a2 = a2 + o2 * o2; b2 = b2 + o2 * w2; k2 = k2 + w2 * w2;
        const uchar4 x = ws.c8[t];
        const float xv[4] = {(float)x.x, (float)x.y, (float)x.z, (float)x.w};
#pragma unroll
        for (int ch = 0; ch < 4; ch++) {
            const float w = ch == ccs ? w2 : w1, o = ch == ccs ? o2 : o1;
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
        else { e0 = e1 = (float)sum[ch] / (float)T; }
        e0 = fminf(fmaxf(e0, 0.0f), 255.0f);
        e1 = fminf(fmaxf(e1, 0.0f), 255.0f);
        ue[0][ch] = cu2u[(int)rintf(e0) * 2 + 1];
        ue[1][ch] = cu2u[(int)rintf(e1) * 2 + 1];
    }
    if (rgb_only) { ue[0][3] = 255; ue[1][3] = 255; }
    if (ue[1][0] + ue[1][1] + ue[1][2] < ue[0][0] + ue[0][1] + ue[0][2]) {  // the decoder would swap
#pragma unroll
        for (int ch = 0; ch < 4; ch++) { const int t = ue[0][ch]; ue[0][ch] = ue[1][ch]; ue[1][ch] = t; }
        for (int pl = 0; pl < 2; pl++)
            for (int i = 0; i < W; i++) qw[pl][i] = (uint8_t)(64 - qw[pl][i]);
    }
    long long err = 0;
    for (int t = 0; t < T; t++) {
        const int w1 = ext_infill(tabs, L, W, bm.dm, qw[0], t), w2 = ext_infill(tabs, L, W, bm.dm, qw[1], t);
        const uchar4 x = ws.c8[t];
        const int xv[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int ch = 0; ch < 4; ch++) {
            const int d = xv[ch] - ext_dec8(ext_lerp(ue[0][ch] * 257, ue[1][ch] * 257, ch == ccs ? w2 : w1));
            err += (long long)c_cwi[ch] * (long long)(d * d);
        }
    }
    if (phys) {
        for (int i = 0; i < 108; i++) sym[i] = 0;
        sym[0] = __float_as_uint((float)err * 1e-4f);
        sym[1] = bm.mode_index; sym[2] = 1; sym[5] = (uint32_t)qc; sym[6] = 1u + (uint32_t)ccs; sym[8] = (uint32_t)cem;
        for (int ch = 0; ch < nint / 2; ch++) { sym[12 + 2 * ch] = (uint32_t)ue[0][ch]; sym[13 + 2 * ch] = (uint32_t)ue[1][ch]; }
        for (int i = 0; i < W; i++) { sym[44 + i] = qw[0][i]; sym[76 + i] = qw[1][i]; }
        // physical block: interleaved plane weights, mode, partition count, format, plane-2
        // component below the weights, colour values (single partition)
        const int q = bm.quant;
        const uint8_t* wscr = tabs + L.off_wscr + q * 32;
        const float levels = (float)c_levels_r[q];
        uint8_t wv[64], wbuf[18];
        for (int i = 0; i < 18; i++) wbuf[i] = 0;
        for (int i = 0; i < W; i++) {
            wv[2 * i] = wscr[(int)((((float)qw[0][i]) / 64.0f) * (levels - 1.0f) + 0.5f)];
            wv[2 * i + 1] = wscr[(int)((((float)qw[1][i]) / 64.0f) * (levels - 1.0f) + 0.5f)];
        }
        const uint32_t wbits = ise_bits(2 * W, q);
        encode_ise(L, tabs, q, 2 * W, wv, wbuf, 0);
        for (int i = 0; i < 16; i++) phys[i] = (uint8_t)bitrev8(wbuf[15 - i]);
        write_bits(bm.mode_index, 11, 0, phys);
        write_bits(0, 2, 11, phys);
        write_bits((uint32_t)cem, 4, 13, phys);
        write_bits((uint32_t)ccs, 2, 128 - wbits - 2, phys);
        const uint8_t* cscr = tabs + L.off_cscr + (qc - 4) * 256;
        uint8_t vals[8];
        for (int k = 0; k < nint; k++) vals[k] = cscr[sym[12 + k]];
        encode_ise(L, tabs, qc, nint, vals, phys, 17);
    }
    return err;
}

__global__ void __launch_bounds__(kExtWarps * 32) k_extend(const __grid_constant__ KernelArgs a, int flags) {
    __shared__ ExtWarp wsm[kExtWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    ExtWarp& ws = wsm[warp];
    const int T = a.L.T, bx = a.L.bx, by = a.L.by;
    constexpr unsigned FULL = 0xffffffffu;
    for (int lb = blockIdx.x * kExtWarps + warp; lb < a.nblocks; lb += gridDim.x * kExtWarps) {
        const int blk = chunk_block(a, lb);
        if (blk < 0) continue;
        const BlockSrc src = block_src(a, blk);
        for (int t = lane; t < T; t += 32) ws.c8[t] = src_rgba8(src, bx, t);
        __syncwarp();
        const uchar4 c0 = ws.c8[0];
        bool same = true, opaque = true, const_a = true;
        int sum[4] = {0, 0, 0, 0};
        for (int t = lane; t < T; t += 32) {
            const uchar4 x = ws.c8[t];
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
            uint8_t raw[16];
            const uint32_t wv4[4] = {v.x, v.y, v.z, v.w};
            for (int i = 0; i < 16; i++) raw[i] = (uint8_t)(wv4[i >> 2] >> (8 * (i & 3)));
            dec::parse_block(raw, bx, by, ws.kb);
        }
        __syncwarp();
        long long es = 0;
        for (int t = lane; t < T; t += 32) {
            uint16_t v16[4];
            dec::texel16(ws.kb, bx, by, t % bx, t / bx, v16);
            const uchar4 x = ws.c8[t];
            const int xv[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int ch = 0; ch < 4; ch++) {
                const int d = xv[ch] - (int)dec::to_unorm8(v16[ch]);
                es += (long long)c_cwi[ch] * (long long)(d * d);
            }
        }
        for (int o = 16; o > 0; o >>= 1) es += __shfl_xor_sync(FULL, es, o);
        // dual-plane candidates: plane-2 component outer, block modes inner
        long long best = LLONG_MAX;
        int best_idx = 0x7FFFFFFF;
        const int nd = a.L.ndual;
        for (int pass = 0; pass < 2; pass++) {
            int ccs_lo = 0, ccs_hi = 3, win_ccs = -1, win_j = -1;
            if (pass == 1) {  // the winner's plane weights again, then its encoding
                long long b = best;
                int bi = best_idx;
                for (int o = 16; o > 0; o >>= 1) {
                    const long long ob = __shfl_xor_sync(FULL, b, o);
                    const int oi = __shfl_xor_sync(FULL, bi, o);
                    if (ob < b || (ob == b && oi < bi)) { b = ob; bi = oi; }
                }
                if (!(b < es)) break;  // the search's block stays
                win_ccs = bi / nd; win_j = bi % nd;
                ccs_lo = ccs_hi = win_ccs;
            }
            for (int ccs = ccs_lo; ccs <= ccs_hi; ccs++) {
                if (ccs == 3 && const_a) continue;
                float mu[4];
#pragma unroll
                for (int ch = 0; ch < 4; ch++) mu[ch] = (float)sum[ch] / (float)T;
                if (lane < 4 && lane != ccs) {  // positive-deviation sums along axis `lane`, in texel order
                    float Sx = 0.0f, Sy = 0.0f, Sz = 0.0f, Sw = 0.0f;
                    for (int t = 0; t < T; t++) {
                        const uchar4 x = ws.c8[t];
                        const float d0 = ccs == 0 ? 0.0f : (float)x.x - mu[0], d1 = ccs == 1 ? 0.0f : (float)x.y - mu[1];
                        const float d2 = ccs == 2 ? 0.0f : (float)x.z - mu[2], d3 = ccs == 3 ? 0.0f : (float)x.w - mu[3];
                        const float dl = lane == 0 ? d0 : lane == 1 ? d1 : lane == 2 ? d2 : d3;
                        if (dl > 0.0f) { Sx = Sx + d0; Sy = Sy + d1; Sz = Sz + d2; Sw = Sw + d3; }
                    }
                    ws.S[lane][0] = Sx; ws.S[lane][1] = Sy; ws.S[lane][2] = Sz; ws.S[lane][3] = Sw;
                }
                __syncwarp();
                int bax = -1;
                float bl = 0.0f;
                for (int ax = 0; ax < 4; ax++) {
                    if (ax == ccs) continue;
                    float l = ws.S[ax][0] * ws.S[ax][0];
                    l = l + ws.S[ax][1] * ws.S[ax][1];
                    l = l + ws.S[ax][2] * ws.S[ax][2];
                    l = l + ws.S[ax][3] * ws.S[ax][3];
                    if (l > bl) { bl = l; bax = ax; }
                }
                float dir[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                if (bax >= 0) {
                    const float len = sqrtf(bl);
#pragma unroll
                    for (int ch = 0; ch < 4; ch++) dir[ch] = ws.S[bax][ch] / len;
                }
                float pmin = 1e30f, pmax = -1e30f;
                int vmin = 255, vmax = 0;
                for (int t = lane; t < T; t += 32) {
                    const uchar4 x = ws.c8[t];
                    const float d0 = ccs == 0 ? 0.0f : (float)x.x - mu[0], d1 = ccs == 1 ? 0.0f : (float)x.y - mu[1];
                    const float d2 = ccs == 2 ? 0.0f : (float)x.z - mu[2], d3 = ccs == 3 ? 0.0f : (float)x.w - mu[3];
                    float v = d0 * dir[0];
                    v = v + d1 * dir[1];
                    v = v + d2 * dir[2];
                    v = v + d3 * dir[3];
                    ws.w1[t] = v;
                    pmin = fminf(pmin, v); pmax = fmaxf(pmax, v);
                    const int c = ccs == 0 ? x.x : ccs == 1 ? x.y : ccs == 2 ? x.z : x.w;
                    vmin = min(vmin, c); vmax = max(vmax, c);
                }
                for (int o = 16; o > 0; o >>= 1) {
                    pmin = fminf(pmin, __shfl_xor_sync(FULL, pmin, o)); pmax = fmaxf(pmax, __shfl_xor_sync(FULL, pmax, o));
                    vmin = min(vmin, __shfl_xor_sync(FULL, vmin, o)); vmax = max(vmax, __shfl_xor_sync(FULL, vmax, o));
                }
                for (int t = lane; t < T; t += 32) {
                    const uchar4 x = ws.c8[t];
                    const int c = ccs == 0 ? x.x : ccs == 1 ? x.y : ccs == 2 ? x.z : x.w;
                    ws.w1[t] = pmax > pmin ? (ws.w1[t] - pmin) / (pmax - pmin) : 0.0f;
                    ws.w2[t] = vmax > vmin ? (float)(c - vmin) / (float)(vmax - vmin) : 0.0f;
                }
                __syncwarp();
                if (pass == 0) {
                    for (int j = lane; j < nd; j += 32) {
                        const long long e = dual_candidate(a, ws, ccs, j, opaque, sum, ws.qw[lane], nullptr, nullptr);
                        if (e < best) { best = e; best_idx = ccs * nd + j; }
                    }
                } else if (lane == 0) {
                    uint8_t phys[18];
                    uint32_t sym[108];
                    for (int i = 0; i < 18; i++) phys[i] = 0;
                    dual_candidate(a, ws, win_ccs, win_j, opaque, sum, ws.qw[0], phys, sym);
                    *dst = make_uint4(phys[0] | (phys[1] << 8) | (phys[2] << 16) | ((uint32_t)phys[3] << 24),
                                      phys[4] | (phys[5] << 8) | (phys[6] << 16) | ((uint32_t)phys[7] << 24),
                                      phys[8] | (phys[9] << 8) | (phys[10] << 16) | ((uint32_t)phys[11] << 24),
                                      phys[12] | (phys[13] << 8) | (phys[14] << 16) | ((uint32_t)phys[15] << 24));
                    if (a.symbolic) {
                        uint32_t* s = a.symbolic + (size_t)blk * 108;
                        for (int i = 0; i < 108; i++) s[i] = sym[i];
                    }
                }
                __syncwarp();  // the next plane-2 component overwrites the plane weights
            }
        }
        __syncwarp();
    }
}

}  // namespace

cudaError_t launch_extend(const KernelArgs& a, int flags, cudaStream_t s) {
    if (!(flags & 3)) return cudaSuccess;
    int grid = (a.nblocks + kExtWarps - 1) / kExtWarps;
    if (a.block_list) grid = std::min(grid, kListGridPack);
    if (grid <= 0) return cudaSuccess;
    k_extend<<<grid, kExtWarps * 32, 0, s>>>(a, flags);
    return cudaGetLastError();
}

size_t refine_smem_bytes(const TableLayout& L, int topn) {
    return (size_t)refine_layout(L.T, L.max_w, refine_pbs(L.T, topn), refine_u8(L.T), false).total;
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
    static size_t limit[kMaxConfigDevices][3];
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxConfigDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> g(mu);
    size_t* m = limit[dev];
    const size_t need[3] = {search_smem_bytes(L), front_smem_bytes(L), refine_smem_bytes(L)};
    if (need[0] <= m[0] && need[1] <= m[1] && need[2] <= m[2]) return cudaSuccess;
    for (int i = 0; i < 3; i++) m[i] = std::max(m[i], need[i]);
    e = configure_search_kernels(m[0], m[1]);
    if (e != cudaSuccess) return e;
    for (auto f : {k_refine<1, false>, k_refine<2, false>, k_refine<4, false>, k_refine<8, false>, k_refine<1, true>,
                   k_refine<2, true>, k_refine<4, true>, k_refine<8, true>})
        if ((e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)m[2])) != cudaSuccess) return e;
    return cudaFuncSetAttribute(k_refine_tail, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)refine_tail_smem_bytes(kTailMaxTexels, kTailMaxTexels));
}

cudaError_t launch_refine(const KernelArgs& a, cudaStream_t s) {
    const int cpb = refine_cpb(a.topn);
    const int npb = a.nblocks * a.slots, pbs = refine_pbs(a.L.T, cpb);
    int grid = (npb + pbs - 1) / pbs;
    if (a.block_list) grid = std::min(grid, kListGridRefine);
    const size_t smem = refine_smem_bytes(a.L, cpb);
    if (refine_u8(a.L.T)) {
        if (cpb == 1) k_refine<1, true><<<grid, kRefineThreads, smem, s>>>(a);
        else if (cpb == 2) k_refine<2, true><<<grid, kRefineThreads, smem, s>>>(a);
        else if (cpb == 4) k_refine<4, true><<<grid, kRefineThreads, smem, s>>>(a);
        else k_refine<8, true><<<grid, kRefineThreads, smem, s>>>(a);
    } else {
        if (cpb == 1) k_refine<1, false><<<grid, kRefineThreads, smem, s>>>(a);
        else if (cpb == 2) k_refine<2, false><<<grid, kRefineThreads, smem, s>>>(a);
        else if (cpb == 4) k_refine<4, false><<<grid, kRefineThreads, smem, s>>>(a);
        else k_refine<8, false><<<grid, kRefineThreads, smem, s>>>(a);
    }
    return cudaGetLastError();
}

cudaError_t launch_refine_tail(const KernelArgs& a, cudaStream_t s) {
    if (!a.tail || a.L.T > kTailMaxTexels) return cudaSuccess;
    const int grid = std::min((a.tail_cap + kRefineThreads - 1) / kRefineThreads, 148 * kTailCtas);
    k_refine_tail<<<std::max(grid, 1), kRefineThreads, refine_tail_smem_bytes(a.L.T, a.L.max_w), s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_select_pack(const KernelArgs& a, cudaStream_t s) {
    int grid = (a.nblocks + 127) / 128;
    if (a.block_list) grid = std::min(grid, kListGridPack);
    k_select_pack<<<grid, 128, 0, s>>>(a);
    return cudaGetLastError();
}

}  // namespace astcb200
