// ASTC LDR decoding on the GPU (no counterpart in the reference, which has no decoder):
// the same texels as the host decoder (decode_block.cuh) for every 128-bit pattern, for
// quality measurement and round-trip checks of large textures without copying them back to
// the host.
//
// k_decode: one CTA of 128 threads per 64 blocks of a block row (of several rows, for images
// narrower than that).  First two threads of different warps parse each block into shared
// memory, one its weights, one its endpoints and partition seeds; then each thread evaluates
// columns of texels, consecutive threads taking consecutive columns, so that a row of the CTA's
// texels is stored as whole lines, and either writes the RGBA8 image or adds up the squared
// error per channel against a reference image (warp reduction, then one 64-bit atomic
// per channel and warp).
//
// The least a decode can move is the blocks and the image (75 MB at 4096x4096 6x6: 11 us), but
// the kernel is bound by its integer instructions: parsing reads a group of sequence-encoded
// values with one funnel shift, decodes trits, quints and unquantises by table, and a texel
// channel is one multiply-add, a shift and a multiply for the rounding to 8 bits.  One thread a
// block with bit-by-bit reads and a texel per thread with its block's set-up repeated, which
// this replaces, took 463 us a call there; this takes 90 us.
#include <cstddef>

#include <cuda_runtime.h>

#include "astcb200.h"
#include "decode_block.cuh"
#include "tables.h"

namespace astcb200 {
namespace {

constexpr int kDecodeThreads = 128;
constexpr int kDecodeBlocks = 64;  // per CTA
constexpr int kWeightRow = 100;    // bytes of a block's weights: planes 48 apart, zeros past the grid; an odd number of words
constexpr int kPlane2 = 48;

// Digits of packed trits (2 bits each) and quints (3 bits each), unquantised weights and
// colours by value, bits | trits << 4 | quints << 5 of the quantisation methods, bits of n
// weights, and the finest colour method of n values in b bits (0: none an LDR block may use),
// all from the decoder's own functions at compile time.
struct DecodeTables {
    uint16_t trits[256], quints[128];
    uint8_t weight[12][32];
    uint8_t colour[17][256];
    uint8_t method[24];
    uint16_t weight_bits[65][12];
    uint8_t colour_method[19][128];
};
constexpr DecodeTables make_tables() {
    DecodeTables t{};
    for (int i = 0; i < 256; i++) {
        int d[5] = {0, 0, 0, 0, 0};
        dec::trit_digits(i, d);
        for (int e = 0; e < 5; e++) t.trits[i] = (uint16_t)(t.trits[i] | d[e] << (2 * e));
    }
    for (int i = 0; i < 128; i++) {
        int d[3] = {0, 0, 0};
        dec::quint_digits(i, d);
        for (int e = 0; e < 3; e++) t.quints[i] = (uint16_t)(t.quints[i] | d[e] << (3 * e));
    }
    int ise[65][21] = {};
    for (int q = 0; q < 21; q++) {
        int b = 0, tr = 0, qu = 0;
        dec::btq(q, b, tr, qu);
        t.method[q] = (uint8_t)(b | tr << 4 | qu << 5);
        for (int n = 0; n <= 64; n++) {
            ise[n][q] = dec::ise_bits(n, q);
            if (q < 12) t.weight_bits[n][q] = (uint16_t)ise[n][q];
        }
        for (int v = 0; v < dec::level_count(q); v++) {
            if (q < 12) t.weight[q][v] = (uint8_t)dec::unq_weight(q, v);
            if (q >= 4) t.colour[q - 4][v] = (uint8_t)dec::unq_color(q, v);
        }
    }
    for (int n = 0; n < 19; n++)
        for (int b = 0; b < 128; b++)
            for (int q = 4; q < 21; q++)
                if (ise[n][q] <= b) t.colour_method[n][b] = (uint8_t)q;
    return t;
}
__device__ const DecodeTables g_tables = make_tables();
constexpr int kSharedTables = sizeof(DecodeTables::trits) + sizeof(DecodeTables::quints) + sizeof(DecodeTables::weight);

constexpr int kWords = 5;      // the block's four words and one of 0: an odd stride
constexpr int kColourRow = 28;  // bytes of a block's colour values: 18, and 8 read past any endpoint's first
struct Shared {
    int4 ep[kDecodeBlocks][4][2];      // per partition: 64 x 257 e0 + 32 + 128 x 64, and 257 (e1 - e0), per channel
    uint32_t words[kDecodeBlocks][kWords];
    uint32_t head[kDecodeBlocks];      // grid width | height << 4 | partitions << 8 | dual << 12 | plane-2 channel << 13
    uint32_t seed[kDecodeBlocks], offs[kDecodeBlocks];  // partition hash: eight 4-bit factors; four 6-bit offsets
    uint8_t w[kDecodeBlocks][kWeightRow];
    uint8_t cv[kDecodeBlocks][kColourRow];
    uint16_t trits[256], quints[128];
    uint8_t weight[12][32];
};

static_assert(offsetof(DecodeTables, weight) == 768 && offsetof(Shared, weight) - offsetof(Shared, trits) == 768 &&
              offsetof(Shared, trits) % 4 == 0, "the tables are copied as words");

// n bits (0..31) at bit `off` of the block, off below 128.
__device__ __forceinline__ uint32_t bits_at(const uint32_t* w, int off, int n) {
    return __funnelshift_r(w[off >> 5], w[(off >> 5) + 1], off & 31) & ((1u << n) - 1u);
}
// The same of the block read backwards (bit i is the block's bit 127 - i).
__device__ __forceinline__ uint32_t bits_back(const uint32_t* w, int off, int n) {
    const int j = 3 - (off >> 5);
    return __funnelshift_r(__brev(w[j]), j > 0 ? __brev(w[j - 1]) : 0u, off & 31) & ((1u << n) - 1u);
}

// Unquantised weights of a block of grid m, zeros after them.
__device__ __forceinline__ void parse_weights(Shared& s, int k, const dec::Mode& m) {
    const uint32_t* w = s.words[k];
    uint8_t* out = s.w[k];
    const int W = m.xw * m.yw, np = m.dual ? 2 : 1, n = W * np;
    const uint32_t method = g_tables.method[m.q];
    const int bits = method & 15;
    const uint32_t mask = (1u << bits) - 1u;
    const uint8_t* unq = s.weight[m.q];
    const int end = g_tables.weight_bits[n][m.q];
    auto put = [&](int i, uint32_t v) { out[m.dual ? (i >> 1) + (i & 1) * kPlane2 : i] = unq[v]; };
    int off = 0;
    // groups of at most 23 bits; the bits of values past the end read as 0
    if (method & 16) {
#pragma unroll 1
        for (int i = 0; i < n; i += 5) {
            uint32_t g = bits_back(w, off, min(5 * bits + 8, end - off)), v[5], T = 0;
            off += 5 * bits + 8;
#pragma unroll
            for (int e = 0; e < 5; e++) {
                const int tb = (e == 2 || e == 4) ? 1 : 2, sh = e == 0 ? 0 : e == 1 ? 2 : e == 2 ? 4 : e == 3 ? 5 : 7;
                v[e] = g & mask;
                T |= ((g >> bits) & ((1u << tb) - 1u)) << sh;
                g >>= bits + tb;
            }
            const uint32_t d = s.trits[T];
#pragma unroll
            for (int e = 0; e < 5; e++)
                if (i + e < n) put(i + e, ((d >> (2 * e)) & 3u) << bits | v[e]);
        }
    } else if (method & 32) {
#pragma unroll 1
        for (int i = 0; i < n; i += 3) {
            uint32_t g = bits_back(w, off, min(3 * bits + 7, end - off)), v[3], Q = 0;
            off += 3 * bits + 7;
#pragma unroll
            for (int e = 0; e < 3; e++) {
                const int qb = e == 0 ? 3 : 2, sh = e == 0 ? 0 : e == 1 ? 3 : 5;
                v[e] = g & mask;
                Q |= ((g >> bits) & ((1u << qb) - 1u)) << sh;
                g >>= bits + qb;
            }
            const uint32_t d = s.quints[Q];
#pragma unroll
            for (int e = 0; e < 3; e++)
                if (i + e < n) put(i + e, ((d >> (3 * e)) & 7u) << bits | v[e]);
        }
    } else {
#pragma unroll 1
        for (int i = 0; i < n; i += 4) {
            const uint32_t g = bits_back(w, off, min(4 * bits, end - off));
            off += 4 * bits;
#pragma unroll
            for (int e = 0; e < 4; e++)
                if (i + e < n) put(i + e, (g >> (e * bits)) & mask);
        }
    }
#pragma unroll 1
    for (int i = W; i <= W + m.xw; i++) { out[i] = 0; if (m.dual) out[i + kPlane2] = 0; }  // the grid's far edges read them with factor 0
}

// nv colour values of method q (4..20) from bit `off` on, unquantised.
__device__ __forceinline__ void parse_colours(Shared& s, int k, int off, int nv, int q) {
    const uint32_t* w = s.words[k];
    uint8_t* out = s.cv[k];
    const uint32_t method = g_tables.method[q];
    const int bits = method & 15;
    const uint32_t mask = (1u << bits) - 1u;
    const uint8_t* unq = g_tables.colour[q - 4];
    if (method & 16) {
#pragma unroll 1
        for (int i = 0; i < nv; i += 5) {
            uint32_t T = 0, v[5];
#pragma unroll
            for (int e = 0; e < 5; e++) {
                const int tb = (e == 2 || e == 4) ? 1 : 2, sh = e == 0 ? 0 : e == 1 ? 2 : e == 2 ? 4 : e == 3 ? 5 : 7;
                const uint32_t g = i + e < nv ? bits_at(w, off, bits + tb) : 0u;
                off += bits + tb;
                v[e] = g & mask;
                T |= (g >> bits) << sh;
            }
            const uint32_t d = s.trits[T];
#pragma unroll
            for (int e = 0; e < 5; e++)
                if (i + e < nv) out[i + e] = unq[((d >> (2 * e)) & 3u) << bits | v[e]];
        }
    } else if (method & 32) {
#pragma unroll 1
        for (int i = 0; i < nv; i += 3) {
            uint32_t Q = 0, v[3];
#pragma unroll
            for (int e = 0; e < 3; e++) {
                const int qb = e == 0 ? 3 : 2, sh = e == 0 ? 0 : e == 1 ? 3 : 5;
                const uint32_t g = i + e < nv ? bits_at(w, off, bits + qb) : 0u;
                off += bits + qb;
                v[e] = g & mask;
                Q |= (g >> bits) << sh;
            }
            const uint32_t d = s.quints[Q];
#pragma unroll
            for (int e = 0; e < 3; e++)
                if (i + e < nv) out[i + e] = unq[((d >> (3 * e)) & 7u) << bits | v[e]];
        }
    } else {
#pragma unroll 1
        for (int i = 0; i < nv; i++, off += bits) out[i] = unq[bits_at(w, off, bits)];
    }
}

// A block of one colour (16 bits a channel): its endpoints' sums, no difference.
__device__ __forceinline__ void constant_block(Shared& s, int k, int c0, int c1, int c2, int c3) {
    s.head[k] = 2u | 2u << 4 | 1u << 8;
    const int add = 32 + 128 * 64;
    s.ep[k][0][0] = make_int4(c0 * 64 + add, c1 * 64 + add, c2 * 64 + add, c3 * 64 + add);
    s.ep[k][0][1] = make_int4(0, 0, 0, 0);
}

// Header, endpoints and partition hash of block k; weights: the weights instead.
__device__ __forceinline__ void parse_part(Shared& s, int k, int bx, int by, bool weights) {
    const uint32_t* w = s.words[k];
    const int mode = (int)bits_at(w, 0, 11);
    if ((mode & 0x1FF) == 0x1FC) {  // void extent
        if (weights) return;
        if (mode & 0x200) constant_block(s, k, 0xFFFF, 0, 0xFFFF, 0xFFFF);  // HDR
        else constant_block(s, k, (int)(w[2] & 0xFFFF), (int)(w[2] >> 16), (int)(w[3] & 0xFFFF), (int)(w[3] >> 16));
        return;
    }
    dec::Mode m{};
    bool ok = dec::decode_grid(mode, m);
    const int nw = m.xw * m.yw * (m.dual ? 2 : 1);
    int wbits = 0;
    if (ok) {
        wbits = nw <= 64 ? (int)g_tables.weight_bits[nw][m.q] : 0;
        ok = wbits >= 24 && wbits <= 96 && m.xw <= bx && m.yw <= by;
    }
    const int pc = (int)bits_at(w, 11, 2) + 1;
    ok = ok && !(pc == 4 && m.dual);
    if (weights) {
        if (ok) parse_weights(s, k, m);
        return;
    }
    uint32_t cems = 0;  // four bits a partition
    int seed = 0, below = 128 - wbits, cstart = 17, nv = 0, ccs = 0;
    if (ok) {
        if (pc == 1) {
            cems = bits_at(w, 13, 4);
        } else {
            seed = (int)bits_at(w, 13, 10);
            cstart = 29;
            const int low = (int)bits_at(w, 23, 6);
            if ((low & 3) == 0) {
                cems = (uint32_t)(low >> 2) * 0x1111u;
            } else {
                const int hs = 3 * pc - 4;
                below -= hs;
                const int et = low | ((int)bits_at(w, below, hs) << 6);
                const int base = (et & 3) - 1;
#pragma unroll
                for (int i = 0; i < 4; i++)
                    if (i < pc) cems |= (uint32_t)(((base + ((et >> (2 + i)) & 1)) << 2) | ((et >> (2 + pc + 2 * i)) & 3)) << (4 * i);
            }
        }
        if (m.dual) { below -= 2; ccs = (int)bits_at(w, below, 2); }
#pragma unroll
        for (int i = 0; i < 4; i++)
            if (i < pc) nv += 2 * (int)((cems >> (4 * i + 2)) & 3u) + 2;
        ok = nv <= 18;
    }
    int cq = 0;
    if (ok) {
        const int avail = below - cstart;
        cq = avail > 0 ? (int)g_tables.colour_method[nv][avail] : 0;
        ok = cq >= 4;
    }
    if (ok) {
        parse_colours(s, k, cstart, nv, cq);
        int vo = 0;
#pragma unroll 1
        for (int i = 0; i < pc; i++) {
            const int cem = (int)((cems >> (4 * i)) & 15u);
            int v[8], e0[4] = {}, e1[4] = {};
#pragma unroll
            for (int j = 0; j < 8; j++) v[j] = s.cv[k][vo + j];
            if (!dec::decode_endpoints(cem, v, e0, e1)) { ok = false; break; }
            const int add = 32 + 128 * 64;
            // (endpoint bytes, as the host decoder keeps them)
#pragma unroll
            for (int c = 0; c < 4; c++) { e0[c] &= 0xFF; e1[c] &= 0xFF; }
            s.ep[k][i][0] = make_int4(e0[0] * (257 * 64) + add, e0[1] * (257 * 64) + add, e0[2] * (257 * 64) + add, e0[3] * (257 * 64) + add);
            s.ep[k][i][1] = make_int4((e1[0] - e0[0]) * 257, (e1[1] - e0[1]) * 257, (e1[2] - e0[2]) * 257, (e1[3] - e0[3]) * 257);
            vo += 2 * (cem >> 2) + 2;
        }
    }
    if (!ok) {
        constant_block(s, k, 0xFFFF, 0, 0xFFFF, 0xFFFF);
        return;
    }
    s.head[k] = (uint32_t)m.xw | (uint32_t)m.yw << 4 | (uint32_t)pc << 8 | (m.dual ? 1u << 12 : 0u) | (uint32_t)ccs << 13;
    if (pc > 1) {  // the factors and offsets of the specification's partition hash (select_partition)
        const int sd = seed + (pc - 1) * 1024;
        const uint32_t r = dec::hash52((uint32_t)sd);
        int sh1, sh2;
        if (sd & 1) { sh1 = (sd & 2) ? 4 : 5; sh2 = pc == 3 ? 6 : 5; } else { sh1 = pc == 3 ? 6 : 5; sh2 = (sd & 2) ? 4 : 5; }
        uint32_t f = 0;
#pragma unroll
        for (int i = 0; i < 8; i++) { const uint32_t v = (r >> (4 * i)) & 0xF; f |= ((v * v) >> ((i & 1) ? sh2 : sh1)) << (4 * i); }
        s.seed[k] = f;
        s.offs[k] = ((r >> 14) & 63u) | ((r >> 10) & 63u) << 6 | ((r >> 6) & 63u) << 12 | ((r >> 2) & 63u) << 18;
    }
}

// v / 257 rounded as the host decoder's to_unorm8 rounds v * 255 / 65535, of v + 128 (below 2^16 + 128).
__device__ __forceinline__ uint32_t unorm8(int v128) { return ((uint32_t)v128 * 65281u) >> 24; }

// CTAs in raster order of groups of kDecodeBlocks blocks: cols blocks wide, kDecodeBlocks / cols block rows high.
template <bool kError>
__global__ void __launch_bounds__(kDecodeThreads) k_decode(const uint8_t* __restrict__ blocks, int bx, int by, int dx, int dy,
                                                            int nbx, int nby, int cols, int groups_x, uchar4* __restrict__ out,
                                                            const uchar4* __restrict__ ref, unsigned long long* __restrict__ sse) {
    __shared__ __align__(16) Shared s;
    const int tid = threadIdx.x;
    const int rows = kDecodeBlocks / cols;
    const int gx = (int)(blockIdx.x % (unsigned)groups_x) * cols, gy = (int)(blockIdx.x / (unsigned)groups_x) * rows;
    {
        const uint32_t* src = reinterpret_cast<const uint32_t*>(g_tables.trits);
        uint32_t* dst = reinterpret_cast<uint32_t*>(s.trits);  // trits, quints and weights: contiguous on both sides
        for (int i = tid; i < kSharedTables / 4; i += kDecodeThreads) dst[i] = src[i];
    }
    for (int i = tid; i < kDecodeBlocks * kWords; i += kDecodeThreads) {
        const int k = i / kWords, j = i % kWords, kx = gx + k % cols, ky = gy + k / cols;
        uint32_t v = 0;
        if (j < 4 && kx < nbx && ky < nby && k < rows * cols) {
            const uint8_t* src = blocks + ((size_t)ky * nbx + kx) * 16 + 4 * j;
            if (((uintptr_t)blocks & 3) == 0) v = *reinterpret_cast<const uint32_t*>(src);
            else v = src[0] | src[1] << 8 | src[2] << 16 | (uint32_t)src[3] << 24;  // any alignment is accepted
        }
        s.words[k][j] = v;
    }
    __syncthreads();
    {
        const int k = tid % kDecodeBlocks;
        if (k < rows * cols) parse_part(s, k, bx, by, tid >= kDecodeBlocks);
    }
    __syncthreads();
    unsigned long long acc[4] = {0, 0, 0, 0};
    const int ds = (1024 + bx / 2) / (bx - 1), dt = (1024 + by / 2) / (by - 1);
    const int small = bx * by < 31 ? 1 : 0;
    const uint32_t per_bx = 0xFFFFFFFFu / (uint32_t)bx + 1u, per_cols = 0xFFFFFFFFu / (uint32_t)cols + 1u;
    for (int col = tid; col < rows * cols * bx; col += kDecodeThreads) {
        const int k = (int)__umulhi((uint32_t)col, per_bx), x = col - k * bx;
        const int kr = cols == 1 ? k : (int)__umulhi((uint32_t)k, per_cols), kx = gx + k - kr * cols;
        const int px = kx * bx + x, py0 = (gy + kr) * by;
        if (kx >= nbx || px >= dx || py0 >= dy) continue;
        const uint32_t h = s.head[k];
        const int xw = h & 15, yw = (h >> 4) & 15, pc = (h >> 8) & 15;
        const int gs = (ds * x * (xw - 1) + 32) >> 6, fs = gs & 15, gt1 = dt * (yw - 1);
        const uint8_t* w = s.w[k] + (gs >> 4);
        int4 b = s.ep[k][0][0], d = s.ep[k][0][1];
        const uint32_t f = s.seed[k], o = s.offs[k];
        const int xs = x << small;
        const int ny = min(by, dy - py0);
        const size_t at0 = (size_t)py0 * dx + px;
#pragma unroll 1
        for (int y = 0; y < ny; y++) {
            const int gt = (gt1 * y + 32) >> 6, ft = gt & 15;
            const int w11 = (fs * ft + 8) >> 4, w10 = ft - w11, w01 = fs - w11, w00 = 16 - fs - ft + w11;
            const uint8_t* g = w + (gt >> 4) * xw;
            const int wt = (g[0] * w00 + g[1] * w01 + g[xw] * w10 + g[xw + 1] * w11 + 8) >> 4;
            if (pc > 1) {
                const uint32_t ys = (uint32_t)y << small, ux = (uint32_t)xs;
                const uint32_t a = ((f & 15u) * ux + ((f >> 4) & 15u) * ys + o) & 63u;
                const uint32_t q = (((f >> 8) & 15u) * ux + ((f >> 12) & 15u) * ys + (o >> 6)) & 63u;
                const uint32_t c = pc > 2 ? (((f >> 16) & 15u) * ux + ((f >> 20) & 15u) * ys + (o >> 12)) & 63u : 0u;
                const uint32_t e = pc > 3 ? (((f >> 24) & 15u) * ux + (f >> 28) * ys + (o >> 18)) & 63u : 0u;
                const int part = a >= q && a >= c && a >= e ? 0 : q >= c && q >= e ? 1 : c >= e ? 2 : 3;
                b = s.ep[k][part][0];
                d = s.ep[k][part][1];
            }
            int v0 = wt, v1 = wt, v2 = wt, v3 = wt;
            if (h & (1u << 12)) {
                const uint8_t* g2 = g + kPlane2;
                const int wt2 = (g2[0] * w00 + g2[1] * w01 + g2[xw] * w10 + g2[xw + 1] * w11 + 8) >> 4, ccs = (int)(h >> 13);
                if (ccs == 0) v0 = wt2; else if (ccs == 1) v1 = wt2; else if (ccs == 2) v2 = wt2; else v3 = wt2;
            }
            const uint32_t r0 = unorm8((b.x + d.x * v0) >> 6), r1 = unorm8((b.y + d.y * v1) >> 6);
            const uint32_t r2 = unorm8((b.z + d.z * v2) >> 6), r3 = unorm8((b.w + d.w * v3) >> 6);
            const size_t at = at0 + (size_t)y * dx;
            if constexpr (kError) {
                const uchar4 r = ref[at];
                const int d0 = (int)r0 - (int)r.x, d1 = (int)r1 - (int)r.y, d2 = (int)r2 - (int)r.z, d3 = (int)r3 - (int)r.w;
                acc[0] += (unsigned long long)(d0 * d0); acc[1] += (unsigned long long)(d1 * d1);
                acc[2] += (unsigned long long)(d2 * d2); acc[3] += (unsigned long long)(d3 * d3);
            } else {
                reinterpret_cast<uint32_t*>(out)[at] = r0 | r1 << 8 | r2 << 16 | r3 << 24;
            }
        }
    }
    if constexpr (kError) {
#pragma unroll
        for (int c = 0; c < 4; c++) {
            unsigned long long t = acc[c];
            for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xFFFFFFFFu, t, o);
            if ((tid & 31) == 0 && t) atomicAdd(&sse[c], t);
        }
    }
}

// image: RGBA8, 4-byte aligned (uchar4 accesses)
int check_args(uint32_t bx, uint32_t by, uint32_t dx, uint32_t dy, const void* blocks, const void* image) {
    if (!blocks || !image || dx == 0 || dy == 0 || ((uintptr_t)image & 3)) return ASTCB200_BAD_ARG;
    if (!valid_footprint((int)bx, (int)by)) return ASTCB200_INVALID_FOOTPRINT;
    const uint64_t nb = (uint64_t)((dx + bx - 1) / bx) * ((dy + by - 1) / by);
    if (nb > (uint64_t)0x7FFFFFFF) return ASTCB200_BAD_ARG;
    return ASTCB200_OK;
}

template <bool kError>
int launch_decode(uint32_t bx, uint32_t by, uint32_t dx, uint32_t dy, const uint8_t* blocks, uint8_t* out, const uint8_t* ref,
                  unsigned long long* sse, cudaStream_t s) {
    const int nbx = (int)((dx + bx - 1) / bx), nby = (int)((dy + by - 1) / by);
    const int cols = nbx < kDecodeBlocks ? nbx : kDecodeBlocks, rows = kDecodeBlocks / cols;
    const int groups_x = (nbx + cols - 1) / cols, groups_y = (nby + rows - 1) / rows;
    k_decode<kError><<<(unsigned)groups_x * (unsigned)groups_y, kDecodeThreads, 0, s>>>(
        blocks, (int)bx, (int)by, (int)dx, (int)dy, nbx, nby, cols, groups_x,
        reinterpret_cast<uchar4*>(out), reinterpret_cast<const uchar4*>(ref), sse);
    return cudaGetLastError() == cudaSuccess ? ASTCB200_OK : ASTCB200_CUDA_ERROR;
}

}  // namespace
}  // namespace astcb200

using namespace astcb200;

extern "C" {

int astcb200_decode_device(uint32_t block_x, uint32_t block_y, uint32_t dim_x, uint32_t dim_y, const uint8_t* d_blocks,
                           uint8_t* d_rgba8, void* cuda_stream) {
    const int rc = check_args(block_x, block_y, dim_x, dim_y, d_blocks, d_rgba8);
    if (rc) return rc;
    return launch_decode<false>(block_x, block_y, dim_x, dim_y, d_blocks, d_rgba8, nullptr, nullptr, (cudaStream_t)cuda_stream);
}

int astcb200_decode_error_device(uint32_t block_x, uint32_t block_y, uint32_t dim_x, uint32_t dim_y, const uint8_t* d_blocks,
                                 const uint8_t* d_ref_rgba8, uint64_t* d_sse, void* cuda_stream) {
    int rc = check_args(block_x, block_y, dim_x, dim_y, d_blocks, d_ref_rgba8);
    if (rc) return rc;
    if (!d_sse) return ASTCB200_BAD_ARG;
    cudaStream_t s = (cudaStream_t)cuda_stream;
    if (cudaMemsetAsync(d_sse, 0, 4 * sizeof(uint64_t), s) != cudaSuccess) return ASTCB200_CUDA_ERROR;
    return launch_decode<true>(block_x, block_y, dim_x, dim_y, d_blocks, nullptr, d_ref_rgba8,
                               reinterpret_cast<unsigned long long*>(d_sse), s);
}

}  // extern "C"
