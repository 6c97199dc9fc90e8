// Device-side ASTC block parser, the same values as decode_block.cuh's parse_block for every
// 128-bit pattern: two threads a block (weights; endpoints and partition seeds), 32-bit words read
// with funnel shifts, integer sequences and unquantisation by tables that the decoder's own
// functions fill at compile time.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "decode_block.cuh"

namespace astcb200 {
namespace dec {
namespace fast {
namespace {

// Digits of packed trits (2 bits each) and quints (3 bits each), unquantised weights and
// colours by value, bits | trits << 4 | quints << 5 of the quantisation methods, bits of n
// weights, and the finest colour method of n values in b bits (0: none an LDR block may use),
// all from the decoder's own functions at compile time.
struct alignas(16) ValueTables {  // k_decode copies them as words
    uint16_t trits[256], quints[128];
    uint8_t weight[12][32];
};
struct DecodeTables {
    ValueTables values;
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
        for (int e = 0; e < 5; e++) t.values.trits[i] = (uint16_t)(t.values.trits[i] | d[e] << (2 * e));
    }
    for (int i = 0; i < 128; i++) {
        int d[3] = {0, 0, 0};
        dec::quint_digits(i, d);
        for (int e = 0; e < 3; e++) t.values.quints[i] = (uint16_t)(t.values.quints[i] | d[e] << (3 * e));
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
            if (q < 12) t.values.weight[q][v] = (uint8_t)dec::unq_weight(q, v);
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

// Parsed blocks in shared memory, arrays by block.
constexpr int kWeightRow = 100;  // bytes of a block's weights: planes 48 apart, zeros past the grid; an odd number of words
constexpr int kPlane2 = 48;
constexpr int kWords = 5;      // the block's four words and one of 0: an odd stride
constexpr int kColourRow = 28;  // bytes of a block's colour values: 18, and 8 read past any endpoint's first
template <int N>
struct Stage {
    int4 ep[N][4][2];      // per partition: 64 x 257 e0 + 32 + 128 x 64, and 257 (e1 - e0), per channel
    uint32_t words[N][kWords];
    uint32_t head[N];      // grid width | height << 4 | partitions << 8 | dual << 12 | plane-2 channel << 13
    uint32_t seed[N], offs[N];  // partition hash: eight 4-bit factors; four 6-bit offsets
    uint8_t w[N][kWeightRow];
    uint8_t cv[N][kColourRow];
};

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
template <int N>
__device__ __forceinline__ void parse_weights(Stage<N>& s, const ValueTables& tables, int k, const dec::Mode& m) {
    const uint32_t* w = s.words[k];
    uint8_t* out = s.w[k];
    const int W = m.xw * m.yw, np = m.dual ? 2 : 1, n = W * np;
    const uint32_t method = g_tables.method[m.q];
    const int bits = method & 15;
    const uint32_t mask = (1u << bits) - 1u;
    const uint8_t* unq = tables.weight[m.q];
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
            const uint32_t d = tables.trits[T];
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
            const uint32_t d = tables.quints[Q];
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
template <int N>
__device__ __forceinline__ void parse_colours(Stage<N>& s, const ValueTables& tables, int k, int off, int nv, int q) {
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
            const uint32_t d = tables.trits[T];
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
            const uint32_t d = tables.quints[Q];
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
template <int N>
__device__ __forceinline__ void constant_block(Stage<N>& s, int k, int c0, int c1, int c2, int c3) {
    s.head[k] = 2u | 2u << 4 | 1u << 8;
    const int add = 32 + 128 * 64;
    s.ep[k][0][0] = make_int4(c0 * 64 + add, c1 * 64 + add, c2 * 64 + add, c3 * 64 + add);
    s.ep[k][0][1] = make_int4(0, 0, 0, 0);
}

// Header, endpoints and partition hash of block k; weights: the weights instead.
template <int N>
__device__ __forceinline__ void parse_part(Stage<N>& s, const ValueTables& tables, int k, int bx, int by, bool weights) {
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
        if (ok) parse_weights(s, tables, k, m);
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
        parse_colours(s, tables, k, cstart, nv, cq);
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

// Partition of texel (x, y) of block k (more than one partition), both doubled in blocks below 31 texels.
__device__ __forceinline__ int texel_partition(uint32_t f, uint32_t o, int pc, uint32_t x, uint32_t y) {
    const uint32_t a = ((f & 15u) * x + ((f >> 4) & 15u) * y + o) & 63u;
    const uint32_t b = (((f >> 8) & 15u) * x + ((f >> 12) & 15u) * y + (o >> 6)) & 63u;
    const uint32_t c = pc > 2 ? (((f >> 16) & 15u) * x + ((f >> 20) & 15u) * y + (o >> 12)) & 63u : 0u;
    const uint32_t e = pc > 3 ? (((f >> 24) & 15u) * x + (f >> 28) * y + (o >> 18)) & 63u : 0u;
    return a >= b && a >= c && a >= e ? 0 : b >= c && b >= e ? 1 : c >= e ? 2 : 3;
}

}  // namespace
}  // namespace fast
}  // namespace dec
}  // namespace astcb200
