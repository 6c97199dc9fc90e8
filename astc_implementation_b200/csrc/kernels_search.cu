// Partition search and front-end kernels of the ASTC encoder (sm_100a).
//
//   k_partition_search  passes 001-007 (shaders/pass001..pass007): k-means over
//                       the block's texels, coverage mismatch against every
//                       selected partitioning, the reference's bitonic ordering,
//                       error estimate of 128 candidates, pick of 4.
//                       One warp per (block, partition count).
//   k_front             passes 01-12 (shaders/pass01..pass12) for one
//                       partitioned block per CTA: ideal endpoints, per
//                       decimation-mode weight solving, per block-mode weight
//                       quantisation error, colour-format search, top-8 pick.
//
// Sums whose order the reference leaves to float atomics are taken in ascending
// texel / weight order, each by one thread or lane, so results are bit-identical
// to the CPU oracle (oracle/astc_oracle.cpp), which fixes the same order; integer
// sums, whose order does not matter, may be split or regrouped.
#include <algorithm>

#include "device_math.cuh"
#include "kernels.h"

namespace astcb200 {

using namespace dev;

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr float ERR_DEFAULT = 1e37f;
__constant__ int c_levels[21] = {2, 3, 4, 5, 6, 8, 10, 12, 16, 20, 24, 32, 40, 48, 64, 80, 96, 128, 160, 192, 256};
__constant__ int c_steps_for_quant[12] = {2, 3, 4, 5, 6, 8, 10, 12, 16, 20, 24, 32};
__constant__ int c_free_bits[4] = {111, 97, 94, 91};  // pass07:5
// pass10's format-class combinations (i | j << 2 | k << 4 | l << 6) for P = 2, 3, 4: every
// tuple of classes 0..3 whose classes lie within one of each other (the pass's i, j, k, l
// loops with their skips), grouped by the total i + j + k + l and, inside a total, in loop
// order; c_combo_off[P - 2][c] .. [c + 1] delimits total c.
__constant__ uint8_t c_combo[78] = {
    0, 4, 1, 5, 9, 6, 10, 14, 11, 15,                                                      // P = 2
    0, 16, 4, 1, 20, 17, 5, 21, 37, 25, 22, 41, 38, 26, 42, 58, 46, 43, 62, 59, 47, 63,     // P = 3
    0, 64, 16, 4, 1, 80, 68, 20, 65, 17, 5, 84, 81, 69, 21, 85, 149, 101, 89, 86, 165, 153,  // P = 4
    105, 150, 102, 90, 169, 166, 154, 106, 170, 234, 186, 174, 171, 250, 238, 190, 235, 187, 175,
    254, 251, 239, 191, 255};
__constant__ uint8_t c_combo_off[3][14] = {{0, 1, 3, 4, 6, 7, 9, 10, 10, 10, 10, 10, 10, 10},
                                           {10, 11, 14, 17, 18, 21, 24, 25, 28, 31, 32, 32, 32, 32},
                                           {32, 33, 37, 43, 47, 48, 52, 58, 62, 63, 67, 73, 77, 78}};

enum { FMT_LUMINANCE = 0, FMT_LUMINANCE_ALPHA = 4, FMT_RGB_SCALE = 6, FMT_RGB = 8, FMT_RGB_SCALE_ALPHA = 10, FMT_RGBA = 12 };

struct Tabs {
    const uint8_t* b;
    const TableLayout* L;
    __device__ const DevDm& dm(int m) const { return reinterpret_cast<const DevDm*>(b + L->off_dm)[m]; }
    __device__ const DevBm& bm(int i) const { return reinterpret_cast<const DevBm*>(b + L->off_bm)[i]; }
    __device__ int bm_order(int j) const { return reinterpret_cast<const uint16_t*>(b + L->off_bm_order)[j]; }
    __device__ const uint32_t* part2(int P, int e) const { return reinterpret_cast<const uint32_t*>(b + L->off_part2) + ((size_t)(P - 2) * 1024 + e) * ((L->T + 15) >> 4); }
    __device__ int part_count(int P, int e, int q) const { return b[L->off_part_counts + ((P - 2) * 1024 + e) * 4 + q]; }
    __device__ uint32_t part_seed(int P, int e) const { return reinterpret_cast<const uint32_t*>(b + L->off_part_info)[(P - 2) * 1024 + e]; }
    __device__ uint64_t cov(int P, int e, int q) const { return reinterpret_cast<const uint64_t*>(b + L->off_cov)[((size_t)(P - 2) * 1024 + e) * 4 + q]; }
    __device__ float2 trig(int i) const { return reinterpret_cast<const float2*>(b + L->off_trig)[i]; }
    __device__ uint4 tw4f(int m, int t) const { return reinterpret_cast<const uint4*>(b + L->off_tw4f)[m * L->T + t]; }
    __device__ uint32_t wt_info(int m, int w) const { return reinterpret_cast<const uint32_t*>(b + L->off_wt_info)[m * 64 + w]; }
    __device__ const uint16_t* witems() const { return reinterpret_cast<const uint16_t*>(b + L->off_witem); }
    __device__ const uint16_t* sitems() const { return reinterpret_cast<const uint16_t*>(b + L->off_sitem); }
    __device__ const uint4* w2tf(int i) const { return reinterpret_cast<const uint4*>(b + L->off_w2tf) + i; }
    __device__ uint32_t wgroup(int i) const { return reinterpret_cast<const uint32_t*>(b + L->off_wgroup)[i]; }
    __device__ const uint4* wgent(int i) const { return reinterpret_cast<const uint4*>(b + L->off_wgent) + 32 * i; }
    __device__ int q2u(int i) const { return b[L->off_q2u + i]; }
    __device__ int q2u_start(int q) const { return b[L->off_q2u_start + q]; }
    __device__ int qmt(int row, int bits) const { return reinterpret_cast<const int8_t*>(b + L->off_qmt)[row * 128 + bits]; }
    __device__ float bqe(int i) const { return reinterpret_cast<const float*>(b + L->off_bqe)[i]; }
};

// Index and contribution of a tw4f or w2tf entry.
__device__ __forceinline__ int entry_index(uint32_t e) { return (int)(e & 0xFFFFu); }
__device__ __forceinline__ float entry_factor(uint32_t e) { return __uint_as_float(e & 0xFFFF0000u); }
// Round to the nearest integer, ties to even, on the FP32 adders: as a float for |v| < 2^22, as
// an integer for 0 <= v < 2^22.
__device__ __forceinline__ float rn_small(float v) { return (v + 12582912.0f) - 12582912.0f; }
__device__ __forceinline__ uint32_t rn_bits(float v) { return fbits(v + 8388608.0f) - 0x4B000000u; }
// Small integers as floats and non-negative floats truncated, without the conversion pipe.
__device__ __forceinline__ float small_float(uint32_t v) { return __uint_as_float(0x4B000000u | v) - 8388608.0f; }
__device__ __forceinline__ uint32_t small_trunc(float v) { return fbits(__fadd_rz(v, 8388608.0f)) - 0x4B000000u; }

__device__ __forceinline__ float dist_sq(float4 a, float4 b) {
    const float4 d = a - b;
    return dot4(d * d, chan_w());
}

// ============================================================ passes 001-007
// A warp searches one partition count of a block (small launches: a CTA of four warps, each
// taking one of the four rounds of 32 candidates).  The kernel waited on
// instruction fetch, branches and the conversion pipe,
// not on memory, so: loops are left rolled,
// sort keys are 32 bits with the reference's partial network on registers and shuffles, the
// mismatch is one matching over popcounts of the overlaps, texel partitions come two bits a
// texel, and sums of truncated texels reuse the truncations.  Measured (B200): 11.6 -> 5.4 ms for
// 65,536 4x4 blocks with FIXED semantics, 6.2 -> 1.1 ms for 9,888 10x8 blocks with the reference's.
constexpr int kSearchWarps = 4;
constexpr int kSearchCtas = 5;
// A launch of few items is as long as one item, so each gets a CTA's four warps then (the
// clustering and the order are made four times, the errors once): up to two waves of CTAs.
constexpr int kSearchWideItems = 148 * kSearchCtas * 2;
constexpr int kSearchKeys = 1024;
// Per warp: texels and their truncations, then the sort keys (dead once the order is known:
// the same bytes hold each lane's partition averages and directions), the first 128 table
// entries of the order, the counting sort's histogram, errors, k-means assignments.
constexpr int kSearchLaneVecs = 4 * 3;  // per lane: average, direction, scale direction of P <= 4 partitions
struct SearchLayout { int px, xi, key, ord, hist, eu, es, asg, zero, total; };
__host__ __device__ inline SearchLayout search_layout(int T) {
    SearchLayout f;
    int o = 0;
    auto take = [&](int bytes) { const int r = o; o += (bytes + 15) & ~15; return r; };
    f.px = take(T * 16);
    f.xi = take(T * 16);
    f.key = take(kSearchLaneVecs * 32 * 16);
    f.ord = take(kPartCandLimit * 2);
    f.hist = take(132 * 4);
    f.eu = take(kPartCandLimit * 4);
    f.es = take(kPartCandLimit * 4);
    f.asg = take(T);
    f.zero = take(T);
    f.total = o;
    return f;
}
static_assert(kSearchLaneVecs * 32 * 16 >= kSearchKeys * 4, "the keys fit the lanes' vectors");
constexpr uint32_t kNoEntry = 0x3FFFu;  // mismatch of an entry that is not selected: after all others

// FIXED semantics of pass005 (full sort): the table entries of the first 128 of all keys
// m << 10 | i in ascending order, into ord.  The mismatch counts m of the sel selected entries
// are at most 64, so a stable counting sort by m in index order gives the full order (sel is
// above 128 for every footprint and partition count).
__device__ __forceinline__ void full_order(const uint32_t* key, uint16_t* ord, uint32_t* hist, uint32_t sel, int lane) {
    for (int b = lane; b < 132; b += 32) hist[b] = 0;
    __syncwarp();
#pragma unroll 1
    for (uint32_t i = lane; i < sel; i += 32) atomicAdd(&hist[key[i] >> 10], 1u);
    __syncwarp();
    uint32_t v[5], s = 0;  // exclusive scan of bins 0..128, five per lane
#pragma unroll
    for (int j = 0; j < 5; j++) { const int b = lane * 5 + j; v[j] = b < 129 ? hist[b] : 0u; s += v[j]; }
    uint32_t incl = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const uint32_t t = __shfl_up_sync(FULL, incl, o); if (lane >= o) incl += t; }
    uint32_t run = incl - s;
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 5; j++) { const int b = lane * 5 + j; if (b < 129) hist[b] = run; run += v[j]; }
    __syncwarp();
    const uint32_t lt = (1u << lane) - 1u;
#pragma unroll 1
    for (uint32_t base = 0; base < sel; base += 32) {
        const uint32_t i = base + lane;
        const bool selected = i < sel;
        const uint32_t m = selected ? key[i] >> 10 : kNoEntry;
        const uint32_t grp = __match_any_sync(FULL, m);
        if (selected) {
            const uint32_t rank = hist[m] + __popc(grp & lt);
            if (rank < (uint32_t)kPartCandLimit) ord[rank] = (uint16_t)i;
        }
        __syncwarp();
        if (selected && 31 - __clz(grp) == lane) hist[m] += __popc(grp);
        __syncwarp();
    }
}

// The reference's pass005: its bitonic network run by 256 invocations, which only compares
// pairs whose lower index is below 256.  Keys 0..255 stay in registers (key lane + 32 r in
// x[r]); only the two steps of distance 256 and 512 reach the others, in shared memory.
__device__ __forceinline__ void partial_order(uint32_t* key, uint16_t* ord, int lane) {
    uint32_t x[8];
#pragma unroll
    for (int r = 0; r < 8; r++) x[r] = key[lane + 32 * r];
    auto within = [&](unsigned k, unsigned j) {  // one step of distance j < 256
        if (j >= 32) {
            const int jr = (int)(j >> 5);
#pragma unroll
            for (int r = 0; r < 8; r++) {
#pragma unroll
                for (int d = 1; d < 8; d <<= 1) {
                    if ((r & d) || jr != d) continue;
                    const bool asc = ((32u * r) & k) == 0;  // k > j >= 32: the lane does not enter
                    const uint32_t lo = min(x[r], x[r | d]), hi = max(x[r], x[r | d]);
                    x[r] = asc ? lo : hi;
                    x[r | d] = asc ? hi : lo;
                }
            }
        } else {
            const bool lower = (lane & j) == 0;
#pragma unroll
            for (int r = 0; r < 8; r++) {
                const uint32_t o = __shfl_xor_sync(FULL, x[r], j);
                const bool asc = ((lane + 32 * r) & k) == 0;
                x[r] = lower == asc ? min(x[r], o) : max(x[r], o);
            }
        }
    };
    auto across = [&](int d) {  // distance d >= 256, ascending (indices below 256)
#pragma unroll
        for (int r = 0; r < 8; r++) {
            uint32_t& o = key[lane + 32 * r + d];
            const uint32_t lo = min(x[r], o), hi = max(x[r], o);
            x[r] = lo;
            o = hi;
        }
    };
#pragma unroll 1
    for (unsigned k = 2; k <= (unsigned)kSearchKeys; k <<= 1) {
        if (k == 1024) across(512);
        if (k >= 512) across(256);
#pragma unroll 1
        for (unsigned j = min(k >> 1, 128u); j > 0; j >>= 1) within(k, j);
    }
#pragma unroll
    for (int r = 0; r < 4; r++) ord[lane + 32 * r] = (uint16_t)(x[r] & 1023u);
}

// wide: this warp is one of four that search the same partition count of a block and only
// takes round `round` of the candidates; the errors go to warp 0's arrays (eu0, es0), and the
// CTA's barrier before pass007 is the caller's.
template <int P>
__device__ __forceinline__ void search_errors(const KernelArgs& a, int blk, uint8_t* ws, int lane, bool wide, int round, float* eu0, float* es0) {
    const Tabs tb{a.tables, &a.L};
    const int T = a.L.T;
    const SearchLayout fl = search_layout(T);
    float4* px = reinterpret_cast<float4*>(ws + fl.px);
    uint4* xi = reinterpret_cast<uint4*>(ws + fl.xi);
    uint32_t* key = reinterpret_cast<uint32_t*>(ws + fl.key);
    uint16_t* ord = reinterpret_cast<uint16_t*>(ws + fl.ord);
    uint8_t* asg = ws + fl.asg;
    uint8_t* zero = ws + fl.zero;  // per texel: bit c set when channel c is 0
    const float4 cw = chan_w();
    const BlockSrc src = block_src(a, blk);
    uint32_t u_all = 0;  // sum over all texels of f2u(|x|^2 weighted), the line error of a zero direction
    bool any_zero = false;
#pragma unroll 1
    for (int t = lane; t < T; t += 32) {
        const float4 x = src_texel(src, a.L.bx, t);
        px[t] = x;
        xi[t] = make_uint4(__float2uint_rz(x.x), __float2uint_rz(x.y), __float2uint_rz(x.z), __float2uint_rz(x.w));
        const int z = (x.x > 0.0f ? 0 : 1) | (x.y > 0.0f ? 0 : 2) | (x.z > 0.0f ? 0 : 4) | (x.w > 0.0f ? 0 : 8);
        zero[t] = (uint8_t)z;
        any_zero |= z != 0;
        u_all += f2u(dot4(x * x, cw));
    }
    any_zero = __any_sync(FULL, any_zero);
    u_all = __reduce_add_sync(FULL, u_all);
    __syncwarp();

    // pass001: farthest-point initial centres; ties pick the highest texel index
    float4 c[P];
    c[0] = px[145897 % T];
    {
        auto dist = [&](int t, int n) {  // to the nearest of the first n centres
            float d = dist_sq(c[0], px[t]);
#pragma unroll
            for (int q = 1; q < P; q++) if (q < n) d = fminf(d, dist_sq(c[q], px[t]));
            return d;
        };
#pragma unroll
        for (int pp = 1; pp < P; pp++) {
            uint32_t mx = 0;
            int idx = -1;
#pragma unroll 1
            for (int t = lane; t < T; t += 32) { const uint32_t d = fbits(dist(t, pp)); if (d >= mx) { mx = d; idx = t; } }
            const uint32_t best = __reduce_max_sync(FULL, mx);
            idx = __reduce_max_sync(FULL, mx == best ? idx : -1);
            c[pp] = px[idx];
        }
    }
    // passes 002/003, four iterations
#pragma unroll 1
    for (int it = 0; it < 4; it++) {
        uint32_t have = 0;
#pragma unroll 1
        for (int t = lane; t < T; t += 32) {
            float best = 1e30f;
            uint32_t as = 0;
            const float4 x = px[t];
#pragma unroll
            for (int q = 0; q < P; q++) { const float d = dist_sq(x, c[q]); if (d < best) { best = d; as = q; } }
            asg[t] = (uint8_t)as;
            have |= 1u << as;
        }
        have = __reduce_or_sync(FULL, have);
        if (have != (1u << P) - 1u && lane < P) asg[lane] = (uint8_t)lane;  // an empty cluster
#pragma unroll
        for (int q = 0; q < P; q++) {
            uint32_t n = 0, s0 = 0, s1 = 0, s2 = 0, s3 = 0;
#pragma unroll 1
            for (int t = lane; t < T; t += 32)
                if (asg[t] == q) { const uint4 x = xi[t]; n++; s0 += x.x; s1 += x.y; s2 += x.z; s3 += x.w; }
            n = __reduce_add_sync(FULL, n);
            s0 = __reduce_add_sync(FULL, s0); s1 = __reduce_add_sync(FULL, s1);
            s2 = __reduce_add_sync(FULL, s2); s3 = __reduce_add_sync(FULL, s3);
            c[q] = mk(0.0f);
            if (n > 0) { const float fc = (float)n; c[q] = make_float4((float)s0 / fc, (float)s1 / fc, (float)s2 / fc, (float)s3 / fc); }
        }
    }
    __syncwarp();
    // pass004: k-means bitmaps over the 64 k-means texels, mismatch per partitioning.  The
    // mismatch is half the smallest sum over assignments x -> y of popc(km_x ^ cov_y); the xor
    // counts popc(km_x) + popc(cov_y) - 2 popc(km_x & cov_y), whose first two terms sum to the
    // same total for every assignment, so it is half that total less the largest matching over
    // the overlaps n.  The cov of an entry split the first min(T, 64) bits between them, and so
    // do the km, so the overlaps of the last row and column follow from the others.
    const int nbits = min(T, 64);
    uint64_t km[P];
    int kn[P];  // of the first nbits
    {
        const int k0 = asg[a.L.kmeans[lane]], k1 = asg[a.L.kmeans[lane + 32]];
        const uint64_t valid = nbits == 64 ? ~0ull : (1ull << nbits) - 1;
#pragma unroll
        for (int q = 0; q < P; q++) {
            const uint32_t lo = __ballot_sync(FULL, k0 == q), hi = __ballot_sync(FULL, k1 == q);
            km[q] = ((uint64_t)lo | ((uint64_t)hi << 32)) & valid;
            kn[q] = __popcll(km[q]);
        }
    }
    const uint32_t half_total = (uint32_t)(64 + nbits) / 2;
    const uint32_t sel = a.L.count_selected[P - 1];
    const uint32_t nkeys = a.fixed ? (sel + 31u) & ~31u : (uint32_t)kSearchKeys;
#pragma unroll 1
    for (uint32_t i = lane; i < nkeys; i += 32) {
        uint32_t m = kNoEntry;
        if (i < sel) {
            int n[P][P], rest = nbits;
#pragma unroll
            for (int y = 0; y < P - 1; y++) {
                const uint64_t cv = tb.cov(P, i, y);
                int col = T <= 32 ? __popc((uint32_t)cv) : __popcll(cv);
                rest -= col;
#pragma unroll
                for (int x = 0; x < P - 1; x++) {
                    n[x][y] = T <= 32 ? __popc((uint32_t)km[x] & (uint32_t)cv) : __popcll(km[x] & cv);
                    col -= n[x][y];
                }
                n[P - 1][y] = col;
            }
#pragma unroll
            for (int x = 0; x < P - 1; x++) {
                int r = kn[x];
#pragma unroll
                for (int y = 0; y < P - 1; y++) r -= n[x][y];
                n[x][P - 1] = r;
                rest -= r;
            }
            n[P - 1][P - 1] = rest;
            int best;
            if (P == 2) {
                best = max(n[0][0] + n[P - 1][P - 1], n[0][P - 1] + n[P - 1][0]);
            } else if (P == 3) {
                best = max(n[0][0] + max(n[1][1] + n[P - 1][P - 1], n[1][P - 1] + n[P - 1][1]),
                           max(n[0][1] + max(n[1][0] + n[P - 1][P - 1], n[1][P - 1] + n[P - 1][0]),
                               n[0][P - 1] + max(n[1][0] + n[P - 1][1], n[1][1] + n[P - 1][0])));
            } else {
                best = 0;
#pragma unroll
                for (int x = 0; x < 4; x++)
#pragma unroll
                    for (int y = x + 1; y < 4; y++) {  // rows 0, 1 on columns x, y, rows 2, 3 on the others
                        const int u = x == 0 ? (y == 1 ? 2 : 1) : 0, v = 6 - x - y - u;
                        const int top = max(n[0][x] + n[1][y], n[0][y] + n[1][x]);
                        const int bot = max(n[P - 2][u] + n[P - 1][v], n[P - 2][v] + n[P - 1][u]);
                        best = max(best, top + bot);
                    }
            }
            m = half_total - (uint32_t)best;
        }
        key[i] = m << 10 | i;
    }
    __syncwarp();
    if (a.fixed) full_order(key, ord, reinterpret_cast<uint32_t*>(ws + fl.hist), sel, lane);
    else partial_order(key, ord, lane);
    __syncwarp();
    // pass006: error estimate of the first 128 ordered partitionings.  The
    // shader keeps avg/dir in per-invocation arrays, so texel t only sees its
    // own partition's average/direction when t < P and its partition is t.
    float wie = T <= 20 ? 0.03f : T <= 31 ? 0.04f : T <= 41 ? 0.05f : 0.055f;
    wie = wie * wie;
    float4* lv = reinterpret_cast<float4*>(key) + lane;  // lane's vectors: (3 q + kind) * 32
#pragma unroll 1
    for (int r = wide ? round : 0; r < (wide ? round + 1 : 4); r++) {
        const int cand = lane + 32 * r;
        const int e = ord[cand];
        const uint32_t* row = tb.part2(P, e);
        // counts and sums of the truncated texels; partition 0's are what the others leave
        uint32_t cnt[P], sm[P][4];
#pragma unroll
        for (int q = 0; q < P; q++) { cnt[q] = 0; sm[q][0] = sm[q][1] = sm[q][2] = sm[q][3] = 0; }
#pragma unroll 1
        for (int w0 = 0; w0 < T; w0 += 16) {
            uint32_t w = row[w0 >> 4];
            const int tn = min(T - w0, 16);
#pragma unroll 1
            for (int t = 0; t < tn; t++, w >>= 2) {
                const uint32_t p = w & 3u;
                const uint4 x = xi[w0 + t];
                sm[0][0] += x.x; sm[0][1] += x.y; sm[0][2] += x.z; sm[0][3] += x.w;
#pragma unroll
                for (int q = 1; q < P; q++) if (p == (uint32_t)q) { cnt[q]++; sm[q][0] += x.x; sm[q][1] += x.y; sm[q][2] += x.z; sm[q][3] += x.w; }
            }
        }
        cnt[0] = (uint32_t)T;
#pragma unroll
        for (int q = 1; q < P; q++) {
            cnt[0] -= cnt[q];
#pragma unroll
            for (int ch = 0; ch < 4; ch++) sm[0][ch] -= sm[q][ch];
        }
        uint32_t usum = u_all, ssum = 0u - (uint32_t)T;
        const uint32_t w_first = row[0];
#pragma unroll
        for (int q = 0; q < P; q++) {
            const float fc = (float)cnt[q];
            const float4 tavg = fc > 0.0f ? make_float4((float)sm[q][0] / fc, (float)sm[q][1] / fc, (float)sm[q][2] / fc, (float)sm[q][3] / fc) : mk(0.0f);
            uint32_t ax[4][4];
            const bool own = ((w_first >> (2 * q)) & 3u) == (uint32_t)q;  // texel q is in partition q
            if (a.fixed) {
                // sums of the deviations along each positive half axis, over the partition's texels
#pragma unroll
                for (int u = 0; u < 4; u++) ax[u][0] = ax[u][1] = ax[u][2] = ax[u][3] = 0;
#pragma unroll 1
                for (int w0 = 0; w0 < T; w0 += 16) {
                    uint32_t w = row[w0 >> 4] ^ (0x55555555u * (uint32_t)q);
                    w = ~(w | w >> 1) & 0x55555555u;
                    if (T - w0 < 16) w &= (1u << (2 * (T - w0))) - 1u;
                    while (w) {
                        const int t = w0 + ((__ffs(w) - 1) >> 1);
                        w &= w - 1;
                        const float4 d = px[t] - tavg;
                        const uint32_t d0 = (uint32_t)__float2int_rz(d.x), d1 = (uint32_t)__float2int_rz(d.y);
                        const uint32_t d2 = (uint32_t)__float2int_rz(d.z), d3 = (uint32_t)__float2int_rz(d.w);
                        if (d.x > 0.0f) { ax[0][0] += d0; ax[0][1] += d1; ax[0][2] += d2; ax[0][3] += d3; }
                        if (d.y > 0.0f) { ax[1][0] += d0; ax[1][1] += d1; ax[1][2] += d2; ax[1][3] += d3; }
                        if (d.z > 0.0f) { ax[2][0] += d0; ax[2][1] += d1; ax[2][2] += d2; ax[2][3] += d3; }
                        if (d.w > 0.0f) { ax[3][0] += d0; ax[3][1] += d1; ax[3][2] += d2; ax[3][3] += d3; }
                    }
                }
            } else {
                // Every texel but texel q sees a zero average: its deviation is itself, so the
                // sums along axis u are the partition's less the texels whose channel u is 0;
                // texel q, when it is of partition q, sees the average.
#pragma unroll
                for (int u = 0; u < 4; u++)
#pragma unroll
                    for (int ch = 0; ch < 4; ch++) ax[u][ch] = sm[q][ch];
                if (any_zero) {
#pragma unroll 1
                    for (int t = 0; t < T; t++) {
                        const int z = zero[t];
                        if (z == 0) continue;  // the same for every lane
                        if (((row[t >> 4] >> (2 * (t & 15))) & 3u) != (uint32_t)q) continue;
                        const uint4 x = xi[t];
#pragma unroll
                        for (int u = 0; u < 4; u++)
                            if ((z >> u) & 1) { ax[u][0] -= x.x; ax[u][1] -= x.y; ax[u][2] -= x.z; ax[u][3] -= x.w; }
                    }
                }
                if (own) {
                    const uint4 x = xi[q];
                    const int z = zero[q];
                    const float4 d = px[q] - tavg;
                    const uint32_t d0 = (uint32_t)__float2int_rz(d.x), d1 = (uint32_t)__float2int_rz(d.y);
                    const uint32_t d2 = (uint32_t)__float2int_rz(d.z), d3 = (uint32_t)__float2int_rz(d.w);
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        if (!((z >> u) & 1)) { ax[u][0] -= x.x; ax[u][1] -= x.y; ax[u][2] -= x.z; ax[u][3] -= x.w; }
                        if (comp(d, u) > 0.0f) { ax[u][0] += d0; ax[u][1] += d1; ax[u][2] += d2; ax[u][3] += d3; }
                    }
                }
            }
            float4 best = mk(0.0f);
            float mp = 0.0f;
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const float4 s = make_float4((float)(int32_t)ax[u][0], (float)(int32_t)ax[u][1], (float)(int32_t)ax[u][2], (float)(int32_t)ax[u][3]);
                const float pr = dot4(s, s);
                if (u == 0 || pr > mp) { mp = pr; best = s; }
            }
            const float4 tdir = normalize4(best);
            if (a.fixed) {
                lv[(3 * q) * 32] = tavg;
                lv[(3 * q + 1) * 32] = tdir;
                lv[(3 * q + 2) * 32] = normalize4(tavg);
            } else {
                // Every texel but those t < P of partition t sees a zero average and direction: its
                // projection is 0, its line error |x|^2 (weighted) and its scale error NaN (the zero
                // direction's normalisation), so f2u gives 0xFFFFFFFF.  The integer sums take those
                // terms for every texel at once (u_all, -T) and the few texels that see their
                // partition's own average and direction are corrected; integer sums do not depend
                // on their order.
                int32_t lmin = 2147483647, lmax = -2147483647;
                if (own) {
                    const float4 x = px[q];
                    usum -= f2u(dot4(x * x, cw));
                    ssum += 1u;
                    const float up = dot4(x, tdir);
                    const float4 uproj = tavg + tdir * dot4(x - tavg, tdir);
                    const float4 udiff = x - uproj;
                    const float4 sd = normalize4(tavg);
                    const float4 sproj = sd * dot4(x, sd);
                    const float4 sdiff = x - sproj;
                    usum += f2u(dot4(udiff * udiff, cw));
                    ssum += f2u(dot4(sdiff * sdiff, cw));
                    const int32_t upi = f2i(up * 4096.0f);
                    lmin = min(lmin, upi); lmax = max(lmax, upi);
                }
                if ((int)cnt[q] > (own ? 1 : 0)) { lmin = min(lmin, 0); lmax = max(lmax, 0); }  // a texel of projection 0
                lv[(3 * q) * 32] = make_float4(__int_as_float(lmin), __int_as_float(lmax), q == 0 ? dot4(tavg, tavg) : 0.0f, 0.0f);
            }
        }
        int32_t lmin[P], lmax[P];
        if (a.fixed) {  // every texel sees its partition's average and direction
            usum = 0u; ssum = 0u;
#pragma unroll
            for (int q = 0; q < P; q++) { lmin[q] = 2147483647; lmax[q] = -2147483647; }
#pragma unroll 1
            for (int w0 = 0; w0 < T; w0 += 16) {
                uint32_t w = row[w0 >> 4];
                const int tn = min(T - w0, 16);
#pragma unroll 1
                for (int t = 0; t < tn; t++, w >>= 2) {
                    const int p = (int)(w & 3u);
                    const float4 av = lv[(3 * p) * 32], ud = lv[(3 * p + 1) * 32], sd = lv[(3 * p + 2) * 32];
                    const float4 x = px[w0 + t];
                    const float up = dot4(x, ud);
                    const float4 uproj = av + ud * dot4(x - av, ud);
                    const float4 udiff = x - uproj;
                    usum += f2u(dot4(udiff * udiff, cw));
                    const float4 sproj = sd * dot4(x, sd);
                    const float4 sdiff = x - sproj;
                    ssum += f2u(dot4(sdiff * sdiff, cw));
                    const int32_t upi = f2i(up * 4096.0f);
#pragma unroll
                    for (int q = 0; q < P; q++) if (p == q) { lmin[q] = min(lmin[q], upi); lmax[q] = max(lmax[q], upi); }
                }
            }
        }
        float tu = (float)usum, ts = (float)ssum;
#pragma unroll
        for (int q = 0; q < P; q++) {
            float sq;  // |average|^2 the scale term sees
            if (a.fixed) {
                const float4 a0 = lv[(3 * q) * 32];
                sq = dot4(a0, a0);
            } else {
                const float4 v = lv[(3 * q) * 32];
                lmin[q] = __float_as_int(v.x); lmax[q] = __float_as_int(v.y);
                sq = v.z;
            }
            const float mn = (float)lmin[q] / 4096.0f, mxv = (float)lmax[q] / 4096.0f;
            const float ll = fmaxf(mxv - mn, 1e-7f);
            const float ew = (float)cnt[q] * wie;
            tu = tu + ew * (ll * ll);
            ts = ts + ew * sq;
        }
        eu0[cand] = tu;
        es0[cand] = ts;
    }
}

// pass007 by one warp: the best 4 by each error (value, then rank), interleaved and
// deduplicated; the rank is used as the table entry (REF-BUG-4, pass007:93,156), in FIXED
// semantics the entry of that rank.
__device__ __forceinline__ void search_picks(const KernelArgs& a, int P, int lb, const float* eu, const float* es, const uint16_t* ord, int lane) {
    uint32_t best[2][4];
#pragma unroll 1
    for (int kind = 0; kind < 2; kind++) {
        const float* v = kind ? es : eu;
        uint32_t taken = 0;  // rounds of this lane already picked
        uint32_t got[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            float mv = 1e30f;
            int mr = -1;
#pragma unroll
            for (int r = 0; r < 4; r++) { const float x = v[lane + 32 * r]; if (!((taken >> r) & 1) && x < mv) { mv = x; mr = r; } }
            const uint32_t bits = mr >= 0 ? fbits(mv) : 0xFFFFFFFFu;  // the errors are never negative
            const uint32_t mn = __reduce_min_sync(FULL, bits);
            const uint32_t idx = mr >= 0 ? (uint32_t)(lane + 32 * mr) : 0xFFFFFFFFu;
            const uint32_t win = mn == 0xFFFFFFFFu ? 0xFFFFFFFFu : __reduce_min_sync(FULL, bits == mn ? idx : 0xFFFFFFFFu);
            if (win == idx && mr >= 0) taken |= 1u << mr;
            got[j] = win == 0xFFFFFFFFu ? 0u : win;
        }
#pragma unroll
        for (int j = 0; j < 4; j++) { if (kind) best[1][j] = got[j]; else best[0][j] = got[j]; }
    }
    uint32_t fin[4] = {0, 0, 0, 0};
    int emitted = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const uint32_t idx = best[i & 1][i >> 1];
        bool seen = emitted >= 4;
#pragma unroll
        for (int j = 0; j < 4; j++) seen |= j < emitted && fin[j] == idx;
#pragma unroll
        for (int j = 0; j < 4; j++) if (!seen && j == emitted) fin[j] = idx;
        emitted += seen ? 0 : 1;
    }
    uint16_t* out = a.picks[lb].v + (P - 2) * 5;
#pragma unroll
    for (int i = 0; i < 4; i++)
        if (lane == i) out[i] = (uint16_t)(a.fixed && i < emitted ? (uint32_t)ord[fin[i]] : fin[i]);
    if (lane == 4) out[4] = (uint16_t)emitted;
}

__host__ __device__ inline bool search_wide(int items) { return items <= kSearchWideItems; }

__global__ void __launch_bounds__(kSearchWarps * 32, kSearchCtas) k_partition_search(const __grid_constant__ KernelArgs a) {
    extern __shared__ __align__(16) uint8_t smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const SearchLayout fl = search_layout(a.L.T);
    const int nb = list_blocks(a);
    const bool wide = search_wide(nb * 3);
    uint8_t* ws = smem + warp * fl.total;
    uint8_t* w0 = wide ? smem : ws;  // where the errors and the order are read for pass007
    float* eu = reinterpret_cast<float*>(w0 + fl.eu);
    float* es = reinterpret_cast<float*>(w0 + fl.es);
    // P-major items: a CTA's warps share P; one pass for a chunk, a grid-stride loop over a block list
    const int first = wide ? blockIdx.x : blockIdx.x * kSearchWarps + warp, step = wide ? gridDim.x : gridDim.x * kSearchWarps;
    for (int item = first; item < nb * 3; item += step) {
        const int lb = item % nb, P = item / nb + 2;
        const int blk = chunk_block(a, lb);
        if (P == 2) search_errors<2>(a, blk, ws, lane, wide, warp, eu, es);
        else if (P == 3) search_errors<3>(a, blk, ws, lane, wide, warp, eu, es);
        else search_errors<4>(a, blk, ws, lane, wide, warp, eu, es);
        if (wide) __syncthreads(); else __syncwarp();
        if (!wide || warp == 0) {
            search_picks(a, P, lb, eu, es, reinterpret_cast<const uint16_t*>(w0 + fl.ord), lane);
            if (a.work && lane == 0) atomicAdd(a.work + 10 + (P - 2), 1ull);
        }
        if (wide) __syncthreads(); else __syncwarp();
    }
}

// ============================================================ passes 01-12
// One CTA of NT threads per partitioned block (front_nt).  Every value is computed by the same
// thread sequence whatever NT is (loops only spread independent items), so results do not
// depend on it.

struct FrontLayout {
    int px, w, wes, tp, dec, lo, hi, bm_err, ints, trig, qf, misc, dml, bml, witem, sitem, setup, total;
};

constexpr int kColourLevels = 17;  // colour quant levels 4..20; the tables below count from level 4
// (the one-partition instance keeps one partition's colour errors and no format combinations: 5.9
// instead of 9.3 KB at 4x4 with the item lists, so 32 of its warps fit on an SM instead of 22; k_front of
// the 262,144 blocks of 2048x2048 2.27 -> 2.02 ms)
template <bool P1>
struct FrontMisc {
    static constexpr int kParts = P1 ? 1 : 4, kCombos = P1 ? 1 : kColourLevels;
    float4 avg[4], dir[4], ep0[4], ep1[4];
    float mn[4], mx[4], lsq[4];
    float min_cutoff;
    uint32_t is_const, gray, calpha;
    uint32_t ece_can_offset[4], ece_can_bc[4];
    float p9[4][4];  // pass09 inputs per partition: rre, are, brgb, ba
    float sxyz[4][3][4];  // pass08: per partition, sums of the deviations along r, g, b (w = 0)
    float acc[4][5];      // pass08: per partition, the five encoding-choice error sums
    float4 axes[4][4];    // pass08: per partition, ub, ua, sb, la
    float cerr[kParts][kColourLevels][4];
    uint8_t cfmt[kParts][kColourLevels][4];
    float combo_err[kCombos][13];
    __align__(4) uint8_t combo_fmt[kCombos][13][4];
    int top[kNumCand];
    int ncand;
    int nlive;  // block modes in the proposal search's list
};

// pass07's buffer in floats, before it in turn the texel channels and projections of pass01,
// pass08's error terms (5 x Tp; Tp = T rounded up to 4), pass02's infilled weights (T per
// decimation mode) and the angular steps of pass04 (kStepFloats each).  The full search's
// pass07 takes one thread per mode (max_w x nt); the proposal search's (`list`) works on
// groups of kListGroup modes (max_w + Tp each), so its launches need less shared memory
// and more of its CTAs fit on an SM.
constexpr int kListGroup = 16;
constexpr int kStepFloats = 7;  // four errors, then span and lowest index, then the offset
__host__ __device__ inline int front_layout_qf_floats(int T, int max_w, int nt, bool list) {
    const int Tp = (T + 3) & ~3;
    int f = list ? kListGroup * (max_w + Tp) : max_w * nt;
    if (f < 5 * Tp) f = 5 * Tp;
    return f;
}
__host__ __device__ inline int take16(int& o, int bytes) { const int r = o; o = (o + bytes + 15) & ~15; return r; }
__host__ __device__ inline FrontLayout front_layout(const TableLayout& L, int nt, bool list, bool p1) {
    const int T = L.T, ndm = L.ndm, nbm = L.nbm, max_w = L.max_w;
    FrontLayout f;
    int o = 0;
    f.px = take16(o, T * 16);
    f.w = take16(o, T * 4);
    f.wes = take16(o, T * 4);
    f.tp = take16(o, T);
    f.dec = take16(o, L.nw_total * 4);
    f.lo = take16(o, ndm * 8 * 4);
    f.hi = take16(o, ndm * 8 * 4);
    f.bm_err = take16(o, nbm * 4);
    f.ints = take16(o, nbm);
    // pass03's table rows are read before pass07's buffer is written: one region, the rows after
    // the steps and pass02's infill
    const int early = ((ndm * (T > kMaxAngularSteps * kStepFloats ? T : kMaxAngularSteps * kStepFloats) * 4) + 15) & ~15;
    const int rows = early + L.nw_total * 2, qf = front_layout_qf_floats(T, max_w, nt, list) * 4;
    f.qf = take16(o, rows > qf ? rows : qf);
    f.trig = f.qf + early;
    f.misc = take16(o, p1 ? (int)sizeof(FrontMisc<true>) : (int)sizeof(FrontMisc<false>));
    f.dml = take16(o, 16 + ndm * 2);
    f.bml = take16(o, nbm * 2);  // the proposal search's block modes, ascending
    f.witem = take16(o, list ? L.nwi * 2 : 0);  // and the weight and step items of its decimation modes
    f.sitem = take16(o, list ? L.nsi * 2 : 0);
    f.setup = take16(o, list ? kListGroup * 32 : 0);  // quantisation of a group's modes
    f.total = o;
    return f;
}

// Quantised weight w of block mode bmi given the dm's ideal decimated weights
// (pass06 range rules + pass07:230-275).  Returns the unquantised value on the
// 0..64 scale and writes the rescaled float weight.
struct BmQuant {
    float low, scale, slb, rscale, qlm1;
    uint32_t q2u_start, top;  // first entry and last level of the quantisation's values
};
__device__ __forceinline__ BmQuant bm_quant_setup(const Tabs& tb, const DevBm& bm, const float* lo, const float* hi, float min_cutoff) {
    float low = lo[bm.quant < 8 ? bm.quant : 0], high = hi[bm.quant < 8 ? bm.quant : 0];
    if (bm.quant >= 8) { low = 0.0f; high = 0.0f; }  // pass05 never writes slots 8..12 (REF-BUG-5 buffer read as 0)
    if (high > 1.02f * min_cutoff) high = 1.0f;
    if (high <= low) { low = 0.0f; high = 1.0f; }
    BmQuant r;
    r.top = (uint32_t)(c_levels[bm.quant] - 1);
    r.qlm1 = (float)r.top;
    float rscale = high - low;
    r.scale = 1.0f / rscale;
    r.slb = low * r.scale;
    r.rscale = rscale / 64.0f;
    r.low = low;
    r.q2u_start = (uint32_t)tb.q2u_start(bm.quant);
    return r;
}
__device__ __forceinline__ uint32_t bm_quant_weight(const Tabs& tb, const BmQuant& s, float ideal, float* qf) {
    const float ix = clampf(ideal * s.scale - s.slb, 0.0f, 1.0f);
    const uint32_t wl = small_trunc(ix * s.qlm1), wh = min(wl + 1, s.top);
    const uint32_t li = (uint32_t)tb.q2u((int)(s.q2u_start + wl)), hi = (uint32_t)tb.q2u((int)(s.q2u_start + wh));
    const bool uh = small_float(li + hi) < (128.0f * ix);
    const uint32_t v = uh ? hi : li;
    *qf = small_float(v) * s.rscale + s.low;
    return v;
}

// Passes 02-05 for the decimation modes of a partitioned block: each step over items of all
// modes at once, a barrier between steps.  Items are (mode, weight) for pass02's sums, (mode,
// texel) for its infill, (mode, weight) for its correction, (mode, angular step) for passes 03
// and 04, (mode, quant level) for pass05.  The full search takes the first and the step items
// from the tables, sorted by their inner loop's length, so that a warp's lanes end together; a
// half-warp per mode, which this replaces, kept 16 of 32 lanes busy (a mode has 4 to 64 weights,
// 1 to 36 texels a weight and 2 to 12 steps).  The proposal search lists the items of its few modes itself.  The sums'
// entries are stored four to a load and, for the sorted items, 32 items side by side; the
// weights of all modes are packed, which with the steps kept in pass07's buffer takes a 10x8
// block from 70 to 51 KB of shared memory and from three to four CTAs.  Measured (B200, 128
// threads): passes 02-05 of 13,312 partitioned blocks at 10x8 3.04 -> 1.43 ms, at 8x8 3.18 ->
// 1.61 ms; with 32 threads 83,200 at 4x4 0.44 -> 0.41 ms.
template <int NT, bool DEEP>
__device__ __forceinline__ void dm_passes(const Tabs& tb, int T, int ndm_run, const int16_t* dm_run, int nw, int ns,
                                          const uint16_t* witems, const uint16_t* sitems, const float* iw,
                                          const float* wes, bool is_const, float* dec, uint16_t* trig, float* lov, float* hiv,
                                          float* buf) {
    const int tid = threadIdx.x;
    const int tmask = is_const ? 0 : -1;
    // item it's mode and weight, and its texel entries, `stride` fours apart
    const int stride = dm_run ? 1 : 32;
    auto weight_item = [&](int it, int& m, int& w, const uint4*& ent, int& n4) {
        uint32_t info;
        const int e = witems[it];
        m = e >> 6; w = e & 63;
        if (dm_run) {
            info = tb.wt_info(m, w);
            ent = tb.w2tf(info & 0xFFFF);
        } else {
            info = tb.wgroup(it >> 5);
            ent = tb.wgent(info & 0xFFFF) + (it & 31);
        }
        n4 = info >> 16;
    };
    // pass02: the ideal decimated weights (padding entries add 0 to sums that are never -0)
#pragma unroll 1
    for (int it = tid; it < nw; it += NT) {
        int m, w, n4;
        const uint4* ent;
        weight_item(it, m, w, ent, n4);
        const DevDm dmi = tb.dm(m);
        float v = iw[w];
        if (dmi.W != T) {
            float ws = 0.0f, tc = 1e-10f;
#pragma unroll (DEEP ? 2 : 1)
            for (; n4 > 0; n4--, ent += stride) {
                const uint4 e4 = *ent;
                const uint32_t e[4] = {e4.x, e4.y, e4.z, e4.w};
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const int t = entry_index(e[k]);
                    const float cwt = entry_factor(e[k]) * wes[t & tmask];
                    ws = ws + iw[t] * cwt;
                    tc = tc + cwt;
                }
            }
            v = ws / tc;
        }
        dec[dmi.w_off + w] = v;
    }
    __syncthreads();
    // the infilled weights less the ideal ones
    float* inf = buf;
    const uint32_t per_t = 0xFFFFFFFFu / (uint32_t)T + 1u;  // n / T is umulhi(n, per_t) for n < 2^16
#pragma unroll 1
    for (int it = tid; it < ndm_run * T; it += NT) {
        const int mi = (int)__umulhi((uint32_t)it, per_t), t = it - mi * T;
        const int m = dm_run ? dm_run[mi] : mi;
        const DevDm dmi = tb.dm(m);
        if (dmi.W == T) continue;
        // the texel's entries in list order; padding entries add dw[0] * 0, which never changes v
        const uint4 e = tb.tw4f(m, t);
        const float* dw = dec + dmi.w_off;
        float v = dw[entry_index(e.x)] * entry_factor(e.x);
        v = v + dw[entry_index(e.y)] * entry_factor(e.y);
        v = v + dw[entry_index(e.z)] * entry_factor(e.z);
        v = v + dw[entry_index(e.w)] * entry_factor(e.w);
        inf[m * T + t] = v - iw[t];
    }
    __syncthreads();
    // the one-step correction, and pass03's table rows (padded to a multiple of four weights with
    // the row of zeros, which changes no sum)
#pragma unroll 1
    for (int it = tid; it < nw; it += NT) {
        int m, w, n4;
        const uint4* ent;
        weight_item(it, m, w, ent, n4);
        const DevDm dmi = tb.dm(m);
        const int W = dmi.W;
        float v = dec[dmi.w_off + w];
        if (W != T) {
            const float* im = inf + m * T;
            float e0 = 1e-10f, e1 = 0.0f;
#pragma unroll (DEEP ? 2 : 1)
            for (; n4 > 0; n4--, ent += stride) {
                const uint4 e4 = *ent;
                const uint32_t e[4] = {e4.x, e4.y, e4.z, e4.w};
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const int t = entry_index(e[k]);
                    const float c = entry_factor(e[k]), sc = wes[t & tmask] * c;
                    e0 = e0 + c * sc;
                    e1 = e1 + im[t] * sc;
                }
            }
            v = v + clampf((e1 * -16.0f) / e0, -0.25f, 0.25f);
            dec[dmi.w_off + w] = v;
        }
        trig[dmi.w_off + w] = (uint16_t)(rn_bits(clampf(v, 0.0f, 1.0f) * (1024.0f - 1.0f)) * 16);
        if (w == W - 1)
            for (int p = W; p & 3; p++) trig[dmi.w_off + p] = 1024 * 16;
    }
    __syncthreads();
    // passes 03 and 04: the angular offset of a step, its rounding error and cut errors over
    // the weights, and its span
    float4* step_err = reinterpret_cast<float4*>(buf);  // e, e + low cut, e + high cut, e + both
    const int nstep = tb.L->ndm * kMaxAngularSteps;
    int2* step_span = reinterpret_cast<int2*>(buf + 4 * nstep);  // span, lowest index (float bits)
    float* ang = buf + 6 * nstep;
#pragma unroll 1
    for (int it = tid; it < ns; it += NT) {
        const int e = sitems[it], m = e >> 4, i = e & 15;
        const DevDm dmi = tb.dm(m);
        const int W = dmi.W;
        const float* dw = dec + dmi.w_off;
        const uint2* rows = reinterpret_cast<const uint2*>(trig + dmi.w_off);
        float ax = 0.0f, ay = 0.0f;
#pragma unroll (DEEP ? 4 : 2)
        for (int j = 0; j < W; j += 4) {  // four table values in flight, summed in weight order
            const uint2 k = rows[j >> 2];
            const float2 c0 = tb.trig((int)(k.x & 0xFFFF) + i), c1 = tb.trig((int)(k.x >> 16) + i);
            const float2 c2 = tb.trig((int)(k.y & 0xFFFF) + i), c3 = tb.trig((int)(k.y >> 16) + i);
            ax = ax + c0.x; ay = ay + c0.y;
            ax = ax + c1.x; ay = ay + c1.y;
            ax = ax + c2.x; ay = ay + c2.y;
            ax = ax + c3.x; ay = ay + c3.y;
        }
        const float off = atan2_search(ay, ax) * (1.0f / (2.0f * 3.14159265358979323846f));
        float mnw = 3.4e38f, mxw = -3.4e38f;
#pragma unroll 4
        for (int j = 0; j < W; j++) { const float v = dw[j]; mnw = fminf(mnw, v); mxw = fmaxf(mxw, v); }
        const float rcp = (float)(i + 1);
        const float minidx = rn_small(mnw * rcp - off), maxidx = rn_small(mxw * rcp - off);
        float ev = 0.0f, cl = 0.0f, ch = 0.0f;
#pragma unroll 2
        for (int j = 0; j < W; j++) {
            const float sv = dw[j] * rcp - off, r = rn_small(sv), d = sv - r, d2 = d + d;
            ev = ev + d * d;
            cl = cl + (r == minidx ? 1.0f - d2 : 0.0f);
            ch = ch + (r == maxidx ? 1.0f + d2 : 0.0f);
        }
        const int sp = min(max((int)rn_small((maxidx - minidx) + 1.0f), 2), (int)dmi.max_quant_steps + 3);
        const float ss = 1.0f / rcp, esc = ss * ss;
        const float err = ev * esc, ecl0 = cl * esc, ech0 = ch * esc;
        const int at = m * kMaxAngularSteps + i;
        step_err[at] = make_float4(err, err + ecl0, err + ech0, (err + ecl0) + ech0);
        step_span[at] = make_int2(sp, __float_as_int(minidx));
        ang[at] = off;
    }
    __syncthreads();
    // pass05: low/high value per quant level from the best step of its span.  The scan over
    // the steps updates span sp with e, sp - 1 with the low cut's error and then the high
    // cut's, sp - 2 with both cuts', each only when strictly below the span's best so far
    // (initially 1e37: step 0 and no low cut when nothing got below); an item runs it for
    // its own span.
#pragma unroll 1
    for (int it = tid; it < ndm_run * 8; it += NT) {
        const int m = dm_run ? dm_run[it >> 3] : it >> 3, q = it & 7;
        const DevDm dmi = tb.dm(m);
        float lo_v = 0.0f, hi_v = 0.0f;
        if (q <= (int)dmi.max_quant_level) {
            const int qs = c_steps_for_quant[q], S = dmi.max_angular_steps, at = m * kMaxAngularSteps;
            float best = 1e37f, lwi = __int_as_float(step_span[at].y);
            int bsi = 0;
#pragma unroll 1
            for (int i = 0; i < S; i++) {
                const float4 e = step_err[at + i];
                const int2 si = step_span[at + i];
                const int d = si.x - qs;
                const bool high = e.z < e.y;
                const float c = d == 0 ? e.x : d == 1 ? (high ? e.z : e.y) : d == 2 ? e.w : 3.4e38f;
                if (c < best) {
                    best = c;
                    bsi = i;
                    lwi = __int_as_float(si.y) + ((d == 2 || (d == 1 && !high)) ? 1.0f : 0.0f);
                }
            }
            const float hwi = (lwi + (float)qs) - 1.0f;
            const float step = 1.0f / (1.0f + (float)bsi);
            const float o = ang[at + bsi];
            lo_v = (o + lwi) * step;
            hi_v = (o + hwi) * step;
        }
        lov[m * 8 + q] = lo_v;
        hiv[m * 8 + q] = hi_v;
    }
}

// Code of the full search only (every block mode) is kept out of line, so that the
// proposal search's path through the front stays compact in the instruction cache (the
// front stalls on instruction fetch).
// pass07 over every block mode, one thread per mode.
template <int kFrontThreads, bool DEEP>
__device__ __noinline__ void pass07_all_modes(const Tabs& tb, int T, int P, int nbm, const float* lov, const float* hiv,
                                              float min_cutoff, const float* dec, float* qfs, const float* iw,
                                              const float* wes, bool is_const, float* bm_err) {
    const int tid = threadIdx.x;
    const int tmask = is_const ? 0 : -1;
    float* qw = qfs + tid;  // this thread's weights, kFrontThreads apart
    // one thread per mode; neighbouring threads get modes of the same decimation
#pragma unroll 1
    for (int j = tid; j < nbm; j += kFrontThreads) {
        const int i = tb.bm_order(j);
        const DevBm bm = tb.bm(i);
        const int bc = c_free_bits[P - 1] - (int)bm.weight_bits;
        if (bm.quant > 11 || bc <= 0) { bm_err[i] = 1e38f; continue; }
        const DevDm dmi = tb.dm(bm.dm);
        const int W = dmi.W;
        const BmQuant s = bm_quant_setup(tb, bm, lov + bm.dm * 8, hiv + bm.dm * 8, min_cutoff);
        const float* dw = dec + dmi.w_off;
#pragma unroll 2
        for (int w = 0; w < W; w++) { float qf; bm_quant_weight(tb, s, dw[w], &qf); qw[w * kFrontThreads] = qf; }
        float err = 0.0f;
        if (W == T) {  // one weight a texel, contribution 1
#pragma unroll 2
            for (int t = 0; t < T; t++) {
                const float d = qw[t * kFrontThreads] - iw[t];
                err = err + (d * d) * wes[t & tmask];
            }
        } else {
#pragma unroll (DEEP ? 4 : 2)
            for (int t = 0; t < T; t++) {
                const uint4 e = tb.tw4f(bm.dm, t);
                float v = qw[entry_index(e.x) * kFrontThreads] * entry_factor(e.x);
                v = v + qw[entry_index(e.y) * kFrontThreads] * entry_factor(e.y);
                v = v + qw[entry_index(e.z) * kFrontThreads] * entry_factor(e.z);
                v = v + qw[entry_index(e.w) * kFrontThreads] * entry_factor(e.w);
                const float d = v - iw[t];
                err = err + (d * d) * wes[t & tmask];
            }
        }
        bm_err[i] = err;
    }
}

// P1: the instance for partitioned blocks of one partition only (the proposal pass's P = 1
// list), with P a constant the compiler folds into every loop bound and branch.
template <int NT, bool P1, bool DEEP>
__device__ void front_body(const KernelArgs& a, const int P_arg, int lb, int blk, int slot_in_block, uint32_t entry, uint8_t* sm) {
    constexpr int kFrontThreads = NT, kFrontWarps = NT / 32;
    const int P = P1 ? 1 : P_arg;
    const Tabs tb{a.tables, &a.L};
    const int T = a.L.T, ndm = a.L.ndm, nbm = a.L.nbm;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const FrontLayout fl = front_layout(a.L, NT, a.bm_mask != nullptr, P1);
    float4* px = reinterpret_cast<float4*>(sm + fl.px);
    float* iw = reinterpret_cast<float*>(sm + fl.w);
    float* wes = reinterpret_cast<float*>(sm + fl.wes);
    uint8_t* tp = sm + fl.tp;
    float* dec = reinterpret_cast<float*>(sm + fl.dec);
    float* lov = reinterpret_cast<float*>(sm + fl.lo);
    float* hiv = reinterpret_cast<float*>(sm + fl.hi);
    float* bm_err = reinterpret_cast<float*>(sm + fl.bm_err);
    uint8_t* mode_ints = sm + fl.ints;  // pass11's integer count per block mode
    float* qfs = reinterpret_cast<float*>(sm + fl.qf);
    FrontMisc<P1>& M = *reinterpret_cast<FrontMisc<P1>*>(sm + fl.misc);
    const float4 cw = chan_w();
    // Partition bytes of texels t..t+3 (t a multiple of 4 below Tp) and of texel t < T.  With one
    // partition they are known, 0 for the block's texels and 0xFF (no partition) for the
    // padding ones, and are not read from shared memory.
    auto tp4 = [&](int t) -> uint32_t {
        if constexpr (P1) {
            uint32_t q = 0;
#pragma unroll
            for (int j = 0; j < 4; j++) q |= (t + j < T ? 0u : 0xFFu) << (8 * j);
            return q;
        } else {
            return *reinterpret_cast<const uint32_t*>(tp + t);
        }
    };
    auto tp1 = [&](int t) -> int {
        if constexpr (P1) return 0;
        else return tp[t];
    };

    // Per-partition sums over the texels are taken in ascending texel order, as the
    // oracle does, by one lane per (partition, channel or term) over the whole block:
    // texels of other partitions add +0.0f.  Every such sum starts at +0.0f and adds
    // terms that are never -0.0f, so it is never -0.0f and adding +0.0f leaves it
    // unchanged: the result is the member-only sum.  The lanes read four texels per
    // step (the block padded to Tp texels whose partition byte matches none).
    const int Tp = (T + 3) & ~3;
    float* pxc = qfs;           // [4][Tp] texel channels, until pass01 ends
    float* prj = qfs + 4 * Tp;  // [Tp] projections on the partition's direction, until iw is set
    float* terms = qfs;         // [5][Tp] pass08 error terms, until they are summed
    // Side work goes to the other warps first (role 0 is warp 1's lane 0); warp 0 takes
    // pass01's chain.  With one warp, roles are its lanes.
    const int role = (tid + kFrontThreads - 32) % kFrontThreads;

    const uint32_t* prow = P > 1 ? tb.part2(P, entry) : nullptr;
    const BlockSrc src = block_src(a, blk);
#pragma unroll 1
    for (int t = tid; t < Tp; t += kFrontThreads) {
        float4 v = mk(0.0f);
        uint8_t q = 0xFF;
        if (t < T) { v = src_texel(src, a.L.bx, t); q = P > 1 ? (prow[t >> 4] >> (2 * (t & 15))) & 3u : 0; px[t] = v; }
        pxc[t] = v.x; pxc[Tp + t] = v.y; pxc[2 * Tp + t] = v.z; pxc[3 * Tp + t] = v.w;
        tp[t] = q;
    }
    __syncthreads();
    // ---------------- pass01: per-partition average, direction, projections
    // lane 4p + c of warp 0 takes partition p, channel c (lanes 16-31 repeat 0-15); all four
    // partitions are computed whatever P is (empty ones feed is_const and min_cutoff)
    const int gp = (lane >> 2) & 3, gc = lane & 3;
    float avg_c = 0.0f;
    if (warp == 0) {
        const float* v = pxc + gc * Tp;
        float s = 0.0f;
        int n = 0;
#pragma unroll 1
        for (int t = 0; t < Tp; t += 4) {
            const float4 x = *reinterpret_cast<const float4*>(v + t);
            const uint32_t q = tp4(t);
            const bool m0 = (int)(q & 0xFF) == gp, m1 = (int)((q >> 8) & 0xFF) == gp;
            const bool m2 = (int)((q >> 16) & 0xFF) == gp, m3 = (int)(q >> 24) == gp;
            s = s + (m0 ? x.x : 0.0f); s = s + (m1 ? x.y : 0.0f);
            s = s + (m2 ? x.z : 0.0f); s = s + (m3 ? x.w : 0.0f);
            n += (int)m0 + (int)m1 + (int)m2 + (int)m3;
        }
        const float cnt = (float)n;  // the oracle's count of 1.0f additions, exact
        avg_c = cnt > 0.0f ? s / cnt : 0.0f;
        if (lane < 16) reinterpret_cast<float*>(&M.avg[gp])[gc] = avg_c;
    }
    __syncthreads();
    if (warp == 0) {
        const float* v = pxc + gc * Tp;
        float dd = 0.0f;
#pragma unroll 1
        for (int t = 0; t < Tp; t += 4) {
            const float4 x = *reinterpret_cast<const float4*>(v + t);
            const uint32_t q = tp4(t);
            const float p0 = fmaxf(x.x - avg_c, 0.0f), p1 = fmaxf(x.y - avg_c, 0.0f);
            const float p2 = fmaxf(x.z - avg_c, 0.0f), p3 = fmaxf(x.w - avg_c, 0.0f);
            dd = dd + ((int)(q & 0xFF) == gp ? p0 * p0 : 0.0f);
            dd = dd + ((int)((q >> 8) & 0xFF) == gp ? p1 * p1 : 0.0f);
            dd = dd + ((int)((q >> 16) & 0xFF) == gp ? p2 * p2 : 0.0f);
            dd = dd + ((int)(q >> 24) == gp ? p3 * p3 : 0.0f);
        }
        const int g0 = lane & ~3;
        const float4 avg = make_float4(__shfl_sync(FULL, avg_c, g0), __shfl_sync(FULL, avg_c, g0 + 1),
                                       __shfl_sync(FULL, avg_c, g0 + 2), __shfl_sync(FULL, avg_c, g0 + 3));
        const float4 d = normalize4(make_float4(__shfl_sync(FULL, dd, g0), __shfl_sync(FULL, dd, g0 + 1),
                                                __shfl_sync(FULL, dd, g0 + 2), __shfl_sync(FULL, dd, g0 + 3)));
        if (lane < 16 && gc == 0) M.dir[gp] = d;
        __syncwarp();
#pragma unroll 1
        for (int t = lane; t < Tp; t += 32) {
            float pr = 0.0f;
            if (t < T) { const int p = tp1(t); pr = dot4(px[t] - M.avg[p], M.dir[p]); }
            prj[t] = pr;
        }
        __syncwarp();
        // range of the projections, taken in texel order as the oracle does
        float mn = 1e10f, mx = -1e10f;
#pragma unroll 1
        for (int t = 0; t < Tp; t += 4) {
            const float4 x = *reinterpret_cast<const float4*>(prj + t);
            const uint32_t q = tp4(t);
            if ((int)(q & 0xFF) == gp) { mn = fminf(mn, x.x); mx = fmaxf(mx, x.x); }
            if ((int)((q >> 8) & 0xFF) == gp) { mn = fminf(mn, x.y); mx = fmaxf(mx, x.y); }
            if ((int)((q >> 16) & 0xFF) == gp) { mn = fminf(mn, x.z); mx = fmaxf(mx, x.z); }
            if ((int)(q >> 24) == gp) { mn = fminf(mn, x.w); mx = fmaxf(mx, x.w); }
        }
        if (mn >= mx) { mn = 0.0f; mx = 1e-7f; }
        const float len = mx - mn;
        const float lsq = len * len;
        float4 e0 = avg, e1 = avg;
        if (!(d.x == 0.0f && d.y == 0.0f && d.z == 0.0f && d.w == 0.0f)) { e0 = avg + d * mn; e1 = avg + d * mx; }
        if (lane < 16 && gc == 0) { M.lsq[gp] = lsq; M.mn[gp] = mn; M.mx[gp] = mx; M.ep0[gp] = e0; M.ep1[gp] = e1; }
        // min_cutoff: the smallest (1 - ep0) / ((ep1 - ep0) + 1e-9) above 0.5 over partitions and
        // channels (10 when none); lane 4p + c computes partition p, channel c, and the minimum
        // of these values (never NaN, never 0) does not depend on the order it is taken in
        const float e0c = comp(e0, gc), e1c = comp(e1, gc);
        const float epc = (1.0f - e0c) / ((e1c - e0c) + 1e-9f);
        float me = (lane < 16 && epc > 0.5f) ? epc : 10.0f;
        for (int o = 16; o > 0; o >>= 1) me = fminf(me, __shfl_xor_sync(FULL, me, o));
        const float l1 = __shfl_sync(FULL, lsq, 4), l2 = __shfl_sync(FULL, lsq, 8), l3 = __shfl_sync(FULL, lsq, 12);
        if (lane == 0) { M.min_cutoff = me; M.is_const = (l1 == lsq && l2 == lsq && l3 == lsq) ? 1u : 0u; }
    }
    // pass08, first part (needs only the averages): role 9p + 3s + c sums channel c of the
    // deviations from the average over the texels of partition p whose channel s is above it
#pragma unroll 1
    for (int v = role; v < 9 * P; v += kFrontThreads) {
        const int p = v / 9, s = (v / 3) % 3, c = v % 3;
        const float as = comp(M.avg[p], s), ac = comp(M.avg[p], c);
        const float* xs = pxc + s * Tp;
        const float* xc = pxc + c * Tp;
        float sum = 0.0f;
#pragma unroll 1
        for (int t = 0; t < Tp; t += 4) {
            const float4 vs = *reinterpret_cast<const float4*>(xs + t), vc = *reinterpret_cast<const float4*>(xc + t);
            const uint32_t q = tp4(t);
            sum = sum + (((int)(q & 0xFF) == p && vs.x - as > 0.0f) ? vc.x - ac : 0.0f);
            sum = sum + (((int)((q >> 8) & 0xFF) == p && vs.y - as > 0.0f) ? vc.y - ac : 0.0f);
            sum = sum + (((int)((q >> 16) & 0xFF) == p && vs.z - as > 0.0f) ? vc.z - ac : 0.0f);
            sum = sum + (((int)(q >> 24) == p && vs.w - as > 0.0f) ? vc.w - ac : 0.0f);
        }
        M.sxyz[p][s][c] = sum;
    }
    if (warp == kFrontWarps - 1) {
        bool gray = true, same_a = true;
#pragma unroll 1
        for (int t = lane; t < T; t += 32) {
            gray = gray && px[t].x == px[t].y && px[t].x == px[t].z;
            same_a = same_a && px[t].w == px[0].w;
        }
        gray = __all_sync(FULL, gray);
        same_a = __all_sync(FULL, same_a);
        if (lane == 0) { M.gray = gray; M.calpha = same_a; }
    }
    __syncthreads();
    const bool is_const = M.is_const != 0;
    const float ew = (((cw.x + cw.y) + cw.z) + cw.w) / 4.0f;
#pragma unroll 1
    for (int t = tid; t < T; t += kFrontThreads) {
        const int p = tp1(t);
        const float span = fmaxf(M.mx[p] - M.mn[p], 1e-6f);
        iw[t] = clampf((prj[t] - M.mn[p]) / span, 0.0f, 1.0f);
        wes[t] = M.lsq[p] * ew;
    }
    // pass08, second part: the encoding-choice axes of partition p (role p)
#pragma unroll 1
    for (int p = role; p < P; p += kFrontThreads) {
        const float4 sx = make_float4(M.sxyz[p][0][0], M.sxyz[p][0][1], M.sxyz[p][0][2], 0.0f);
        const float4 sy = make_float4(M.sxyz[p][1][0], M.sxyz[p][1][1], M.sxyz[p][1][2], 0.0f);
        const float4 sz = make_float4(M.sxyz[p][2][0], M.sxyz[p][2][1], M.sxyz[p][2][2], 0.0f);
        const float pxx = dot4(sx, sx), pyy = dot4(sy, sy), pzz = dot4(sz, sz);
        float4 bv = sx; float bs = pxx;
        if (pyy > bs) { bv = sy; bs = pyy; }
        if (pzz > bs) { bv = sz; bs = pzz; }
        float4 avg = M.avg[p]; avg.w = 0.0f;
        const float4 ub = normalize4(bv);
        const float4 lbv = normalize4(make_float4(1.0f, 1.0f, 1.0f, 0.0f));
        M.axes[p][0] = ub;
        M.axes[p][1] = avg - ub * dot4(avg, ub);
        M.axes[p][2] = normalize4(avg);
        M.axes[p][3] = avg - lbv * dot4(avg, lbv);
        const float4 e0 = M.ep0[p], e1 = M.ep1[p];
        const float lim = 0.12f * 65536.0f;
        M.ece_can_offset[p] = fabsf(e1.x - e0.x) < lim && fabsf(e1.y - e0.y) < lim && fabsf(e1.z - e0.z) < lim;
        M.ece_can_bc[p] = (M.gray && M.calpha) ? 0 : 1;
        // pass09 inputs of this partition; the 4 x 21 cells are filled later, one per role
        const float ps = (float)(P == 1 ? T : tb.part_count(P, entry, p));
        const float4 e0h = vmax(e0 - mk(65535.0f), mk(0.0f)), e1h = vmax(e1 - mk(65535.0f), mk(0.0f));
        const float4 e0l = vmin(e0, mk(0.0f)), e1l = vmin(e1, mk(0.0f));
        const float4 sre = ((e0l * e0l + e1l * e1l) + e0h * e0h) + e1h * e1h;
        M.p9[p][0] = (dot3(sre, cw) * 0.5f) * ps;
        M.p9[p][1] = ((sre.w * cw.w) * 0.5f) * ps;
        M.p9[p][2] = ((cw.x + cw.y) + cw.z) * ps;
        M.p9[p][3] = cw.w * ps;
    }

    // Block-mode subset of the proposal search: only its modes and their
    // decimation modes are evaluated; the others never become candidates.
    const uint64_t* bmm = a.bm_mask ? a.bm_mask + ((size_t)lb * 4 + (P - 1)) * kMaskWords : nullptr;
    uint32_t* flags = reinterpret_cast<uint32_t*>(sm + fl.dml);  // 4 words: one bit per decimation mode
    int16_t* list = reinterpret_cast<int16_t*>(sm + fl.dml + 16);
    uint16_t* witems = reinterpret_cast<uint16_t*>(sm + fl.witem);
    uint16_t* sitems = reinterpret_cast<uint16_t*>(sm + fl.sitem);
    if (bmm && tid < 4) flags[tid] = 0;
    __syncthreads();
    int16_t* blist = reinterpret_cast<int16_t*>(sm + fl.bml);
    if (bmm) {
#pragma unroll 1
        for (int i = tid; i < nbm; i += kFrontThreads)
            if ((bmm[i >> 6] >> (i & 63)) & 1) { const int d = tb.bm(i).dm; atomicOr(&flags[d >> 5], 1u << (d & 31)); }
        if (warp == 0) {  // the masked block modes in ascending order: each 32-bit half word is its own ballot
            int n = 0;
#pragma unroll 1
            for (int i0 = 0; i0 < nbm; i0 += 32) {
                uint32_t b = (uint32_t)(bmm[i0 >> 6] >> (i0 & 63));
                if (nbm - i0 < 32) b &= (1u << (nbm - i0)) - 1u;
                if ((b >> lane) & 1u) blist[n + __popc(b & ((1u << lane) - 1u))] = (int16_t)(i0 + lane);
                n += __popc(b);
            }
            if (lane == 0) M.nlive = n;
        }
    }
    // pass08 error terms of every texel against its partition's axes
#pragma unroll 1
    for (int t = tid; t < Tp; t += kFrontThreads) {
        float t0 = 0.0f, t1 = 0.0f, t2 = 0.0f, t3 = 0.0f, t4 = 0.0f;
        if (t < T) {
            const int p = tp1(t);
            const float4 ub = M.axes[p][0], ua = M.axes[p][1], sb = M.axes[p][2], la = M.axes[p][3];
            const float4 lbv = normalize4(make_float4(1.0f, 1.0f, 1.0f, 0.0f));
            float4 rgb = px[t]; rgb.w = 0.0f;
            const float ad = px[t].w - 65536.0f;
            t0 = (ad * ad) * cw.w;
            const float4 du = (ua + ub * dot3(rgb, ub)) - rgb;
            t1 = dot3(du * du, cw);
            const float4 ds = sb * dot3(rgb, sb) - rgb;
            t2 = dot3(ds * ds, cw);
            const float4 dl = (la + lbv * dot3(rgb, lbv)) - rgb;
            t3 = dot3(dl * dl, cw);
            const float4 dn = lbv * dot3(rgb, lbv) - rgb;
            t4 = dot3(dn * dn, cw);
        }
        terms[t] = t0; terms[Tp + t] = t1; terms[2 * Tp + t] = t2; terms[3 * Tp + t] = t3; terms[4 * Tp + t] = t4;
    }
    __syncthreads();
    // the decimation modes to run (warp 0): the decimated ones first, whose pass02 makes them
    // the longest, so that the warps taking them in turn finish closer together; pass08
    // sums (role 5p + k)
    if (bmm && warp == 0) {
        int n = 0;
#pragma unroll 1
        for (int pass = 0; pass < 2; pass++)
#pragma unroll 1
            for (int d0 = 0; d0 < ndm; d0 += 32) {
                const int d = d0 + lane;
                const bool f = d < ndm && ((flags[d >> 5] >> (d & 31)) & 1) && ((tb.dm(d).W == T) == (pass == 1));
                const uint32_t b = __ballot_sync(FULL, f);
                if (f) list[n + __popc(b & ((1u << lane) - 1))] = (int16_t)d;
                n += __popc(b);
            }
        __syncwarp();
        int nw = 0, ns = 0;  // their weights and angular steps as dm_passes' items
#pragma unroll 1
        for (int i = 0; i < n; i++) {
            const int d = list[i];
            const DevDm dmi = tb.dm(d);
            for (int w = lane; w < (int)dmi.W; w += 32) witems[nw + w] = (uint16_t)(d << 6 | w);
            if (lane < (int)dmi.max_angular_steps) sitems[ns + lane] = (uint16_t)(d << 4 | lane);
            nw += dmi.W;
            ns += dmi.max_angular_steps;
        }
        if (lane == 0) { flags[0] = n; flags[1] = nw; flags[2] = ns; }  // the flags are no longer needed
    }
#pragma unroll 1
    for (int v = role; v < 5 * P; v += kFrontThreads) {
        const int p = v / 5, k = v % 5;
        const float* x = terms + k * Tp;
        float s = 0.0f;
#pragma unroll 1
        for (int t = 0; t < Tp; t += 4) {
            const float4 y = *reinterpret_cast<const float4*>(x + t);
            const uint32_t q = tp4(t);
            s = s + ((int)(q & 0xFF) == p ? y.x : 0.0f); s = s + ((int)((q >> 8) & 0xFF) == p ? y.y : 0.0f);
            s = s + ((int)((q >> 16) & 0xFF) == p ? y.z : 0.0f); s = s + ((int)(q >> 24) == p ? y.w : 0.0f);
        }
        M.acc[p][k] = s;
    }
    __syncthreads();
    const int ndm_run = bmm ? (int)flags[0] : ndm;
    const int16_t* dm_run = bmm ? list : nullptr;
    // ---------------- pass09: colour error per partition, quant level and integer count
    // (role 17p + level; runs beside passes 02-05, which do not read it)
#pragma unroll 1
    for (int c = role; c < P * kColourLevels; c += kFrontThreads) {
        const int p = c / kColourLevels, i = c % kColourLevels;
        const float rre = M.p9[p][0], are = M.p9[p][1], brgb = M.p9[p][2], ba = M.p9[p][3];
        const bool cbc = M.ece_can_bc[p] == 1, coe = M.ece_can_offset[p] == 1;
        const float bcrgba = cbc ? 0.625f : 1.0f, oergba = coe ? 0.5f : 1.0f, bcrgb = cbc ? 0.5f : 1.0f, oergb = coe ? 0.25f : 1.0f;
        const float acc0 = M.acc[p][0], acc1 = M.acc[p][1], acc2 = M.acc[p][2], acc4 = M.acc[p][4];
        const float rgbs_e = (acc2 - acc1) * 0.7f, lum_e = (acc4 - acc1) * 3.0f, ad_e = acc0 * 3.0f;
        const float orgba = i >= 15 ? 1.0f : oergba, orgb = i >= 15 ? 1.0f : oergb;
        const float bq = tb.bqe(i);
        const float qrgb = brgb * bq, qrgba = (brgb + ba) * bq;
        M.cerr[p][i][3] = (((qrgba * bcrgba) * orgba) + rre) + are; M.cfmt[p][i][3] = FMT_RGBA;
        const float full = (((qrgb * bcrgb) * orgb) + rre) + ad_e;
        const float rgbsa = ((qrgba + rgbs_e) + rre) + are;
        if (rgbsa < full) { M.cerr[p][i][2] = rgbsa; M.cfmt[p][i][2] = FMT_RGB_SCALE_ALPHA; }
        else { M.cerr[p][i][2] = full; M.cfmt[p][i][2] = FMT_RGB; }
        const float lrgbs = ((qrgb + rre) + ad_e) + rgbs_e;
        const float la_e = ((qrgba + rre) + are) + lum_e;
        if (lrgbs < la_e) { M.cerr[p][i][1] = lrgbs; M.cfmt[p][i][1] = FMT_RGB_SCALE; }
        else { M.cerr[p][i][1] = la_e; M.cfmt[p][i][1] = FMT_LUMINANCE_ALPHA; }
        M.cerr[p][i][0] = ((qrgb + rre) + ad_e) + lum_e; M.cfmt[p][i][0] = FMT_LUMINANCE;
    }

    // ---------------- passes 02-05
    dm_passes<NT, DEEP>(tb, T, ndm_run, dm_run, bmm ? (int)flags[1] : a.L.nwi, bmm ? (int)flags[2] : a.L.nsi, bmm ? witems : tb.witems(),
                        bmm ? sitems : tb.sitems(), iw, wes, is_const, dec, reinterpret_cast<uint16_t*>(sm + fl.trig), lov, hiv, qfs);
    __syncthreads();

    // ---------------- pass07: weight quantisation error per block mode
    const int nlist = bmm ? M.nlive : nbm;  // block modes evaluated: the list, or all of them
    if (!bmm) pass07_all_modes<kFrontThreads, DEEP>(tb, T, P, nbm, lov, hiv, M.min_cutoff, dec, qfs, iw, wes, is_const, bm_err);
    // ---------------- pass10: best format combination per quant level and integer total
    // One item per (quant level, integer total), beside pass07 (role-indexed): the format
    // combinations with that total, in the order the one-thread loops visit them (i, j, k, l
    // ascending, each format class within one of the others), so the first minimum is the same.
    if (P > 1) {
        const int NC = P == 2 ? 7 : P == 3 ? 10 : 13;
#pragma unroll 1
        for (int it = role; it < kColourLevels * NC; it += kFrontThreads) {
            const int q = it / NC, c = it - q * NC;
            float be = ERR_DEFAULT;
            uint32_t bf = 0;
#pragma unroll 1
            for (int o = c_combo_off[P - 2][c]; o < c_combo_off[P - 2][c + 1]; o++) {
                const uint32_t cb = c_combo[o];
                const int i = cb & 3, j = (cb >> 2) & 3, k = (cb >> 4) & 3, l = cb >> 6;
                float e;
                if (P == 2) e = fminf(M.cerr[0][q][i] + M.cerr[1][q][j], 1e10f);
                else if (P == 3) e = fminf((M.cerr[0][q][i] + M.cerr[1][q][j]) + M.cerr[2][q][k], 1e10f);
                else e = fminf(((M.cerr[0][q][i] + M.cerr[1][q][j]) + M.cerr[2][q][k]) + M.cerr[3][q][l], 1e10f);
                if (e < be) { be = e; bf = cb; }
            }
            M.combo_err[q][c] = be;
            uint8_t* f = M.combo_fmt[q][c];
            f[0] = M.cfmt[0][q][bf & 3]; f[1] = M.cfmt[1][q][(bf >> 2) & 3];
            f[2] = P > 2 ? M.cfmt[2][q][(bf >> 4) & 3] : 0;
            f[3] = P > 3 ? M.cfmt[3][q][bf >> 6] : 0;
        }
    }
    if (bmm) {
        // The proposal search's few block modes, in groups that fit the buffer: the quantised
        // weights (one thread per mode and weight), the error terms (one per mode and
        // texel), then each mode's sum in texel order (padding texels add +0.0f to a sum of
        // non-negative terms).  Each value is the one-thread-per-mode loop's.
        const int mw = a.L.max_w;
        const int qf_floats = front_layout_qf_floats(T, mw, kFrontThreads, true);
        const int G = qf_floats / (mw + Tp);
        float* qw = qfs;           // [G][mw]
        float* et = qfs + G * mw;  // [G][Tp]
        float4* setup = reinterpret_cast<float4*>(sm + fl.setup);  // [G][2]; last word: weights (0: a mode that cannot be used) |
                                                                   // first weight << 8 | decimation mode << 24
        const uint32_t per_w = 0xFFFFFFFFu / (uint32_t)mw + 1u, per_t = 0xFFFFFFFFu / (uint32_t)Tp + 1u;  // n / mw is umulhi(n, per_w)
#pragma unroll 1
        for (int g0 = 0; g0 < nlist; g0 += G) {
            const int g = min(G, nlist - g0);
#pragma unroll 1
            for (int k = tid; k < g; k += kFrontThreads) {
                const DevBm bm = tb.bm(blist[g0 + k]);
                const bool usable = bm.quant <= 11 && c_free_bits[P - 1] > (int)bm.weight_bits;
                BmQuant s{};
                const DevDm dmi = tb.dm(bm.dm);
                if (usable) s = bm_quant_setup(tb, bm, lov + bm.dm * 8, hiv + bm.dm * 8, M.min_cutoff);
                setup[2 * k] = make_float4(s.low, s.scale, s.slb, s.rscale);
                setup[2 * k + 1] = make_float4(s.qlm1, __uint_as_float(s.q2u_start), __uint_as_float(s.top),
                                               __uint_as_float(usable ? (uint32_t)dmi.W | (uint32_t)dmi.w_off << 8 | (uint32_t)bm.dm << 24 : 0u));
            }
            __syncthreads();
#pragma unroll 1
            for (int it = tid; it < g * mw; it += kFrontThreads) {
                const int k = (int)__umulhi((uint32_t)it, per_w), w = it - k * mw;
                const float4 b = setup[2 * k + 1];
                const uint32_t wd = __float_as_uint(b.w);
                if (w >= (int)(wd & 0xFF)) continue;
                const float4 q = setup[2 * k];
                const BmQuant s{q.x, q.y, q.z, q.w, b.x, __float_as_uint(b.y), __float_as_uint(b.z)};
                bm_quant_weight(tb, s, dec[((wd >> 8) & 0xFFFF) + w], &qw[k * mw + w]);
            }
            __syncthreads();
#pragma unroll 1
            for (int it = tid; it < g * Tp; it += kFrontThreads) {
                const int k = (int)__umulhi((uint32_t)it, per_t), t = it - k * Tp;
                const uint32_t wd = __float_as_uint(setup[2 * k + 1].w);
                float term = 0.0f;
                if (t < T && wd != 0) {
                    const uint4 e = tb.tw4f((int)(wd >> 24), t);
                    const float* qk = qw + k * mw;
                    float v = qk[entry_index(e.x)] * entry_factor(e.x);
                    v = v + qk[entry_index(e.y)] * entry_factor(e.y);
                    v = v + qk[entry_index(e.z)] * entry_factor(e.z);
                    v = v + qk[entry_index(e.w)] * entry_factor(e.w);
                    const float d = v - iw[t];
                    term = (d * d) * wes[is_const ? 0 : t];
                }
                et[k * Tp + t] = term;
            }
            __syncthreads();
            // (the next group's setups follow a barrier, its weights are not read here)
#pragma unroll 1
            for (int k = tid; k < g; k += kFrontThreads) {
                const int i = blist[g0 + k];
                if (__float_as_uint(setup[2 * k + 1].w) == 0) { bm_err[i] = 1e38f; continue; }
                const float* x = et + k * Tp;
                float err = 0.0f;
#pragma unroll 1
                for (int t = 0; t < Tp; t += 4) {
                    const float4 y = *reinterpret_cast<const float4*>(x + t);
                    err = err + y.x; err = err + y.y; err = err + y.z; err = err + y.w;
                }
                bm_err[i] = err;
            }
            if (g0 + G < nlist) __syncthreads();
        }
    }
    __syncthreads();
    // ---------------- pass11: best colour combination per block mode, its error added to the
    // weights'
#pragma unroll 1
    for (int k = tid; k < nlist; k += kFrontThreads) {
        const int i = bmm ? blist[k] : k;
        const float werr = bm_err[i];
        if (werr >= ERR_DEFAULT) { bm_err[i] = ERR_DEFAULT; continue; }
        const int bits = c_free_bits[P - 1] - (int)tb.bm(i).weight_bits;
        const int lo = P == 1 ? 1 : P, hi = P == 1 ? 4 : P == 2 ? 8 : 9;
        float best = ERR_DEFAULT;
        int ints = 0;
#pragma unroll 1
        for (int ic = lo; ic <= hi; ic++) {
            const int ql = tb.qmt(ic, bits);
            if (ql < 4) { if (P == 1) continue; break; }
            const float e = P == 1 ? M.cerr[0][ql - 4][ic - 1] : M.combo_err[ql - 4][ic - P];
            if (e < best) { best = e; ints = ic; }
        }
        bm_err[i] = best + werr;
        mode_ints[i] = (uint8_t)ints;
    }
    __syncthreads();
    // ---------------- pass12: the 8 best trials (first minimum wins ties)
    // warp 0 picks them in order: each round the (error, index)-smallest mode after the
    // previous pick
    if (warp == 0 && bmm && nlist <= 32) {
        // up to 32 listed modes, one per lane: a usable mode's pick position is the number
        // of usable modes before it in (error, index) order
        const int i = lane < nlist ? blist[lane] : 0x7FFFFFFF;
        const float e = lane < nlist ? bm_err[i] : ERR_DEFAULT;
        const bool ok = e < ERR_DEFAULT;
        int rank = 0;
#pragma unroll 1
        for (int j = 0; j < nlist; j++) {
            const float ej = __shfl_sync(FULL, e, j);
            const int ij = __shfl_sync(FULL, i, j);
            rank += (ej < ERR_DEFAULT && (ej < e || (ej == e && ij < i))) ? 1 : 0;
        }
        const int nok = __popc(__ballot_sync(FULL, ok));
        if (ok && rank < kNumCand) M.top[rank] = i;
        if (lane >= nok && lane < kNumCand) M.top[lane] = -1;
    } else if (warp == 0) {
        // each lane keeps the best of its own modes (in a key that orders like the error) and
        // looks for its next one only when its best was picked
        uint32_t mine = 0xFFFFFFFFu;
        int mi = 0x7FFFFFFF;
        float pv = -3.4e38f;  // the lane's last pick
        int pi = -1;
        bool look = true;
#pragma unroll 1
        for (int r = 0; r < kNumCand; r++) {
            if (look) {
                float be = ERR_DEFAULT;
                mi = 0x7FFFFFFF;
#pragma unroll 1
                for (int k = lane; k < nlist; k += 32) {
                    const int i = bmm ? blist[k] : k;
                    const float e = bm_err[i];
                    if (e < be && (e > pv || (e == pv && i > pi))) { be = e; mi = i; }  // a lane's modes ascend
                }
                const uint32_t u = fbits(be + 0.0f);
                mine = mi == 0x7FFFFFFF ? 0xFFFFFFFFu : ((u & 0x80000000u) ? ~u : (u | 0x80000000u));
                pv = be;
                look = false;
            }
            const uint32_t best = __reduce_min_sync(FULL, mine);
            if (best == 0xFFFFFFFFu) {  // fewer than kNumCand usable modes
                if (lane >= r && lane < kNumCand) M.top[lane] = -1;
                break;
            }
            const uint32_t bi = __reduce_min_sync(FULL, mine == best ? (uint32_t)mi : 0xFFFFFFFFu);
            if (lane == 0) M.top[r] = (int)bi;
            if ((uint32_t)mi == bi) { pi = mi; look = true; }
        }
    }
    __syncthreads();
    PBRec& rec = a.pbrec[(size_t)lb * a.slots + slot_in_block];
    if (a.work && tid == 0) {
        int nbm_run = nbm;
        if (bmm) {
            nbm_run = 0;
#pragma unroll 1
            for (int w = 0; w < kMaskWords; w++) {
                const int lo = w * 64;
                if (lo >= nbm) break;
                const uint64_t valid = nbm - lo >= 64 ? ~0ull : ((1ull << (nbm - lo)) - 1);
                nbm_run += __popcll(bmm[w] & valid);
            }
        }
        atomicAdd(a.work + (P - 1), 1ull);
        atomicAdd(a.work + 4, (unsigned long long)ndm_run);
        atomicAdd(a.work + 5, (unsigned long long)nbm_run);
    }
    if (tid == 0) {
        int n = 0;
        while (n < a.topn && M.top[n] >= 0) n++;
        M.ncand = n;
        rec.P = P; rec.entry = entry; rec.ncand = n;
        rec.seed = P > 1 ? tb.part_seed(P, entry) : 0;
    }
    if (tid < 4) { rec.avg[tid] = M.avg[tid]; rec.ep0[tid] = M.ep0[tid]; rec.ep1[tid] = M.ep1[tid]; }
    __syncthreads();
    // candidate initial state: the trial's quantised weights (REF-BUG-6: only
    // floor(W/4)*4 weights are packed by pass07, the rest read as 0; FIXED semantics: all W)
    const int ncand = M.ncand;
#pragma unroll 1
    for (int k = tid >> 3; k < ncand; k += kFrontThreads / 8) {
        const int i = M.top[k];
        const DevBm bm = tb.bm(i);
        const DevDm dmi = tb.dm(bm.dm);
        CandInit& c = rec.c[k];
        if ((tid & 7) == 0) {
            const int bits = c_free_bits[P - 1] - (int)bm.weight_bits, ints = mode_ints[i];
            const int ql = tb.qmt(ints, bits), qlm = P == 1 ? ql : tb.qmt(ints, bits + (P == 2 ? 2 : P == 3 ? 5 : 8));
            uint32_t fmt = 0;
            if (P == 1) fmt = ql >= 4 ? M.cfmt[0][ql - 4][ints - 1] : (uint32_t)FMT_LUMINANCE;
            else if (ql >= 4) fmt = *reinterpret_cast<const uint32_t*>(M.combo_fmt[ql - 4][ints - P]);
            // bm, ql, qlm and the four formats: 8-byte aligned in PBRec
            *reinterpret_cast<uint2*>(&c) = make_uint2((uint32_t)i | (uint32_t)(ql & 0xFF) << 16 | (uint32_t)(qlm & 0xFF) << 24, fmt);
        }
        const BmQuant s = bm_quant_setup(tb, bm, lov + bm.dm * 8, hiv + bm.dm * 8, M.min_cutoff);
        const int packed_w = a.fixed ? dmi.W : (dmi.W / 4) * 4;
        const float* dw = dec + dmi.w_off;
#pragma unroll 1
        for (int j = tid & 7; j < 16; j += 8) {  // four weights a word
            uint32_t word = 0;
#pragma unroll 1
            for (int w = 4 * j; w < min(4 * j + 4, packed_w); w++) {
                float qf;
                word |= bm_quant_weight(tb, s, dw[w], &qf) << (8 * (w & 3));
            }
            reinterpret_cast<uint32_t*>(c.qw)[j] = word;
        }
    }
}

// Resident CTAs of 128 threads the register budget is sized for.
constexpr int kFrontMinBlocks128 = 8;
// DEEP: the instances for blocks of kDeepTexels or more, of which shared memory leaves four CTAs of
// 128 threads or fewer: they wait for table loads, so the loops around those are unrolled into the
// registers that are free.  Measured (B200, 2,048 blocks) without / with: 8x6 2.48 / 2.64 ms, 8x8 5.00 /
// 4.61, 10x8 6.71 / 6.06, 12x12 15.3 / 13.4; 6x6 1.52 / 1.79.
constexpr int kDeepTexels = 60;
constexpr int front_min_ctas(int nt, bool deep) {
    return deep ? (nt >= 256 ? 2 : 5) : kFrontMinBlocks128 * 128 / nt > 32 ? 32 : kFrontMinBlocks128 * 128 / nt;
}
template <int NT, bool P1, bool DEEP>
__global__ void __launch_bounds__(NT, front_min_ctas(NT, DEEP)) k_front(const __grid_constant__ KernelArgs a) {
    extern __shared__ __align__(16) uint8_t smem[];
    // Items: every slot of every block in slot-major order (co-resident CTAs work on the
    // same partition count), or the proposal pass's work list grouped by partition count.
    const int nb = list_blocks(a);
    const int items = a.pb_list ? pb_total(a) : nb * a.slots;
    for (int li = blockIdx.x; li < items; li += gridDim.x) {
        int k, lb;
        if (a.pb_list) pb_item(a, li, lb, k);
        else { k = li / nb; lb = li % nb; }
        const int blk = chunk_block(a, lb);
        int P = 1, entry = 0;
        bool present = true;
        if (k > 0 && a.prop) {
            const PropPicks& pp = a.prop[lb];
            present = k - 1 < (int)pp.n;
            const int v = present ? pp.v[k - 1] : 0;
            P = 2 + (v >> 10); entry = v & 1023;
        } else if (k > 0) {
            P = 2 + (k - 1) / 4;
            const uint16_t* pk = a.picks[lb].v + (P - 2) * 5;
            const int i = (k - 1) % 4;
            present = i < pk[4];
            entry = present ? pk[i] : 0;
        }
        if (!present) {
            if (threadIdx.x == 0) { PBRec& rec = a.pbrec[(size_t)lb * a.slots + k]; rec.P = P; rec.ncand = 0; rec.entry = 0; rec.seed = 0; }
            continue;  // uniform across the CTA
        }
        front_body<NT, P1, DEEP>(a, P, lb, blk, k, entry, smem);
        __syncthreads();  // the next item reuses shared memory
    }
}

}  // namespace

// Threads per partitioned block.  Small blocks have few items per step (4x4: 6 decimation
// modes, 53 block modes), so one warp, whose barriers are cheap and of which more are resident,
// is fastest; large ones hold enough for more, and their shared memory, the same for any
// number of threads but for pass07's weights, limits the resident CTAs to two or three.
// Measured (B200, 2,048 blocks, all 13 partitioned blocks), 32 / 64 / 128 / 256 threads, in us: 4x4
// 411 / 465 / 567 / 995, 5x4 584 / 651 / 680 / 1110, 5x5 928 / 895 / 893 / 1304, 6x6 2198 / 1616 /
// 1542 / 1836, 10x8 15259 / 8785 / 6768 / 8017, 12x10 40427 / 21252 / 12438 / 11803, 12x12 74917 /
// 40147 / 23795 / 15542.  Proposal search's lists of 1024x1024: 4x4 861 / 1060 / 1377, 6x6 712 / 669
// / 720.  A launch that leaves SMs without a warp is as long as one item: 128 threads then.  (Full searches
// of 1 to 45 blocks with 256 there instead: 12x12 5 to 8 % less; 12x10 4 to 8 % less, but 4 % more for 32
// blocks; 10x10 5 % less up to 16 blocks, 4 % more from 32.)
static int front_nt(int T, bool list, int items) {
    if (items < 148 * 4) return 128;
    if (T <= 20) return 32;
    if (list) return 64;
    return T >= 120 ? 256 : 128;
}
static int front_nt(const KernelArgs& a) {
    if (a.front_threads == 32 || a.front_threads == 64 || a.front_threads == 128) return a.front_threads;
    return front_nt(a.L.T, a.bm_mask != nullptr, a.nblocks * a.slots);
}

size_t search_smem_bytes(const TableLayout& L) { return (size_t)kSearchWarps * search_layout(L.T).total; }
static size_t front_smem_bytes(const TableLayout& L, int nt, bool list, bool p1) { return (size_t)front_layout(L, nt, list, p1).total; }
size_t front_smem_bytes(const TableLayout& L) {  // the largest over the launches of this footprint
    return std::max(front_smem_bytes(L, 128, false, false), front_smem_bytes(L, front_nt(L.T, false, 1 << 30), false, false));
}

cudaError_t configure_search_kernels(size_t search_bytes, size_t front_bytes) {
    cudaError_t e = cudaFuncSetAttribute(k_partition_search, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)search_bytes);
    // the largest shared-memory carveout: occupancy of the front is bounded by shared memory
    for (auto f : {k_front<256, false, true>, k_front<128, false, true>, k_front<128, false, false>, k_front<64, false, false>,
                   k_front<32, false, false>, k_front<128, true, false>, k_front<64, true, false>, k_front<32, true, false>}) {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)front_bytes);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    }
    return e;
}

cudaError_t launch_partition_search(const KernelArgs& a, cudaStream_t s) {
    const int items = a.nblocks * 3;
    int grid = search_wide(items) ? items : (items + kSearchWarps - 1) / kSearchWarps;
    if (a.block_list) grid = std::min(items, kListGridSearch);
    k_partition_search<<<grid, kSearchWarps * 32, search_smem_bytes(a.L), s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_front(const KernelArgs& a, cudaStream_t s, int* launched) {
    const int nt = front_nt(a);
    int grid = a.nblocks * a.slots;
    if (a.block_list) grid = std::min(grid, kListGridFront * 128 / nt);
    auto go = [&](const KernelArgs& k, bool p1) {
        if (launched) ++*launched;
        const size_t smem = front_smem_bytes(a.L, nt, a.bm_mask != nullptr, p1);
        if (nt == 32) { if (p1) k_front<32, true, false><<<grid, 32, smem, s>>>(k); else k_front<32, false, false><<<grid, 32, smem, s>>>(k); }
        else if (nt == 64) { if (p1) k_front<64, true, false><<<grid, 64, smem, s>>>(k); else k_front<64, false, false><<<grid, 64, smem, s>>>(k); }
        else if (nt == 256) k_front<256, false, true><<<grid, 256, smem, s>>>(k);
        else if (p1) k_front<128, true, false><<<grid, 128, smem, s>>>(k);
        else if (a.L.T >= kDeepTexels) k_front<128, false, true><<<grid, 128, smem, s>>>(k);
        else k_front<128, false, false><<<grid, 128, smem, s>>>(k);
    };
    if (a.pb_list && a.pb_from == 0 && a.pb_to == 0) {
        // the proposal pass's work lists: P = 1 by its own instance, then P = 2..4
        KernelArgs k1 = a, k2 = a;
        k1.pb_from = 0; k1.pb_to = 1;
        k2.pb_from = 1; k2.pb_to = 4;
        go(k1, true);
        go(k2, false);
    } else {
        go(a, false);
    }
    return cudaGetLastError();
}

}  // namespace astcb200
