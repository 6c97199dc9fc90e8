// Training kernels of the proposal network (FP32 throughout, deterministic:
// every output element is summed in a fixed order).
//
//   k_gemm      C = A . B (+ bias) (ReLU), A and B addressed by arbitrary row and
//               column strides, so forward (X W^T), input gradient (dY W) and
//               weight gradient (dY^T X) are the same kernel; k_gemm_short for
//               products of few terms.
//   k_xent      softmax cross-entropy of the partition head (all valid
//               partitionings and the single-partition class) plus that of the
//               block-mode head of the label's partition count; writes dZ
//               (already divided by the batch) and the two losses per row.
//   k_relu_bwd, k_colsum (bias gradients), k_adam.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "astcb200.h"
#include "mlp.h"

namespace astcb200 {
namespace {

namespace cg = cooperative_groups;

// 128x64 tiles, 16-deep K slices double-buffered in shared memory, 8x8 outputs a thread of 128:
// four 16-byte shared loads for 64 multiply-adds, so the FP32 pipe is the bound.  The network's
// products have few tiles (a 256x256 gradient eight) and long sums (2,048 rows), so K is split
// over the CTAs of a thread-block cluster (at most 8, as many as fill the GPU), whose partial
// tiles are added in rank order through distributed shared memory: no workspace, and the order
// depends on the shape only.  Measured (B200, one step at 4x4, 2,048 rows): one 64x64 tile a CTA
// without a split and 4x4 outputs a thread 743 us, this with k_gemm_short and k_colsum below 186 us.
constexpr int kBM = 128, kBN = 64, kBK = 16, kGemmThreads = 128;
constexpr int kMaxSplit = 8, kSplitK = 2 * 4 * kBK;  // terms from which a sum is split
constexpr int kRowA = kBM + 4, kRowB = kBN + 4;  // floats of a K row in shared memory
constexpr int kStageFloats = kBK * (kRowA + kRowB);

// Loads a `rows` x kBK slice (rows along the stride s_r, K along s_k) of a matrix of n_r x n_k, zeros
// outside, into registers: kind 0 four floats along K, 1 four along the rows, 2 and 3 single floats,
// consecutive threads on consecutive rows or on consecutive fours of a row.
template <int ROWS>
struct Slice {
    static constexpr int kVec = ROWS * kBK / 4 / kGemmThreads;
    float4 v[kVec];
    __device__ __forceinline__ void load(const float* __restrict__ p, int kind, int r0, int k0, int n_r, int n_k, long long s_r, long long s_k) {
#pragma unroll
        for (int j = 0; j < kVec; j++) {
            const int e = threadIdx.x + j * kGemmThreads;
            // along K: consecutive threads on consecutive fours of a row; else on consecutive rows
            const int r = r0 + (kind == 1 ? (e % (ROWS / 4)) * 4 : kind != 2 ? e / (kBK / 4) : e % ROWS);
            const int k = k0 + (kind == 1 ? e / (ROWS / 4) : kind != 2 ? (e % (kBK / 4)) * 4 : (e / ROWS) * 4);
            float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (kind >= 2) {
                if (r < n_r) {
                    if (k < n_k) x.x = p[r * s_r + k * s_k];
                    if (k + 1 < n_k) x.y = p[r * s_r + (k + 1) * s_k];
                    if (k + 2 < n_k) x.z = p[r * s_r + (k + 2) * s_k];
                    if (k + 3 < n_k) x.w = p[r * s_r + (k + 3) * s_k];
                }
            } else if (r < n_r && k < n_k) {  // the extent along the four is a multiple of 4
                x = *reinterpret_cast<const float4*>(p + r * s_r + k * s_k);
            }
            v[j] = x;
        }
    }
    __device__ __forceinline__ void store(float* sm, int row_floats, int kind) const {  // [kBK][row_floats]
#pragma unroll
        for (int j = 0; j < kVec; j++) {
            const int e = threadIdx.x + j * kGemmThreads;
            if (kind == 1) {
                *reinterpret_cast<float4*>(sm + (e / (ROWS / 4)) * row_floats + (e % (ROWS / 4)) * 4) = v[j];
            } else {
                const int r = kind != 2 ? e / (kBK / 4) : e % ROWS, k = kind != 2 ? (e % (kBK / 4)) * 4 : (e / ROWS) * 4;
                sm[k * row_floats + r] = v[j].x;
                sm[(k + 1) * row_floats + r] = v[j].y;
                sm[(k + 2) * row_floats + r] = v[j].z;
                sm[(k + 3) * row_floats + r] = v[j].w;
            }
        }
    }
};

__global__ void __launch_bounds__(kGemmThreads, 3) k_gemm(const float* __restrict__ A, const float* __restrict__ B, float* __restrict__ C,
                                                          int M, int N, int K, long long sa_i, long long sa_l, long long sb_l,
                                                          long long sb_j, int kind_a, int kind_b, const float* __restrict__ bias,
                                                          int relu, int accumulate) {
    // two stages, afterwards the partial tile [kBM][kRowB]
    __shared__ __align__(16) float sm[2 * kStageFloats > kBM * kRowB ? 2 * kStageFloats : kBM * kRowB];
    float* part = sm;
    cg::cluster_group cl = cg::this_cluster();
    const int split = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const int tid = threadIdx.x, tx = tid % 8, ty = tid / 8;  // 8 x 16 threads of 8 x 8 outputs
    const int tiles_n = (N + kBN - 1) / kBN, tile = (int)(blockIdx.x / (unsigned)split);
    const int i0 = tile / tiles_n * kBM, j0 = tile % tiles_n * kBN;
    // this CTA's K range: whole slices, in rank order
    const int slices = (K + kBK - 1) / kBK, per = (slices + split - 1) / split;
    const int s0 = min(rank * per, slices), s1 = min(s0 + per, slices);
    float acc[8][8] = {};
    Slice<kBM> sa;
    Slice<kBN> sb;
    if (s0 < s1) {
        sa.load(A, kind_a, i0, s0 * kBK, M, K, sa_i, sa_l);
        sb.load(B, kind_b, j0, s0 * kBK, N, K, sb_j, sb_l);
        sa.store(sm, kRowA, kind_a);
        sb.store(sm + kBK * kRowA, kRowB, kind_b);
    }
    __syncthreads();
    for (int sl = s0; sl < s1; sl++) {
        const float* as = sm + ((sl - s0) & 1) * kStageFloats;
        const float* bs = as + kBK * kRowA;
        const bool more = sl + 1 < s1;
        if (more) {
            sa.load(A, kind_a, i0, (sl + 1) * kBK, M, K, sa_i, sa_l);
            sb.load(B, kind_b, j0, (sl + 1) * kBK, N, K, sb_j, sb_l);
        }
#pragma unroll
        for (int l = 0; l < kBK; l++) {
            // rows 4 ty and 64 + 4 ty on, columns 4 tx and 32 + 4 tx on: neighbouring threads on neighbouring banks
            const float4 a0 = *reinterpret_cast<const float4*>(as + l * kRowA + 4 * ty), a1 = *reinterpret_cast<const float4*>(as + l * kRowA + 64 + 4 * ty);
            const float4 b0 = *reinterpret_cast<const float4*>(bs + l * kRowB + 4 * tx), b1 = *reinterpret_cast<const float4*>(bs + l * kRowB + 32 + 4 * tx);
            const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w}, b[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
            for (int r = 0; r < 8; r++)
#pragma unroll
                for (int c = 0; c < 8; c++) acc[r][c] = fmaf(a[r], b[c], acc[r][c]);
        }
        if (more) {
            float* nx = sm + ((sl - s0 + 1) & 1) * kStageFloats;
            sa.store(nx, kRowA, kind_a);
            sb.store(nx + kBK * kRowA, kRowB, kind_b);
        }
        __syncthreads();
    }
    auto write = [&](int gi, int gj, float v) {
        if (gi >= M || gj >= N) return;
        if (accumulate) v += C[(size_t)gi * N + gj];
        if (bias) v += bias[gj];
        if (relu) v = fmaxf(v, 0.0f);
        C[(size_t)gi * N + gj] = v;
    };
    if (split == 1) {
#pragma unroll
        for (int r = 0; r < 8; r++)
#pragma unroll
            for (int c = 0; c < 8; c++) write(i0 + (r >> 2) * 64 + 4 * ty + (r & 3), j0 + (c >> 2) * 32 + 4 * tx + (c & 3), acc[r][c]);
        return;
    }
#pragma unroll
    for (int r = 0; r < 8; r++)
#pragma unroll
        for (int c = 0; c < 2; c++)
            *reinterpret_cast<float4*>(part + ((r >> 2) * 64 + 4 * ty + (r & 3)) * kRowB + c * 32 + 4 * tx) =
                make_float4(acc[r][4 * c], acc[r][4 * c + 1], acc[r][4 * c + 2], acc[r][4 * c + 3]);
    cl.sync();
    // each CTA adds up its share of the tile's rows from all of them, in rank order
    const int rows = kBM / split;
    for (int e = tid; e < rows * (kBN / 4); e += kGemmThreads) {
        const int r = rank * rows + e / (kBN / 4), c = (e % (kBN / 4)) * 4;
        float4 t = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        for (int q = 0; q < split; q++) {
            const float4 x = *reinterpret_cast<const float4*>(cl.map_shared_rank(part, q) + r * kRowB + c);
            t.x += x.x; t.y += x.y; t.z += x.z; t.w += x.w;
        }
        write(i0 + r, j0 + c, t.x);
        write(i0 + r, j0 + c + 1, t.y);
        write(i0 + r, j0 + c + 2, t.z);
        write(i0 + r, j0 + c + 3, t.w);
    }
    cl.sync();  // the others may still be reading this CTA's tile
}

// Products of few terms (short_product), whose sums k_gemm would not split, in the same order: 64x64 tiles of 4x4 outputs a
// thread, four times as many threads on an output as k_gemm's, and little code.  They are bound by the call's latency
// or, with one slice of terms, by writing C.  Measured (B200, k_gemm / this, along-K operands): 16x16x16 11.4 / 8.3 us,
// 33x4097x7 12.2 / 8.3, 8192x4096x16 76 / 67; 256x256x64 15.6 / 12.5, 2048x256x64 15.7 / 14.2, 20000x8x64 (313 tiles) 18.0 /
// 16.5, 2048x700x127 (352) 34 / 28; 2048x1408x32 (704) 18.1 / 18.8, x64 23.8 / 28.5.
constexpr int kShortTile = 64, kShortTiles = 3 * 148;
__host__ inline long long short_tiles(int M, int N) {
    return (long long)((N + kShortTile - 1) / kShortTile) * ((M + kShortTile - 1) / kShortTile);
}
__host__ inline bool short_product(int M, int N, int K) { return K <= kBK || (K < kSplitK && short_tiles(M, N) <= kShortTiles); }
__global__ void __launch_bounds__(256) k_gemm_short(const float* __restrict__ A, const float* __restrict__ B, float* __restrict__ C,
                                                    int M, int N, int K, long long sa_i, long long sa_l, long long sb_l, long long sb_j,
                                                    const float* __restrict__ bias, int relu, int accumulate) {
    __shared__ __align__(16) float as[kBK][kShortTile + 4], bs[kBK][kShortTile + 4];
    const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
    const int tiles_n = (N + kShortTile - 1) / kShortTile;
    const int i0 = (int)(blockIdx.x / (unsigned)tiles_n) * kShortTile, j0 = (int)(blockIdx.x % (unsigned)tiles_n) * kShortTile;
    const bool a_k = sa_l == 1, b_k = sb_l == 1;  // consecutive threads along K, or along the rows
    float acc[4][4] = {};
#pragma unroll 1
    for (int k0 = 0; k0 < K; k0 += kBK) {
        if (k0 > 0) __syncthreads();
#pragma unroll
        for (int j = 0; j < kBK * kShortTile / 256; j++) {
            const int e = tid + 256 * j, l0 = e / kShortTile, r0 = e % kShortTile, l1 = e % kBK, r1 = e / kBK;
            const int la = a_k ? l1 : l0, ra = a_k ? r1 : r0, lb = b_k ? l1 : l0, rb = b_k ? r1 : r0;
            as[la][ra] = k0 + la < K && i0 + ra < M ? A[(i0 + ra) * sa_i + (k0 + la) * sa_l] : 0.0f;
            bs[lb][rb] = k0 + lb < K && j0 + rb < N ? B[(k0 + lb) * sb_l + (j0 + rb) * sb_j] : 0.0f;
        }
        __syncthreads();
        const int ln = min(kBK, K - k0);
#pragma unroll 2
        for (int l = 0; l < ln; l++) {
            const float4 a4 = *reinterpret_cast<const float4*>(&as[l][4 * ty]), b4 = *reinterpret_cast<const float4*>(&bs[l][4 * tx]);
            const float a[4] = {a4.x, a4.y, a4.z, a4.w}, b[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
            for (int r = 0; r < 4; r++)
#pragma unroll
                for (int c = 0; c < 4; c++) acc[r][c] = fmaf(a[r], b[c], acc[r][c]);
        }
    }
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const int gi = i0 + 4 * ty + r, gj = j0 + 4 * tx + c;
            if (gi >= M || gj >= N) continue;
            float v = acc[r][c];
            if (accumulate) v += C[(size_t)gi * N + gj];
            if (bias) v += bias[gj];
            if (relu) v = fmaxf(v, 0.0f);
            C[(size_t)gi * N + gj] = v;
        }
}

struct XentShape {
    int nout, nbm, head_stride, batch;
    mlp::Shape cls;  // class plan (p1, part_base, head_base)
};
__device__ __forceinline__ float wmax(float v) {
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
    return v;
}
__device__ __forceinline__ float wsum(float v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    return v;
}

__global__ void __launch_bounds__(128) k_xent(const float* __restrict__ Z, const int* __restrict__ part_label,
                                               const int* __restrict__ bm_label, XentShape s, float* __restrict__ dZ,
                                               float* __restrict__ loss) {
    const int lane = threadIdx.x & 31;
    const int b = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (b >= s.batch) return;
    const float* z = Z + (size_t)b * s.nout;
    float* g = dZ + (size_t)b * s.nout;
    const float inv_b = 1.0f / (float)s.batch;
    const int pl = part_label[b], bl = bm_label[b];
    // partition head
    float mx = -3.0e38f;
    const int p1 = s.cls.p1, hb = s.cls.head_base;
    for (int c = lane; c <= p1; c += 32) mx = fmaxf(mx, z[c]);
    mx = wmax(mx);
    float se = 0.0f;
    for (int c = lane; c <= p1; c += 32) se += expf(z[c] - mx);
    se = wsum(se);
    for (int c = lane; c < hb; c += 32) {
        float v = 0.0f;
        if (c <= p1) v = (expf(z[c] - mx) / se - (c == pl ? 1.0f : 0.0f)) * inv_b;
        g[c] = v;
    }
    // block-mode head of the label's partition count
    const int head = mlp::head_of_class(s.cls, pl);
    const int h0 = hb + head * s.head_stride;
    float hm = -3.0e38f;
    for (int c = lane; c < s.nbm; c += 32) hm = fmaxf(hm, z[h0 + c]);
    hm = wmax(hm);
    float hs = 0.0f;
    for (int c = lane; c < s.nbm; c += 32) hs += expf(z[h0 + c] - hm);
    hs = wsum(hs);
    for (int c = hb + lane; c < s.nout; c += 32) {
        float v = 0.0f;
        const int k = c - h0;
        if (k >= 0 && k < s.nbm) v = (expf(z[c] - hm) / hs - (k == bl ? 1.0f : 0.0f)) * inv_b;
        g[c] = v;
    }
    if (lane == 0) {
        loss[2 * b] = logf(se) + mx - z[pl];
        loss[2 * b + 1] = logf(hs) + hm - z[h0 + bl];
    }
}

__global__ void k_relu_bwd(float* __restrict__ dh, const float* __restrict__ h, size_t n) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        if (!(h[i] > 0.0f)) dh[i] = 0.0f;
}

// 32 columns a CTA, each summed by 32 threads over every 32nd row (consecutive threads on
// consecutive columns), their sums added in order: one thread a column, which this replaces,
// waited for 2,048 loads one after another.
constexpr int kColsumGroups = 32;
// The same sums, in the same order, by one thread a column.
__global__ void __launch_bounds__(128) k_colsum_wide(const float* __restrict__ dy, float* __restrict__ db, int rows, int cols) {
    const int j = blockIdx.x * 128 + threadIdx.x;
    if (j >= cols) return;
    float s[kColsumGroups] = {};
    for (int r0 = 0; r0 < rows; r0 += kColsumGroups)
#pragma unroll
        for (int q = 0; q < kColsumGroups; q++)
            if (r0 + q < rows) s[q] += dy[(size_t)(r0 + q) * cols + j];
    float t = 0.0f;
#pragma unroll
    for (int q = 0; q < kColsumGroups; q++) t += s[q];
    db[j] = t;
}
__global__ void __launch_bounds__(32 * kColsumGroups) k_colsum(const float* __restrict__ dy, float* __restrict__ db, int rows, int cols) {
    __shared__ float part[kColsumGroups][32];
    const int c = threadIdx.x & 31, g = threadIdx.x >> 5, j = blockIdx.x * 32 + c;
    float s = 0.0f;
    if (j < cols) {
#pragma unroll 8
        for (int r = g; r < rows; r += kColsumGroups) s += dy[(size_t)r * cols + j];
    }
    part[g][c] = s;
    __syncthreads();
    if (g == 0 && j < cols) {
        float t = 0.0f;
        for (int q = 0; q < kColsumGroups; q++) t += part[q][c];
        db[j] = t;
    }
}

__global__ void k_adam(float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m, float* __restrict__ v, size_t n,
                       float lr, float b1, float b2, float eps, float c1, float c2) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.0f - b1) * gi;
        const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        w[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    }
}

int launch_status() { return cudaGetLastError() == cudaSuccess ? ASTCB200_OK : ASTCB200_CUDA_ERROR; }

}  // namespace
}  // namespace astcb200

using namespace astcb200;

extern "C" {

int astcb200_train_gemm(const float* A, const float* B, float* C, int M, int N, int K, int64_t sa_i, int64_t sa_l, int64_t sb_l,
                        int64_t sb_j, const float* bias, int relu, int accumulate, void* stream) {
    if (!A || !B || !C || M <= 0 || N <= 0 || K <= 0) return ASTCB200_BAD_ARG;
    if (short_product(M, N, K)) {
        const long long tiles = short_tiles(M, N);
        if (tiles > 0x7FFFFFFFll) return ASTCB200_CUDA_ERROR;
        k_gemm_short<<<(unsigned)tiles, 256, 0, (cudaStream_t)stream>>>(A, B, C, M, N, K, sa_i, sa_l, sb_l, sb_j, bias, relu, accumulate);
        return launch_status();
    }
    // four floats at a time along a stride of 1, when every row starts on 16 bytes and the extent is a multiple of four
    auto kind = [](const float* p, int n_r, int n_k, int64_t s_r, int64_t s_k) {
        const bool aligned = ((uintptr_t)p & 15) == 0;
        if (aligned && s_k == 1 && s_r % 4 == 0 && n_k % 4 == 0) return 0;
        if (aligned && s_r == 1 && s_k % 4 == 0 && n_r % 4 == 0) return 1;
        return s_k == 1 ? 3 : 2;
    };
    const int kind_a = kind(A, M, K, sa_i, sa_l), kind_b = kind(B, N, K, sb_j, sb_l);
    const long long tiles = (long long)((N + kBN - 1) / kBN) * ((M + kBM - 1) / kBM);
    // CTAs for two on every SM where K allows at least four slices each
    int split = 1;
    while (split < kMaxSplit && tiles * split < 296 && K / (2 * split) >= 4 * kBK) split *= 2;
    cudaLaunchConfig_t cfg = {};
    if (tiles * split > 0x7FFFFFFFll) return ASTCB200_CUDA_ERROR;
    cfg.gridDim = dim3((unsigned)(tiles * split));
    cfg.blockDim = dim3(kGemmThreads);
    cfg.stream = (cudaStream_t)stream;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)split; at.val.clusterDim.y = 1; at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = split > 1 ? 1 : 0;
    if (cudaLaunchKernelEx(&cfg, k_gemm, A, B, C, M, N, K, (long long)sa_i, (long long)sa_l, (long long)sb_l, (long long)sb_j, kind_a, kind_b,
                           bias, relu, accumulate) != cudaSuccess) {
        cudaGetLastError();
        return ASTCB200_CUDA_ERROR;
    }
    return launch_status();
}

int astcb200_train_xent(const float* Z, uint32_t nout, const int32_t* part_label, const int32_t* bm_label, uint32_t batch,
                        uint32_t nbm, uint32_t head_stride, const uint32_t* sel3, float* dZ, float* loss_rows, void* stream) {
    if (!Z || !part_label || !bm_label || !sel3 || !dZ || !loss_rows || batch == 0) return ASTCB200_BAD_ARG;
    XentShape s;
    s.cls = mlp::shape_for(0, (int)nbm, sel3);
    if (nbm > head_stride || nout < (uint32_t)s.cls.head_base + 4 * head_stride) return ASTCB200_BAD_ARG;
    s.nout = (int)nout; s.nbm = (int)nbm; s.head_stride = (int)head_stride; s.batch = (int)batch;
    k_xent<<<(batch + 3) / 4, 128, 0, (cudaStream_t)stream>>>(Z, part_label, bm_label, s, dZ, loss_rows);
    return launch_status();
}

int astcb200_train_relu_backward(float* dH, const float* H, size_t n, void* stream) {
    if (!dH || !H) return ASTCB200_BAD_ARG;
    k_relu_bwd<<<1184, 256, 0, (cudaStream_t)stream>>>(dH, H, n);
    return launch_status();
}

int astcb200_train_colsum(const float* dY, float* db, uint32_t rows, uint32_t cols, void* stream) {
    if (!dY || !db) return ASTCB200_BAD_ARG;
    // Many columns of few rows: 1,024 threads a CTA for 32 columns would mostly wait for their launch.  Measured (B200, 32
    // threads a column / one): 8x100000 14.4 / 8.7 us, 32x16384 8.7 / 6.9, 128x32768 12.6 / 10.8, 128x100000 23.0 / 15.2;
    // 128x16384 8.9 / 10.5, 256x100000 25 / 52, and no difference below 4,096 columns of 32 rows.
    if (rows <= 32 ? cols >= 4096 : rows <= 128 && cols >= 32768) {
        k_colsum_wide<<<(cols + 127) / 128, 128, 0, (cudaStream_t)stream>>>(dY, db, (int)rows, (int)cols);
        return launch_status();
    }
    k_colsum<<<(cols + 31) / 32, 32 * kColsumGroups, 0, (cudaStream_t)stream>>>(dY, db, (int)rows, (int)cols);
    return launch_status();
}

int astcb200_train_adam(float* w, const float* g, float* m, float* v, size_t n, float lr, float beta1, float beta2, float eps,
                        uint32_t step, void* stream) {
    if (!w || !g || !m || !v || step == 0) return ASTCB200_BAD_ARG;
    const float c1 = 1.0f - powf(beta1, (float)step), c2 = 1.0f - powf(beta2, (float)step);
    k_adam<<<1184, 256, 0, (cudaStream_t)stream>>>(w, g, m, v, n, lr, beta1, beta2, eps, c1, c2);
    return launch_status();
}

}  // extern "C"
