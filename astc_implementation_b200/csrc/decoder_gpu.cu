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
#include <cuda_runtime.h>

#include <cstddef>

#include "astcb200.h"
#include "decode_fast.cuh"
#include "streamless.h"
#include "tables.h"

namespace astcb200 {

using namespace dec::fast;

namespace {

constexpr int kDecodeThreads = 128;
constexpr int kDecodeBlocks = 64;  // per CTA

// CTAs in raster order of groups of kDecodeBlocks blocks: cols blocks wide, kDecodeBlocks / cols block rows high.
template <bool kError>
__global__ void __launch_bounds__(kDecodeThreads) k_decode(const uint8_t* __restrict__ blocks, int bx, int by, int dx, int dy,
                                                            int nbx, int nby, int cols, int groups_x, uchar4* __restrict__ out,
                                                            const uchar4* __restrict__ ref, unsigned long long* __restrict__ sse) {
    __shared__ __align__(16) Stage<kDecodeBlocks> s;
    __shared__ ValueTables tables;
    const int tid = threadIdx.x;
    const int rows = kDecodeBlocks / cols;
    const int gx = (int)(blockIdx.x % (unsigned)groups_x) * cols, gy = (int)(blockIdx.x / (unsigned)groups_x) * rows;
    {
        static_assert(alignof(DecodeTables) % 4 == 0 && offsetof(DecodeTables, values) % 4 == 0 && sizeof(ValueTables) % 4 == 0,
                      "the tables are copied as words");
        const uint32_t* src = reinterpret_cast<const uint32_t*>(&g_tables.values);
        uint32_t* dst = reinterpret_cast<uint32_t*>(&tables);
        for (int i = tid; i < (int)sizeof(ValueTables) / 4; i += kDecodeThreads) dst[i] = src[i];
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
        if (k < rows * cols) parse_part(s, tables, k, bx, by, tid >= kDecodeBlocks);
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
                const int part = texel_partition(f, o, pc, (uint32_t)xs, (uint32_t)y << small);
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
    if (await_streamless(blocks, (size_t)nbx * nby * 16, s) != cudaSuccess) return ASTCB200_CUDA_ERROR;
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
