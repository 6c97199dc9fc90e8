// Learned proposal: network inference on the tcgen05 tensor cores and the
// selection of partitionings, block modes and routes from its logits.
//
// k_mlp_logits: one CTA per 128 blocks, eight epilogue warps (two threads per block row, each
// taking half of a row's accumulator columns), one warp that issues the MMAs of layer 3 and one
// that fetches its weights.  The block texels are
// staged in shared memory as bf16 in the tensor core's K-major core-matrix
// layout; each layer is a chain of tcgen05.mma (M=128, K=16 per instruction,
// A and B from shared memory, FP32 accumulators in tensor memory) issued by
// one thread.  Weights arrive by bulk copies (cp.async.bulk, completion on an
// mbarrier) already laid out on the host in the same core-matrix order.  The
// two hidden layers' epilogues (bias, ReLU, bf16) read the accumulators with
// tcgen05.ld and write the next layer's A operand in place; layer 3 runs in
// 64-column chunks through four weight buffers and eight accumulator buffers (all 512
// tensor-memory columns): the fetching thread, the issuing thread and the epilogue warps only
// meet at mbarriers (weights landed; weights consumed; accumulator full; accumulator read).
// The layer-3 epilogue adds the bias and stores its 32 logits as four 32-byte sectors; CTAs start the
// chunk sequence at different chunks so that they do not all fetch the same weights
// from L2 at once.  Two CTA barriers a chunk and a 256-byte bulk copy per row and chunk out of
// a staging buffer, which this replaces, kept the tensor pipe at 12 % and took 885 us for
// 262,144 blocks at 4x4 (231 GFLOP, 1.48 GB of logits: 225 us to write); this takes 568 us.
// Every wait on an mbarrier is bounded (error_flag[1] polls, 0 = 2^24); a thread that gives up
// makes its CTA give up: it sets error_flag[0], waits (bounded by 2^24 polls) for its own copies
// and MMAs in flight, frees its tensor memory and returns.
//
// k_select: one warp per block turns the logits into the proposal search's
// inputs: a softmax over the partition classes, the best partitionings (in
// probability order, until the proposed mass reaches the coverage), the best
// block modes of each partition count as bit masks, and the route: blocks
// whose best-kmax mass is below the threshold take the full search.
#include <cuda_bf16.h>

#include "mlp.h"

namespace astcb200 {
namespace mlp {
namespace {

constexpr uint32_t kOffA = 0;                 // 64 KB: X, then H1, then H2 (128 rows x up to 256 bf16)
constexpr uint32_t kOffW = 65536;             // 128 KB: W1, W2, then the W3 chunks of 32 KB
constexpr uint32_t kW3Buf = kChunkN * 256 * 2;               // one W3 chunk (bf16)
constexpr int kWBufs = 4;                     // weight buffers of layer 3
constexpr int kAccBufs = 8;                   // its accumulator buffers, kChunkN tensor-memory columns each
constexpr uint32_t kOffBar = kOffW + kWBufs * kW3Buf;         // mbarriers and flags
static_assert(kOffBar == 196608 && kOffBar + 1024 + 1024 == (uint32_t)kMlpSmemBytes, "shared memory plan");
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kWaitLimit = 1u << 24;     // polls of an mbarrier before a CTA gives up
constexpr uint32_t kCopyPiece = 32768;        // bytes per bulk copy instruction

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_test_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Waits for the phase of parity `parity` to complete, at most `limit` polls.  Limits below
// 2^16 (set by tests of the give-up path) poll with the non-blocking test_wait, so that a
// wait for work still in flight gives up at once; larger ones use try_wait, which may
// suspend the thread until the phase completes.
__device__ bool mbar_wait(uint64_t* bar, uint32_t parity, uint32_t limit = kWaitLimit) {
    if (limit < (1u << 16)) {
        for (uint32_t i = 0; i < limit; i++)
            if (mbar_test_wait(bar, parity)) return true;
        return false;
    }
    for (uint32_t i = 0; i < limit; i++)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
// One thread: expect `bytes` on bar and copy them in pieces.
__device__ void load_weights(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    mbar_expect_tx(bar, bytes);
    for (uint32_t o = 0; o < bytes; o += kCopyPiece)
        bulk_load(static_cast<uint8_t*>(dst) + o, static_cast<const uint8_t*>(src) + o, min(kCopyPiece, bytes - o), bar);
}

__device__ __forceinline__ void tc_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void async_proxy_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// Shared-memory matrix descriptor: no swizzle, K-major core matrices; lbo =
// bytes between K-adjacent core matrices, sbo = bytes between M/N-adjacent
// ones; descriptor version 1 (bits 46-47), base offset 0.
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((saddr >> 4) & 0x3FFF) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) | (1ull << 46);
}
// Instruction descriptor of kind::f16: bf16 A and B (K-major), FP32 accumulator.
__host__ __device__ constexpr uint32_t instr_desc(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
static_assert(kAccBufs * kChunkN == (int)kTmemCols, "layer 3 uses every column");
static_assert(instr_desc(128, 256) == 0x08400490u, "instruction descriptor layout");

__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc)
        : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// 32 consecutive FP32 columns of the calling thread's tensor-memory lane.
__device__ __forceinline__ void tmem_load32(uint32_t taddr, float* v) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ uint32_t bf16_bits(float f) {
    return (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(f));
}
__device__ __forceinline__ uint4 pack8(const float* v) {
    return make_uint4(bf16_bits(v[0]) | (bf16_bits(v[1]) << 16), bf16_bits(v[2]) | (bf16_bits(v[3]) << 16),
                      bf16_bits(v[4]) | (bf16_bits(v[5]) << 16), bf16_bits(v[6]) | (bf16_bits(v[7]) << 16));
}

// Hidden-layer epilogue: accumulator columns [col0 + c0, col0 + c0 + 128) of this thread's
// row (c0: its half of the 256) -> bias, ReLU, bf16 -> the A operand (128 rows x 256) of the
// next layer.
__device__ void hidden_epilogue(uint32_t tmem_row, uint32_t col0, int c0, const float* __restrict__ bias, uint8_t* sA, int m) {
    for (int c = c0; c < c0 + 128; c += 32) {
        float v[32];
        tmem_load32(tmem_row + col0 + c, v);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const float4* b4 = reinterpret_cast<const float4*>(bias + c + q * 8);
            const float4 b0 = __ldg(b4), b1 = __ldg(b4 + 1);
            const float b[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
            float h[8];
#pragma unroll
            for (int i = 0; i < 8; i++) h[i] = fmaxf(v[q * 8 + i] + b[i], 0.0f);
            *reinterpret_cast<uint4*>(sA + core_index(m, c + q * 8, kTileRows) * 2) = pack8(h);
        }
    }
}

constexpr int kEpilogueThreads = 2 * kTileRows;  // two threads per row, each taking half of the columns
constexpr int kMlpThreads = kEpilogueThreads + 64;  // and the warps of the layer-3 issuer and fetcher

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Eight consecutive floats, one sector.
__device__ __forceinline__ void store8(float* p, const float* v) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]),
                 "f"(v[5]), "f"(v[6]), "f"(v[7])
                 : "memory");
}

__global__ void __launch_bounds__(kMlpThreads, 1)
    k_mlp_logits(const __grid_constant__ KernelArgs a, const __grid_constant__ Net net, float* __restrict__ logits, int* error_flag) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sA = sm + kOffA;
    uint8_t* sW = sm + kOffW;
    uint64_t* bw = reinterpret_cast<uint64_t*>(sm + kOffBar);  // weights of layers 1 and 2
    uint64_t* bm = bw + 1;                                     // their MMAs
    uint64_t* w_full = bw + 2;                                 // [kWBufs] layer 3: weights landed
    uint64_t* w_free = w_full + kWBufs;                        // [kWBufs] and consumed
    uint64_t* acc_full = w_free + kWBufs;                      // [kAccBufs] accumulator complete
    uint64_t* acc_free = acc_full + kAccBufs;                  // [kAccBufs] and read (by the eight epilogue warps)
    constexpr int kBars = 2 + 2 * kWBufs + 2 * kAccBufs;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bw + kBars);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(bw + kBars + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // this thread's row (block) in the tile and tensor-memory lane; warps w and w + 4 share
    // the lanes of quarter w and split the columns (half)
    const bool epilogue = tid < kEpilogueThreads;
    const int m = tid % kTileRows, half = tid / kTileRows;
    const int lb = blockIdx.x * kTileRows + m;
    const Shape& S = net.s;
    const int nchunks = S.nout / kChunkN;
    // CTAs walk the layer-3 chunks from different starting points, so that at any moment they
    // read different parts of the weights from L2 instead of all the same chunk
    const int j0 = blockIdx.x % nchunks;
    auto chunk_of = [&](int j) { const int c = j0 + j; return c < nchunks ? c : c - nchunks; };
    const uint32_t wl = error_flag[1] ? (uint32_t)error_flag[1] : kWaitLimit;  // polls per wait

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int i = 0; i < kBars - kAccBufs; i++) mbar_init(&bw[i], 1);
        for (int i = 0; i < kAccBufs; i++) mbar_init(&acc_free[i], kEpilogueThreads / 32);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    tc_before();
    __syncthreads();
    tc_after();
    const uint32_t tmem = *tmem_slot;
    const uint32_t tmem_row = tmem + ((uint32_t)((warp & 3) * 32) << 16);

    // thread 0's bookkeeping of layers 1 and 2: a phase counts as done only once a wait saw it
    // complete, so the drain after a give-up waits for the rest
    uint32_t w_issued = 0, w_done = 0, m_issued = 0, m_done = 0;  // only the waits of all threads advance m_done
    int fetched = 0, issued = 0;  // layer-3 chunks the fetching and the issuing thread have started
    bool ok = true;

    if (tid == 0) { load_weights(sW, net.w1, 256u * S.k0p * 2, bw); w_issued++; }

    // stage the block's texels (RGBA8 / 255 -> bf16), zero rows past the chunk
    if (epilogue) {
        const int blk = lb < a.nblocks ? chunk_block(a, lb) : -1;
        const int T = a.L.T;
        BlockSrc src{};
        if (blk >= 0) src = block_src(a, blk);
        for (int j = half; j < S.k0p / 8; j += 2) {
            float v[8];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int t = 2 * j + h;
                uchar4 p = make_uchar4(0, 0, 0, 0);
                if (blk >= 0 && t < T) p = src_rgba8(src, a.L.bx, t);
                v[4 * h + 0] = (float)p.x / 255.0f; v[4 * h + 1] = (float)p.y / 255.0f;
                v[4 * h + 2] = (float)p.z / 255.0f; v[4 * h + 3] = (float)p.w / 255.0f;
            }
            *reinterpret_cast<uint4*>(sA + core_index(m, 8 * j, kTileRows) * 2) = pack8(v);
        }
    }
    async_proxy_fence();
    tc_before();
    __syncthreads();

    const uint32_t a_base = smem_u32(sA), w_base = smem_u32(sW);
    constexpr uint32_t kLboA = (kTileRows / 8) * 128, kLboW256 = (256 / 8) * 128, kLboW3 = (kChunkN / 8) * 128;
    // one of layers 1 and 2: thread 0 issues its MMAs once its weights have landed, all threads wait
    auto dense = [&](uint32_t d_tmem, int ksteps) -> bool {
        if (tid == 0) {
            tc_after();
            if (!mbar_wait(bw, w_done & 1, wl)) *abort_flag = 1;
            else {
                w_done++;
                for (int kk = 0; kk < ksteps; kk++)
                    mma_bf16(d_tmem, smem_desc(a_base + kk * 2 * kLboA, kLboA, 128), smem_desc(w_base + kk * 2 * kLboW256, kLboW256, 128),
                             instr_desc(128, 256), kk > 0);
                mma_commit(bm);
                m_issued++;
            }
        }
        __syncthreads();
        if (*abort_flag) return false;
        ok = mbar_wait(bm, m_done & 1, wl);
        if (ok) m_done++;
        if (__syncthreads_or(!ok)) { *abort_flag = 1; return false; }
        tc_after();
        return true;
    };

    // ---- layer 1: X (128 x k0p) . W1^T -> tensor memory columns [0, 256)
    if (!dense(tmem, S.k0p / 16)) goto cleanup;
    if (tid == 0) { load_weights(sW, net.w2, 256u * 256u * 2, bw); w_issued++; }
    if (epilogue) hidden_epilogue(tmem_row, 0, half * 128, net.b1, sA, m);
    async_proxy_fence();
    tc_before();
    __syncthreads();

    // ---- layer 2: H1 (128 x 256) . W2^T -> columns [256, 512)
    if (!dense(tmem + 256, 16)) goto cleanup;
    if (tid == kEpilogueThreads + 32) {  // the fetcher: W2 is consumed
        for (; fetched < kWBufs && fetched < nchunks; fetched++)
            load_weights(sW + fetched * kW3Buf, net.w3 + (size_t)chunk_of(fetched) * kChunkN * 256, kW3Buf, &w_full[fetched]);
    }
    if (epilogue) hidden_epilogue(tmem_row, 256, half * 128, net.b2, sA, m);
    async_proxy_fence();
    tc_before();
    __syncthreads();

    // ---- layer 3: H2 (128 x 256) . W3^T in chunks of 64 columns.  Use u of a buffer waits for phase
    // u of its full barrier and phase u - 1 of its free one.
    {
        auto wait = [&](uint64_t* bar, int phase) -> bool {  // false: this thread or another gave up
            for (uint32_t i = 0; i < wl; i++) {
                if (wl < (1u << 16) ? mbar_test_wait(bar, (uint32_t)phase & 1u) : mbar_try_wait(bar, (uint32_t)phase & 1u)) return true;
                if (*abort_flag) return false;
            }
            *abort_flag = 1;
            return false;
        };
        if (epilogue) {
            const bool store = lb < a.nblocks;
            float* out_row = logits + (size_t)lb * S.nout + half * 32;
            for (int j = 0; j < nchunks; j++) {
                const int b = j % kAccBufs, c0 = chunk_of(j) * kChunkN;
                // this thread's 32 biases of the chunk, loaded before the wait so that it hides them
                float bv[32], v[32];
                const float4* bias4 = reinterpret_cast<const float4*>(net.b3 + c0 + half * 32);
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    const float4 t = __ldg(bias4 + q);
                    bv[4 * q] = t.x; bv[4 * q + 1] = t.y; bv[4 * q + 2] = t.z; bv[4 * q + 3] = t.w;
                }
                if (!__all_sync(0xFFFFFFFFu, wait(&acc_full[b], j / kAccBufs))) break;  // the tensor-memory load takes whole warps
                tc_after();
                tmem_load32(tmem_row + b * kChunkN + half * 32, v);
                tc_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_free[b]);
                if (store) {
#pragma unroll
                    for (int i = 0; i < 32; i++) v[i] = v[i] + bv[i];
#pragma unroll
                    for (int q = 0; q < 4; q++) store8(out_row + c0 + 8 * q, v + 8 * q);
                }
            }
        } else if (tid == kEpilogueThreads) {  // the issuer
            tc_after();
            for (int j = 0; j < nchunks; j++) {
                const int wb = j % kWBufs, b = j % kAccBufs;
                if (!wait(&w_full[wb], j / kWBufs)) break;
                if (j >= kAccBufs) {
                    if (!wait(&acc_free[b], j / kAccBufs - 1)) break;
                    tc_after();
                }
                for (int kk = 0; kk < 16; kk++)
                    mma_bf16(tmem + b * kChunkN, smem_desc(a_base + kk * 2 * kLboA, kLboA, 128),
                             smem_desc(w_base + wb * kW3Buf + kk * 2 * kLboW3, kLboW3, 128), instr_desc(128, kChunkN), kk > 0);
                mma_commit(&w_free[wb]);
                mma_commit(&acc_full[b]);
                issued = j + 1;
            }
        } else if (tid == kEpilogueThreads + 32) {  // the fetcher
            for (int j = fetched; j < nchunks; j++) {
                const int wb = j % kWBufs;
                if (!wait(&w_free[wb], j / kWBufs - 1)) break;
                load_weights(sW + wb * kW3Buf, net.w3 + (size_t)chunk_of(j) * kChunkN * 256, kW3Buf, &w_full[wb]);
                fetched = j + 1;
            }
        }
    }

cleanup:
    __syncthreads();
    if (*abort_flag) {
        // give up: record it, then let our own copies and MMAs drain (bounded) before the
        // shared and tensor memory are released
        if (tid == 0) {
            atomicExch(error_flag, 1);  // error_flag[0]
            while (w_done < w_issued) { mbar_wait(bw, w_done & 1); w_done++; }
            for (uint32_t i = m_done; i < m_issued; i++) mbar_wait(bm, i & 1);
        }
        // the last copy into each buffer, and the last chunk's MMAs (commits complete in order)
        for (int j = fetched > kWBufs ? fetched - kWBufs : 0; j < fetched; j++) mbar_wait(&w_full[j % kWBufs], (uint32_t)(j / kWBufs) & 1u);
        if (issued) mbar_wait(&acc_full[(issued - 1) % kAccBufs], (uint32_t)((issued - 1) / kAccBufs) & 1u);
    }
    tc_before();
    __syncthreads();
    tc_after();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
}

// ------------------------------------------------------------ selection

__device__ __forceinline__ float warp_max(float v) {
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
    return v;
}
__device__ __forceinline__ float warp_sum(float v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    return v;
}

// Monotone map of a finite float to an unsigned key (larger value, larger key).
__device__ __forceinline__ uint32_t okey(float v) {
    const uint32_t u = __float_as_uint(v);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float okey_value(uint32_t k) {
    return __uint_as_float((k & 0x80000000u) ? (k ^ 0x80000000u) : ~k);
}

// The kbm best of nbm modes (at most 32 NW) by (logit descending, index ascending) as a bit mask, 64
// modes per lane from lane 0; lane l holds modes l + 32 u.  One pick per round; when kbm is above
// half the modes, the rounds pick the others instead, worst first (logit ascending, index
// descending): the same set in fewer rounds.  A lane has its two best at hand and looks for more
// only when both were picked.
template <int NW>
__device__ __forceinline__ uint64_t mode_mask(const float* h, int nbm, int kbm, int lane) {
    constexpr uint32_t kFull = 0xFFFFFFFFu;
    const int kk = kbm < nbm ? kbm : nbm;
    const bool worst = 2 * kk > nbm;
    const int rounds = worst ? nbm - kk : kk;
    uint32_t key[NW];  // 0: absent or picked
#pragma unroll
    for (int u = 0; u < NW; u++) {
        const int c = lane + 32 * u;
        key[u] = 0;
        if (c < nbm) { const uint32_t k = okey(h[c] + 0.0f); key[u] = worst ? ~k : k; }  // -0 as +0
    }
    uint32_t picked = 0, k1 = 0, k2 = 0;
    int u1 = 0, u2 = 0;
    bool look = true;
#pragma unroll 1
    for (int k = 0; k < rounds; k++) {
        if (look) {
            k1 = k2 = 0;
#pragma unroll
            for (int i = 0; i < NW; i++) {
                const int u = worst ? NW - 1 - i : i;  // the first of equal keys: the lowest index, the highest when picking the worst
                const uint32_t x = worst ? key[NW - 1 - i] : key[i];
                if (((picked >> u) & 1) || x == 0) continue;
                if (x > k1) { k2 = k1; u2 = u1; k1 = x; u1 = u; }
                else if (x > k2) { k2 = x; u2 = u; }
            }
            look = false;
        }
        const uint32_t best = __reduce_max_sync(kFull, k1);
        if (best == 0u) break;
        const uint32_t idx = (uint32_t)(lane + 32 * u1);
        const uint32_t ci = worst ? __reduce_max_sync(kFull, k1 == best ? idx : 0u) : __reduce_min_sync(kFull, k1 == best ? idx : 0xFFFFFFFFu);
        if (k1 == best && idx == ci) {
            picked |= 1u << u1;
            look = k2 == 0;
            k1 = k2; u1 = u2; k2 = 0;
        }
    }
    uint64_t word = 0;
#pragma unroll
    for (int u = 0; u < NW; u++) {
        const bool valid = lane + 32 * u < nbm;
        const uint32_t chosen = __ballot_sync(kFull, valid && (((picked >> u) & 1) != 0) != worst);
        if (lane == (u >> 1)) word |= (uint64_t)chosen << (32 * (u & 1));
    }
    return word;
}

// One warp per block, kSelectWarps a CTA, which take their places in the lists together: one
// atomic per list and CTA.  (One per block put 262,144 additions on each of two addresses.)  Most
// blocks' single-partition probability reaches the coverage on its own; they need the softmax
// alone, not the ranking of the partitionings; the others collect the logits that can be among the
// kmax best, a few more than kmax, one a lane, and pick with two redux steps each.
// Measured (B200, 262,144 blocks of 1,408 logits): 875 -> 470 us, of which 225 is reading them.
constexpr int kSelectWarps = 8;
constexpr int kHeld = 36;  // partition logits a lane keeps in registers (of 35 at 4x4 and 6x6); more are read again
__global__ void __launch_bounds__(kSelectWarps * 32, 3) k_select(const __grid_constant__ KernelArgs a, const __grid_constant__ Shape S,
                                                              const float* __restrict__ logits, const __grid_constant__ Select sel,
                                                              const __grid_constant__ Routes r) {
    constexpr uint32_t kFull = 0xFFFFFFFFu;
    // per warp: its place counts (0 proposal list, 1 full-search list, 2..5 partitioned blocks of
    // P = 1..4), then the CTA's first places
    __shared__ int places[6][kSelectWarps];
    __shared__ int base[6];
    __shared__ float cand_v[kSelectWarps][32];
    __shared__ int cand_c[kSelectWarps][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int lb = blockIdx.x * kSelectWarps + warp;
    const int blk = lb < a.nblocks ? chunk_block(a, lb) : -1;
    const bool live = blk >= 0;
    const float* z = logits + (size_t)(live ? lb : 0) * S.nout;
    bool confident = false, skip_p1 = false;
    int used = 0;
    uint16_t picks[kMaxProposals];
    if (live) {
        // the softmax maximum and each lane's best partitioning logit (absent classes: -infinity, which
        // adds 0 to the sum whatever the maximum is)
        float v[kHeld], mx = -3.0e38f, lm = -3.0e38f;
#pragma unroll
        for (int i = 0; i < kHeld; i++) { const int c = lane + 32 * i; v[i] = c <= S.p1 ? z[c] : -INFINITY; }
#pragma unroll
        for (int i = 0; i < kHeld; i++) { mx = fmaxf(mx, v[i]); if (lane + 32 * i != S.p1) lm = fmaxf(lm, v[i]); }
        for (int c = lane + 32 * kHeld; c <= S.p1; c += 32) { const float x = z[c]; mx = fmaxf(mx, x); if (c < S.p1) lm = fmaxf(lm, x); }
        mx = warp_max(mx);
        float se = 0.0f;
#pragma unroll
        for (int i = 0; i < kHeld; i++) se += __expf(v[i] - mx);
        for (int c = lane + 32 * kHeld; c <= S.p1; c += 32) se += __expf(z[c] - mx);
        se = warp_sum(se);
        const float p1 = __expf(z[S.p1] - mx) / se;
        // the masses only add to p1: at or above both limits the block is confident and proposes nothing
        confident = p1 >= sel.threshold && p1 >= sel.coverage && !r.confidence;
        if (!confident) {
            // The kmax-th largest of the 32 lane maxima bounds the kmax-th largest logit from below
            // (those lanes' maxima are kmax distinct logits at least that large), so only logits at
            // or above it can be among the kmax best.
            float theta = 3.0e38f;
            if (sel.kmax >= 1) {
                int rank = 0;  // lanes ahead of this one in (maximum descending, lane ascending) order
                for (int j = 0; j < 32; j++) {
                    const float o = __shfl_sync(kFull, lm, j);
                    rank += (o > lm || (o == lm && j < lane)) ? 1 : 0;
                }
                const uint32_t at = __ballot_sync(kFull, rank == sel.kmax - 1);
                theta = __shfl_sync(kFull, lm, __ffs(at) - 1);
            }
            // the partitionings at or above the bound, at most 32 of them kept
            int ncand = 0;
            auto collect = [&](float x, int c) {
                const bool in = x >= theta && x > -3.0e38f && c < S.p1;
                const uint32_t m = __ballot_sync(kFull, in);
                if (m == 0u) return;
                const int at = ncand + __popc(m & ((1u << lane) - 1u));
                if (in && at < 32) { cand_v[warp][at] = x; cand_c[warp][at] = c; }
                ncand += __popc(m);
            };
#pragma unroll
            for (int i = 0; i < kHeld; i++) collect(v[i], lane + 32 * i);
#pragma unroll 1
            for (int c0 = 32 * kHeld; c0 < S.p1; c0 += 32) collect(c0 + lane < S.p1 ? z[c0 + lane] : -3.0e38f, c0 + lane);
            __syncwarp();
            // the kmax best, by value, the first class of equal ones
            float mass[kMaxProposals];
            int n = 0;
            float acc = p1;
            uint32_t key = 0;
            int mine = 0x7FFFFFFF;
            if (lane < ncand) { key = okey(cand_v[warp][lane]); mine = cand_c[warp][lane]; }
            uint32_t last = 0xFFFFFFFFu;  // the last pick
            int last_c = -1;
#pragma unroll 1
            for (int k = 0; k < sel.kmax; k++) {
                if (ncand > 32) {  // (equal logits, or a large kmax) each lane's best after the last pick
                    key = 0; mine = 0x7FFFFFFF;
                    for (int c = lane; c < S.p1; c += 32) {
                        const float x = z[c];
                        if (!(x >= theta && x > -3.0e38f)) continue;
                        const uint32_t u = okey(x);
                        if ((u < last || (u == last && c > last_c)) && u > key) { key = u; mine = c; }
                    }
                }
                const uint32_t best = __reduce_max_sync(kFull, key);
                if (best == 0u) break;
                const uint32_t ci = __reduce_min_sync(kFull, key == best ? (uint32_t)mine : 0xFFFFFFFFu);
                if ((uint32_t)mine == ci) key = 0;
                last = best; last_c = (int)ci;
                picks[n] = (uint16_t)pick_of_class(S, (int)ci);
                acc += __expf(okey_value(best) - mx) / se;
                mass[n] = acc;
                n++;
            }
            confident = acc >= sel.threshold;
            if (r.confidence && lane == 0) r.confidence[lb] = acc;
            // propose the shortest best-first prefix whose mass reaches the coverage
            used = n;
            for (int k = 0; k < n; k++)
                if (mass[k] >= sel.coverage) { used = k + 1; break; }
            if (p1 >= sel.coverage) used = 0;
            skip_p1 = used > 0 && p1 < sel.p1_floor;
        }
    }
    // places in the lists
    if (lane < 6) {
        int n = 0;
        if (live && confident) {
            if (lane == 0) n = 1;
            else if (lane == 2) n = skip_p1 ? 0 : 1;
            else if (lane > 2) for (int k = 0; k < used; k++) n += (picks[k] >> 10) == lane - 3 ? 1 : 0;
        } else if (live && lane == 1) {
            n = 1;
        }
        places[lane][warp] = n;
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        int t = 0;
        for (int w = 0; w < kSelectWarps; w++) { const int n = places[threadIdx.x][w]; places[threadIdx.x][w] = t; t += n; }
        base[threadIdx.x] = t > 0 ? atomicAdd(&r.counts[threadIdx.x], t) : 0;
    }
    __syncthreads();
    if (!live) return;
    if (!confident) {
        if (lane == 0) { const int pos = base[1] + places[1][warp]; r.full[pos] = blk; r.full_err[pos] = 3e38f; }
        return;
    }
    const int pos = base[0] + places[0][warp];
    uint32_t heads = skip_p1 ? 0u : 1u;  // block-mode heads the front will read: P = 1 and the proposed counts
    for (int k = 0; k < used; k++) heads |= 2u << (picks[k] >> 10);
    if (lane == 0) {
        r.pruned[pos] = blk;
        PropPicks& pp = r.prop[pos];
        pp.n = (uint16_t)used;
        pp.flags = skip_p1 ? 1 : 0;
        for (int k = 0; k < kMaxProposals; k++) pp.v[k] = k < used ? picks[k] : 0;
        // the work list: slot 0 (P = 1) and one slot per proposed partitioning, by P
        if (!skip_p1) r.pb_list[base[2] + places[2][warp]] = (uint32_t)pos << 5;
        int at[3] = {base[3] + places[3][warp], base[4] + places[4][warp], base[5] + places[5][warp]};
        for (int k = 0; k < used; k++) {
            const int p = picks[k] >> 10;  // list 1 + p of P = 2 + p
            const int i = p == 0 ? at[0]++ : p == 1 ? at[1]++ : at[2]++;
            r.pb_list[(size_t)(1 + p) * r.pb_stride + i] = ((uint32_t)pos << 5) | (uint32_t)(k + 1);
        }
    }
    // block-mode masks: the kbm best modes of each needed head; lane l holds modes l + 32u.
    // When kbm covers every mode, each needed head's mask is every mode (the ranking would
    // pick them all).
    uint64_t* mk = r.masks + (size_t)pos * 4 * kMaskWords;
    if (sel.kbm >= S.nbm) {
        if (lane < 4 * kMaskWords) {
            const int p = lane / kMaskWords, w = lane % kMaskWords;
            const int lo = w * 64;
            const uint64_t all = S.nbm - lo >= 64 ? ~0ull : S.nbm > lo ? ((1ull << (S.nbm - lo)) - 1) : 0ull;
            mk[lane] = ((heads >> p) & 1) ? all : 0ull;
        }
        return;
    }
#pragma unroll 1
    for (int p = 0; p < 4; p++) {
        if (!((heads >> p) & 1)) continue;
        const float* h = z + S.head_base + p * S.nbm_pad;
        const uint64_t word = S.nbm <= 64 ? mode_mask<2>(h, S.nbm, sel.kbm, lane) : mode_mask<2 * kMaskWords>(h, S.nbm, sel.kbm, lane);
        if (lane < kMaskWords) mk[p * kMaskWords + lane] = word;
    }
}

}  // namespace

cudaError_t configure_mlp() {
    return cudaFuncSetAttribute(k_mlp_logits, cudaFuncAttributeMaxDynamicSharedMemorySize, kMlpSmemBytes);
}

cudaError_t launch_mlp_logits(const KernelArgs& a, const Net& net, float* logits, int* error_flag, cudaStream_t s) {
    const int grid = (a.nblocks + kTileRows - 1) / kTileRows;
    k_mlp_logits<<<grid, kMlpThreads, kMlpSmemBytes, s>>>(a, net, logits, error_flag);
    return cudaGetLastError();
}

cudaError_t launch_select(const KernelArgs& a, const Net& net, const float* logits, const Select& sel, const Routes& r,
                          cudaStream_t s) {
    const int grid = (a.nblocks + kSelectWarps - 1) / kSelectWarps;
    constexpr int threads = kSelectWarps * 32;
    k_select<<<grid, threads, 0, s>>>(a, net.s, logits, sel, r);
    return cudaGetLastError();
}

}  // namespace mlp
}  // namespace astcb200
