// Device encodes that were given no stream run on their context's own, which nothing else is ordered
// with.  The entry points that read blocks on the legacy default stream (containers, decoding) wait
// for such an encode of the blocks they read; no other work of the process does.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

struct astcb200_ctx;

namespace astcb200 {

// Output ranges of a context's encodes without a stream since its stream was last waited for.
struct StreamlessOutputs {
    static constexpr int kMax = 64;  // more are kept as their hull
    struct Range { uintptr_t lo, hi; };
    Range r[kMax];
    int n = 0;
    cudaEvent_t done = nullptr;      // after the last of them
    StreamlessOutputs *prev = nullptr, *next = nullptr;  // every context's, while it exists
};

cudaError_t register_streamless(StreamlessOutputs& s);
void release_streamless(StreamlessOutputs& s);  // of a context whose stream has been waited for
// Blocks [p, p + bytes) were queued on `stream`: call it for each output, then record_streamless.
void add_streamless(StreamlessOutputs& s, const void* p, size_t bytes);
cudaError_t record_streamless(StreamlessOutputs& s, cudaStream_t stream);
void clear_streamless(StreamlessOutputs& s);  // the context's stream has been waited for
// A reader of [p, p + bytes) on `reader`: on the legacy default stream it waits for the encodes above.
cudaError_t await_streamless(const void* p, size_t bytes, cudaStream_t reader);

}  // namespace astcb200
