#include "streamless.h"

#include <algorithm>
#include <mutex>

namespace astcb200 {

namespace {

std::mutex g_mutex;                    // of the list and of every entry in it
StreamlessOutputs* g_first = nullptr;

bool is_legacy(cudaStream_t s) { return s == nullptr || s == cudaStreamLegacy; }

}  // namespace

cudaError_t register_streamless(StreamlessOutputs& s) {
    const cudaError_t e = cudaEventCreateWithFlags(&s.done, cudaEventDisableTiming);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> g(g_mutex);
    s.next = g_first;
    if (g_first) g_first->prev = &s;
    g_first = &s;
    return cudaSuccess;
}

void release_streamless(StreamlessOutputs& s) {
    if (!s.done) return;
    {
        std::lock_guard<std::mutex> g(g_mutex);
        (s.prev ? s.prev->next : g_first) = s.next;
        if (s.next) s.next->prev = s.prev;
    }
    cudaEventDestroy(s.done);
    s.done = nullptr;
}

void add_streamless(StreamlessOutputs& s, const void* p, size_t bytes) {
    const uintptr_t lo = (uintptr_t)p, hi = lo + bytes;
    std::lock_guard<std::mutex> g(g_mutex);
    for (int i = 0; i < s.n; i++)
        if (lo <= s.r[i].hi && s.r[i].lo <= hi) {  // overlapping or adjacent
            s.r[i] = {std::min(lo, s.r[i].lo), std::max(hi, s.r[i].hi)};
            return;
        }
    if (s.n < StreamlessOutputs::kMax) {
        s.r[s.n++] = {lo, hi};
        return;
    }
    StreamlessOutputs::Range hull{lo, hi};
    for (int i = 0; i < s.n; i++) hull = {std::min(hull.lo, s.r[i].lo), std::max(hull.hi, s.r[i].hi)};
    s.r[0] = hull;
    s.n = 1;
}

cudaError_t record_streamless(StreamlessOutputs& s, cudaStream_t stream) {
    std::lock_guard<std::mutex> g(g_mutex);
    return cudaEventRecord(s.done, stream);
}

void clear_streamless(StreamlessOutputs& s) {
    std::lock_guard<std::mutex> g(g_mutex);
    s.n = 0;
}

cudaError_t await_streamless(const void* p, size_t bytes, cudaStream_t reader) {
    if (!is_legacy(reader)) return cudaSuccess;
    const uintptr_t lo = (uintptr_t)p, hi = lo + bytes;
    std::lock_guard<std::mutex> g(g_mutex);
    for (const StreamlessOutputs* s = g_first; s; s = s->next)
        for (int i = 0; i < s->n; i++)
            if (lo < s->r[i].hi && s->r[i].lo < hi) {
                const cudaError_t e = cudaStreamWaitEvent(reader, s->done, 0);
                if (e != cudaSuccess) return e;
                break;
            }
    return cudaSuccess;
}

}  // namespace astcb200
