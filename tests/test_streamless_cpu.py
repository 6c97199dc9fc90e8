"""Which readers wait for encodes that were given no stream, with the CUDA calls replaced by counters."""
import os
import subprocess

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "astc_implementation_b200", "csrc")

PROGRAM = r"""
#include "streamless.h"
#include <cstdio>
#include <cstdlib>
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); std::exit(1); } } while (0)

static int events = 0, records = 0, waits = 0;
static cudaEvent_t last = nullptr;
extern "C" {
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)(uintptr_t)(++events); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { records++; return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t e, unsigned) { waits++; last = e; return cudaSuccess; }
}
using namespace astcb200;

static int read(uintptr_t at, size_t n, cudaStream_t s = nullptr) {
    waits = 0;
    CHECK(await_streamless((const void*)at, n, s) == cudaSuccess);
    return waits;
}

int main() {
    StreamlessOutputs a, b;
    CHECK(register_streamless(a) == cudaSuccess && register_streamless(b) == cudaSuccess);
    cudaStream_t own = (cudaStream_t)(uintptr_t)0x100;
    CHECK(read(0, ~(size_t)0) == 0);
    add_streamless(a, (void*)0x1000, 0x100);
    CHECK(record_streamless(a, own) == cudaSuccess && records == 1);
    CHECK(read(0x1000, 16) == 1 && last == a.done);
    CHECK(read(0x10FF, 1) == 1 && read(0x1100, 16) == 0 && read(0xFF0, 16) == 0 && read(0xFF0, 17) == 1);
    CHECK(read(0x1000, 16, cudaStreamLegacy) == 1);
    CHECK(read(0x1000, 16, own) == 0);  // a caller with a stream orders it itself
    add_streamless(b, (void*)0x1080, 0x100);
    CHECK(record_streamless(b, own) == cudaSuccess);
    CHECK(read(0x1000, 16) == 1 && read(0x1090, 16) == 2 && read(0x1170, 16) == 1 && last == b.done);
    clear_streamless(a);
    CHECK(read(0x1000, 16) == 0 && read(0x1090, 16) == 1);
    for (int i = 0; i < 1000; i++) add_streamless(a, (void*)(uintptr_t)(0x100000 + 0x1000 * i), 0x10);  // bounded, none lost
    CHECK(a.n <= StreamlessOutputs::kMax);
    for (int i = 0; i < 1000; i++) CHECK(read(0x100000 + 0x1000 * i, 16) == 1);
    release_streamless(b);
    CHECK(read(0x1090, 16) == 0);
    release_streamless(a);
    release_streamless(a);
    CHECK(read(0, ~(size_t)0) == 0);
    return 0;
}
"""


def test_readers_wait_for_the_encodes_of_their_blocks_only(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", CSRC, "-I", "/usr/local/cuda/include", str(src),
                           os.path.join(CSRC, "streamless.cpp"), "-o", str(exe), "-pthread"])
    subprocess.check_call([str(exe)])
