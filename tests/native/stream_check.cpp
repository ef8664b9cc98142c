// A call's stream and buffers at its end, against a CUDA runtime of this file that writes down what
// it is asked for: the stream is waited for before it goes, after its buffers were freed on it.
#include <stdio.h>

#include <string>

#include "train_common.h"

static std::string calls;
static int freed;

extern "C" {
cudaError_t cudaMalloc(void **p, size_t) { return *p = &freed, cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaFree(void *) { return calls += "free ", cudaSuccess; }
cudaError_t cudaFreeAsync(void *, cudaStream_t s) { return calls += s ? "free-on-stream " : "free-on-null ", cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return calls += "wait ", cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return calls += "destroy ", cudaSuccess; }
}

namespace cumf {
cudaError_t scratch_alloc(void **p, size_t, cudaStream_t) { return *p = &freed, cudaSuccess; }
}

using namespace cumf;

static cudaStream_t handle() { return reinterpret_cast<cudaStream_t>(&freed); }

static int call(bool fails) {  // as the calls of the library are laid out
    Stream stream;
    stream.s = handle();
    DevBuf a, b;
    if (a.alloc(100, stream.s) != cudaSuccess) return 1;
    if (fails) return 1;  // with a copy still in flight
    return b.alloc(100) != cudaSuccess;
}

static int bad = 0;

static void expect(const char *what, const std::string &want) {
    if (calls != want) {
        printf("%s: %s, want %s\n", what, calls.c_str(), want.c_str());
        ++bad;
    }
    calls.clear();
}

int main() {
    call(false);
    expect("call", "free free-on-stream wait destroy ");
    call(true);
    expect("failed call", "free-on-stream wait destroy ");
    { Stream none; }
    expect("no stream", "");
    printf("bad %d\n", bad);
    return bad != 0;
}
