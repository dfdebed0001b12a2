// The device arrays' setup (host_ctx.h) against a CUDA runtime that only writes
// down its calls: what runs on the legacy stream has to be waited for before
// alloc() or upload() returns, since the contexts' streams do not wait for it.
#include <cstdio>
#include <cstdlib>

#include "../mallard_gb300/csrc/host_ctx.h"

static int pending = 0;  // operations on the legacy stream nobody has waited for
static bool legacy(cudaStream_t s) { return s == cudaStreamLegacy; }

extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) {
    *p = std::malloc(n);
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMemset(void*, int, size_t) {
    ++pending;
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void*, const void*, size_t, cudaMemcpyKind) {
    ++pending;
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    if (legacy(s)) pending = 0;
    return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
}

int main() {
    DevArray<double> a;
    a.alloc(100);
    std::printf("alloc=%d\n", pending);
    a.upload(std::vector<double>(50, 1.0));
    std::printf("upload=%d\n", pending);
    a.upload(std::vector<double>());
    std::printf("empty=%d\n", pending);
    return 0;
}
