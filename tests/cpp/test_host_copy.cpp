// Copies into pageable memory (hila_b200/csrc/host_copy.cpp) over a fake CUDA runtime: without
// streams or page-locked chunks to be had, with only some, and with threads.  No GPU involved.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <vector>

#include "host_copy.h"

namespace {
std::mutex mu;
int streams_left, chunks_left, streams, chunks, copies, plain, last_error, copy_fails;
}  // namespace

extern "C" {
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
    if (streams_left-- <= 0) return (cudaError_t)(last_error = cudaErrorMemoryAllocation);
    streams++;
    *s = (cudaStream_t)&streams;
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return streams--, cudaSuccess; }
cudaError_t cudaMallocHost(void **p, size_t n) {
    if (chunks_left-- <= 0) return (cudaError_t)(last_error = cudaErrorMemoryAllocation);
    chunks++;
    *p = std::malloc(n);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) { return chunks--, std::free(p), cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *) {
    a->type = cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t st) {
    std::lock_guard<std::mutex> lk(mu);
    copies++;
    if (!st) plain++;
    if (copy_fails) return cudaErrorUnknown;
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetLastError() {
    const int e = last_error;
    last_error = 0;
    return (cudaError_t)e;
}
const char *cudaGetErrorString(cudaError_t) { return "made to fail"; }
}
void hw::set_error(const char *, ...) {}

int main() {
    int failures = 0;
    const size_t sizes[] = {1, hw::kCopyMin - 1, hw::kCopyMin, 3 * hw::kCopyChunk + 5, 11 * hw::kCopyChunk};
    for (size_t bytes : sizes)
        for (int ns : {0, 1, 2, 99})
            for (int nc : {0, 1, 3, 99}) {
                std::vector<char> src(bytes), dst(bytes, 1);
                for (size_t i = 0; i < bytes; i++) src[i] = (char)(i * 2654435761u >> 13);
                streams_left = ns, chunks_left = nc, copies = plain = 0;
                {
                    hw::HostCopier C;
                    const int rc = C.copy(0, nullptr, dst.data(), src.data(), bytes);
                    const bool threads = bytes >= hw::kCopyMin && ns >= 2 && nc >= 2;
                    if (rc != HW_OK || dst != src || last_error || (plain == 0) != threads) {
                        std::printf("FAILED: %zu bytes, %d streams, %d chunks: %d\n", bytes, ns, nc, rc);
                        failures++;
                    }
                    streams_left = chunks_left = 99;  // to be had again
                    std::fill(dst.begin(), dst.end(), 1);
                    if (C.copy(0, nullptr, dst.data(), src.data(), bytes) != HW_OK || dst != src) failures++;
                    copy_fails = 1;
                    if (C.copy(0, nullptr, dst.data(), src.data(), bytes) != HW_ERR_CUDA) failures++;
                    copy_fails = 0;
                }
                if (streams || chunks) failures++;
            }
    if (failures == 0) std::printf("host copies passed\n");
    return failures;
}
