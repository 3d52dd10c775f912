// The CUDA runtime calls of the read-back code on host memory, counted, for a
// machine without a GPU: "device" memory is host memory and every copy is done when it
// is queued.
#pragma once

#include <cstdlib>
#include <cstring>

#include <cuda_runtime.h>

struct FakeCounts {
    int syncs = 0, copies = 0, pins = 0, unpins = 0;
    size_t pinned = 0;
};
inline FakeCounts fake;
inline char* fake_pinned[2] = {};  // a caller's pinned range

extern "C" {
inline cudaError_t cudaStreamSynchronize(cudaStream_t) { ++fake.syncs; return cudaSuccess; }
inline cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    __atomic_add_fetch(&fake.copies, 1, __ATOMIC_RELAXED);
    std::memcpy(d, s, n);
    return cudaSuccess;
}
inline cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
    ++fake.pins;
    fake.pinned += n;
    *p = std::malloc(n);
    return cudaSuccess;
}
inline cudaError_t cudaFreeHost(void* p) { ++fake.unpins; std::free(p); return cudaSuccess; }
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
inline cudaError_t cudaSetDevice(int) { return cudaSuccess; }
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = reinterpret_cast<cudaEvent_t>(1); return cudaSuccess; }
inline cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
inline cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
inline cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    const char* c = static_cast<const char*>(p);
    a->type = c >= fake_pinned[0] && c < fake_pinned[1] ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
}
