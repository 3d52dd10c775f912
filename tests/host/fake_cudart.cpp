// A CUDA runtime that runs nothing, on host memory: kernels, graphs and memsets are
// reported in the order in which a stream would come to them, and fail where the test says so.
#include <cstdlib>
#include <cstring>
#include <functional>
#include <vector>

#include <cuda_runtime_api.h>

bool fake_launch_fails(const void* kernel);
bool fake_graph_fails();
void fake_kernel_ran(const void* kernel);
void fake_cleared(void* p);

namespace {
using Work = std::function<void()>;
std::vector<Work> recorded;
std::vector<std::vector<Work>> graphs;
bool capturing = false;
cudaError_t last = cudaSuccess;

void submit(Work w) {
    if (capturing) recorded.push_back(w);
    else w();
}
cudaError_t launch(const void* f) {
    if (fake_launch_fails(f)) return last = cudaErrorMemoryAllocation;
    submit([f] { fake_kernel_ran(f); });
    return cudaSuccess;
}
cudaError_t clear(void* p) {
    submit([p] { fake_cleared(p); });
    return cudaSuccess;
}
}  // namespace

extern "C" {
// what compiled kernels call to register and launch themselves
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
char __cudaInitModule(void**) { return 0; }
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void*) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) { *k = (cudaKernel_t)f; return cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void**, size_t, cudaStream_t) { return launch((const void*)k); }
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t, cudaStream_t) { return launch(f); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void* f, void**) { return launch(f); }

cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { capturing = true; recorded.clear(); return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { capturing = false; *g = (cudaGraph_t)1; return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
    graphs.push_back(recorded);
    *e = (cudaGraphExec_t)graphs.size();  // its number + 1
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t) {
    if (fake_graph_fails()) return cudaErrorMemoryAllocation;
    for (const Work& w : graphs[(size_t)e - 1]) w();
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }

cudaError_t cudaMalloc(void** p, size_t n) { *p = std::calloc(1, n); return *p ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFree(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = std::malloc(n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemset(void* p, int, size_t) { return clear(p); }
cudaError_t cudaMemsetAsync(void* p, int, size_t, cudaStream_t) { return clear(p); }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)1; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) { *s = cudaStreamCaptureStatusNone; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)1; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)1; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1.f; return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t) { return "told to fail"; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) { *v = a == cudaDevAttrMultiProcessorCount ? 148 : 232448; return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) { std::memset(a, 0, sizeof(*a)); return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) { a->type = cudaMemoryTypeUnregistered; return cudaSuccess; }
}
