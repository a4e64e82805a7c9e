// A stand-in for the parts of the CUDA runtime that libfbp calls, for tests of
// its host code without a GPU (loaded in front of libcudart): memory is host
// memory, kernels are counted instead of run, and an allocation can be made to
// fail.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <set>

static std::set<void*> live;
static int fail_in = 0;  // > 0: that many allocations from now, one fails
static int launches = 0, graph_launches = 0;
static int* token() { return static_cast<int*>(std::calloc(1, sizeof(int))); }

extern "C" {

void fake_fail_allocation(int n) { fail_in = n; }
int fake_launches() { return launches; }
int fake_graph_launches() { return graph_launches; }
int fake_live_allocations() { return (int)live.size(); }

cudaError_t cudaGetDeviceCount(int* n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaPeekAtLastError() { return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) {
    std::memset(p, 0, sizeof *p);
    p->major = 10;
    p->minor = 3;
    p->multiProcessorCount = 152;
    p->sharedMemPerBlockOptin = 227 * 1024;
    return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t n) {
    if (fail_in > 0 && --fail_in == 0) return *p = nullptr, cudaErrorMemoryAllocation;
    *p = std::calloc(1, n ? n : 1);
    live.insert(*p);
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    if (p && !live.erase(p)) return cudaErrorInvalidValue;
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int v, size_t n) { return std::memset(p, v, n), cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { return std::memset(p, v, n), cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    return std::memcpy(d, s, n), cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) { return std::memset(a, 0, sizeof *a), cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
    return *n = 2, cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return *e = (cudaEvent_t)token(), cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return std::free(e), cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return *s = (cudaStream_t)token(), cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { return std::free(s), cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { return *g = (cudaGraph_t)token(), cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
    return *e = (cudaGraphExec_t)token(), cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return ++graph_launches, cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { return std::free(g), cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { return std::free(e), cudaSuccess; }

unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void*) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* m, void*) {
    return *g = dim3{1, 1, 1}, *b = dim3{1, 1, 1}, *m = 0, cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t*, const void*) { return cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3, dim3, void**, size_t, cudaStream_t) { return ++launches, cudaSuccess; }
}
