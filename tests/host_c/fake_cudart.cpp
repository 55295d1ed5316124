// The CUDA runtime calls of a batch step, doing nothing but note which streams
// have work that the host has not waited for.
#include <cuda_runtime_api.h>

#include <cstdint>
#include <set>

std::set<cudaStream_t> busy;
int refuse_graph;
const void* device_memory;   // the one address that is device memory; all others are unregistered host memory

static cudaStream_t next_stream() {
    static uintptr_t n = 0x1000;
    return (cudaStream_t)(n += 16);
}
extern "C" {
cudaError_t cudaStreamCreate(cudaStream_t* s) { return *s = next_stream(), cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return *e = (cudaEvent_t)next_stream(), cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return busy.clear(), cudaSuccess; }   // the joined origin stream
cudaError_t cudaStreamSynchronize(cudaStream_t s) { return busy.erase(s), cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { return *g = nullptr, cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* g, cudaGraph_t, unsigned long long) {
    return *g = nullptr, refuse_graph ? cudaErrorInvalidValue : cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    a->type = p == device_memory ? cudaMemoryTypeDevice : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t*, int) { return cudaErrorNotSupported; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMallocAsync(void**, size_t, cudaStream_t) { return cudaErrorNotSupported; }
cudaError_t cudaFreeAsync(void*, cudaStream_t) { return cudaSuccess; }
// what nvcc's start-up code calls
void** __cudaRegisterFatBinary(void*) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
char __cudaInitModule(void**) { return 1; }
}
