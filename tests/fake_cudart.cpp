// fake_cudart.cpp — the CUDA runtime calls of batch.cu without a GPU: memory is host
// memory, copies are done at once, a stream knows the launches before its next one
// and an event is a copy of that set.  Stream capture is refused.
#include "fake_cudart.h"

#include <cstdlib>
#include <cstring>

extern "C" {
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "injected"; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) { return *p = std::calloc(1, n), cudaSuccess; }
cudaError_t cudaFree(void* p) { return std::free(p), cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return cudaMalloc(p, n); }
cudaError_t cudaFreeHost(void* p) { return cudaFree(p); }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
  return std::memcpy(d, s, n), cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  return std::memcpy(d, s, n), cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  return *s = reinterpret_cast<cudaStream_t>(new Stream), cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { return delete &of(s), cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
  const Stream& x = *reinterpret_cast<Stream*>(e);
  of(s).before.insert(x.before.begin(), x.before.end());
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  return *e = reinterpret_cast<cudaEvent_t>(new Stream), cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return delete reinterpret_cast<Stream*>(e), cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  return reinterpret_cast<Stream*>(e)->before = of(s).before, cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 1.f, cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorUnknown; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t*) { return cudaErrorUnknown; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t*, cudaGraph_t, unsigned long long) {
  return cudaErrorUnknown;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorUnknown; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
// what the compiler adds to a file with device code
void** __cudaRegisterFatBinary(void*) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*,
                            dim3*, int*) {}
}
