#include "fake_runtime.h"

std::vector<Call> calls;
Runtime runtime;

extern "C" {
cudaError_t cudaMalloc(void** p, size_t bytes) { *p = std::malloc(bytes); return cudaSuccess; }
cudaError_t cudaFree(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() {
    const cudaError_t e = runtime.last;
    runtime.last = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    *e = static_cast<cudaEvent_t>(std::malloc(1));
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) { std::free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { calls.push_back({"record", s, e}); return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
    calls.push_back({"wait", s, e});
    return cudaSuccess;
}
cudaError_t cudaStreamQuery(cudaStream_t s) {
    calls.push_back({"query", s, nullptr});
    return runtime.last = runtime.query();
}
cudaError_t cudaGetDeviceCount(int* count) { *count = 2; return cudaSuccess; }
cudaError_t cudaMemcpy(void* to, const void*, size_t, cudaMemcpyKind) {
    calls.push_back({"copy", nullptr, to});
    return cudaSuccess;
}
cudaError_t cudaGetDeviceFlags(unsigned* flags) { *flags = runtime.flags; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    calls.push_back({"synchronize", s, nullptr});
    return runtime.synchronize;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* kernel, void**) {
    calls.push_back({"launch", c->stream, kernel});
    return runtime.launch;
}
}

// Registration of a program's device code, of which there is none to run.
extern "C" {
void** __cudaRegisterFatBinary(void*) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
char __cudaInitModule(void**) { return 0; }
}
