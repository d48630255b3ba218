// The CUDA runtime calls that the library's host code makes, recorded instead
// of run: a program linked with fake_runtime.cpp in place of the runtime tests
// the host's side of stream ordering and error handling without a GPU.
#pragma once
#include <cuda_runtime_api.h>

#include <cstdio>
#include <cstdlib>
#include <functional>
#include <string>
#include <vector>

struct Call {
    std::string name;
    const void* stream;
    const void* object;
};
extern std::vector<Call> calls;

// What the calls return.
struct Runtime {
    cudaError_t last = cudaSuccess;         // the thread's last error
    cudaError_t launch = cudaSuccess;       // of a kernel launch (not noted as the last error)
    cudaError_t synchronize = cudaSuccess;  // of cudaStreamSynchronize
    unsigned flags = cudaDeviceScheduleAuto | cudaDeviceMapHost;
    std::function<cudaError_t()> query;     // of cudaStreamQuery (noted as the last error)
};
extern Runtime runtime;

#define EXPECT(x)                                                              \
    do {                                                                       \
        if (!(x)) {                                                            \
            std::printf("%s:%d: %s does not hold\n", __FILE__, __LINE__, #x);  \
            std::exit(1);                                                      \
        }                                                                      \
    } while (0)

inline cudaStream_t stream(size_t i) { return reinterpret_cast<cudaStream_t>(16 * i); }
