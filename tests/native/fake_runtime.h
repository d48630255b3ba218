// The CUDA runtime calls that the library's host code makes, recorded instead
// of run: a program linked with fake_runtime.cpp in place of the runtime tests
// the host's side of stream ordering and error handling without a GPU.
#pragma once
#include <cuda_runtime_api.h>

#include <cstdio>
#include <cstdlib>
#include <string>
#include <vector>

struct Call {
    std::string name;
    const void* stream;
    const void* object;
};
extern std::vector<Call> calls;

#define EXPECT(x)                                                              \
    do {                                                                       \
        if (!(x)) {                                                            \
            std::printf("%s:%d: %s does not hold\n", __FILE__, __LINE__, #x);  \
            std::exit(1);                                                      \
        }                                                                      \
    } while (0)

inline cudaStream_t stream(size_t i) { return reinterpret_cast<cudaStream_t>(16 * i); }
