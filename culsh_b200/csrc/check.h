// Error plumbing of the host code.
#pragma once

#include <cuda_runtime_api.h>

#include <cstdarg>
#include <cstddef>
#include <cstdio>
#include <stdexcept>
#include <string>

#include "../../include/culsh_b200.h"

namespace culsh_b200 {

// ---------------------------------------------------------------------------------------
// Errors: host code throws Error, the C ABI catches it and returns the status code.
// ---------------------------------------------------------------------------------------
struct Error : public std::runtime_error {
    int status;
    Error(int s, const std::string& m) : std::runtime_error(m), status(s) {}
};

[[noreturn]] inline void fail(int status, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    throw Error(status, buf);
}

#define CU_CHECK(call)                                                                      \
    do {                                                                                    \
        cudaError_t e__ = (call);                                                           \
        if (e__ != cudaSuccess)                                                             \
            ::culsh_b200::fail(e__ == cudaErrorMemoryAllocation ? CULSH_ERR_ALLOC           \
                                                                : CULSH_ERR_CUDA,           \
                               "%s failed: %s (%s:%d)", #call, cudaGetErrorString(e__),     \
                               __FILE__, __LINE__);                                         \
    } while (0)

inline size_t ceil_div(size_t a, size_t b) { return (a + b - 1) / b; }

}  // namespace culsh_b200
