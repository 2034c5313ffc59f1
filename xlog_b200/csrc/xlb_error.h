// Failures on the host: the exception that carries a status to the C boundary, and calls of the CUDA
// runtime.  No device code, so that host-only parts of the library can be built without nvcc.
#pragma once
#include <cuda_runtime_api.h>

#include <cstdarg>
#include <cstdio>
#include <string>

#include "../../include/xlb.h"

struct XlbError {
    xlb_status st;
    std::string msg;
};

[[noreturn]] inline void xlb_fail(xlb_status st, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    throw XlbError{st, buf};
}

// A failing call of the runtime also leaves its error on the thread, for the next cudaGetLastError:
// left there it would be reported once more, as a failure of whatever is launched next.  So every call
// goes through one of these three, and whoever handles a failure has taken it off the thread.
// (cudaErrorNotReady, the answer of a query, is no error and never left there.)
inline cudaError_t cuda_take(cudaError_t e) {
    if (e != cudaSuccess && e != cudaErrorNotReady) cudaGetLastError();
    return e;
}
#define CUDA_OK(expr)                                                                            \
    do {                                                                                         \
        cudaError_t e__ = cuda_take(expr);                                                       \
        if (e__ != cudaSuccess)                                                                  \
            xlb_fail(e__ == cudaErrorMemoryAllocation ? XLB_ERR_RESOURCE_EXHAUSTED : XLB_ERR_CUDA, \
                     "%s failed: %s (%s:%d)", #expr, cudaGetErrorString(e__), __FILE__, __LINE__); \
    } while (0)
#define CUDA_QUIET(expr) ((void)cuda_take(expr))  // nothing can be done about a failure (a destructor, a timer)
