// A stand-in for the few calls of the CUDA runtime that the host-only parts of the library make: each
// call can be told to fail, and a failure stays on the thread until it is taken, as the runtime's does.
#pragma once
#include <cuda_runtime_api.h>

#include <atomic>
#include <chrono>
#include <thread>

struct FakeRuntime {
    std::atomic<int> fail_register{0}, fail_unregister{0};
    std::atomic<int> register_ms{0};       // how long a registration takes
    std::atomic<int> registered{0};        // blocks registered now
    std::atomic<int> last_device{-1};      // device current on the thread of the last (un)registration
    std::atomic<int> touched_devices{0};   // bit d: device d was made current, or used, by some thread
};
static FakeRuntime fake;
static thread_local cudaError_t fake_left = cudaSuccess;
static thread_local int fake_device = 0;

static cudaError_t fake_end(cudaError_t e) {
    if (e != cudaSuccess) fake_left = e;
    return e;
}
static void fake_use() {
    fake.last_device = fake_device;
    fake.touched_devices |= 1 << fake_device;
}
extern "C" {
cudaError_t cudaGetLastError(void) {
    const cudaError_t e = fake_left;
    fake_left = cudaSuccess;
    return e;
}
cudaError_t cudaPeekAtLastError(void) { return fake_left; }
const char* cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaGetDevice(int* d) {
    *d = fake_device;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int d) {
    fake_device = d;
    fake.touched_devices |= 1 << d;
    return cudaSuccess;
}
cudaError_t cudaHostRegister(void*, size_t, unsigned) {
    fake_use();
    std::this_thread::sleep_for(std::chrono::milliseconds(fake.register_ms));
    if (fake.fail_register) return fake_end(cudaErrorMemoryAllocation);
    ++fake.registered;
    return cudaSuccess;
}
cudaError_t cudaHostUnregister(void*) {
    fake_use();
    --fake.registered;
    return fake_end(fake.fail_unregister ? cudaErrorHostMemoryNotRegistered : cudaSuccess);
}
}
