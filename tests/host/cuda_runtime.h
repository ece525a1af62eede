// The few CUDA calls that csrc/cuda/host_copy.hpp makes, on host memory: copies are done at once, and
// from the `fail_after`-th on they fail, the first with error 1, the later ones with error 2 a while later.
#pragma once

#include <atomic>
#include <chrono>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <thread>

typedef int cudaError_t;
typedef void* cudaStream_t;
typedef void* cudaEvent_t;
enum { cudaSuccess = 0, cudaHostRegisterDefault = 0, cudaMemoryTypeUnregistered = 0, cudaEventDisableTiming = 2, cudaStreamNonBlocking = 1, cudaMemcpyDeviceToHost = 2 };
struct cudaPointerAttributes {
    int type;
};

namespace fake {
inline std::atomic<int> copies{0};
inline int fail_after = 1 << 30;
inline bool may_register = true;
}  // namespace fake

inline cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) { a->type = cudaMemoryTypeUnregistered; return cudaSuccess; }
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline cudaError_t cudaSetDevice(int) { return cudaSuccess; }
inline cudaError_t cudaMallocHost(char** p, uint64_t bytes) { *p = static_cast<char*>(std::malloc(bytes)); return cudaSuccess; }
inline cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
inline cudaError_t cudaHostRegister(void*, uint64_t, int) { return fake::may_register ? cudaSuccess : 1; }
inline cudaError_t cudaHostUnregister(void*) { return cudaSuccess; }
inline cudaError_t cudaHostGetDevicePointer(void** device, void* host, int) { *device = host; return cudaSuccess; }
inline cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, int) { *s = s; return cudaSuccess; }
inline cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, int) { return cudaSuccess; }
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, int) { *e = e; return cudaSuccess; }
inline cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
inline cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
inline cudaError_t cudaMemcpyAsync(void* to, const void* from, uint64_t bytes, int, cudaStream_t) {
    const int n = fake::copies++;
    if (n > fake::fail_after) {
        std::this_thread::sleep_for(std::chrono::milliseconds(100));
        return 2;
    }
    if (n == fake::fail_after) return 1;
    std::memcpy(to, from, bytes);
    return cudaSuccess;
}
