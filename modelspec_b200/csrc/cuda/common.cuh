// Shared device helpers and the host-side launch check.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <initializer_list>
#include <set>
#include <stdexcept>
#include <string>
#include <vector>

namespace msx {
namespace k {

struct CudaError : std::runtime_error {
    cudaError_t code;
    CudaError(const std::string& what, cudaError_t c) : std::runtime_error(what), code(c) {}
};

inline void check(cudaError_t e, const char* what) {
    if (e != cudaSuccess)
        throw CudaError(std::string(what) + ": " + cudaGetErrorName(e) + " (" + cudaGetErrorString(e) + ")", e);
}

// After a kernel launch: reports a launch-configuration error without synchronising. The error
// is taken (cudaGetLastError), not peeked at, so a non-sticky error that this thread left behind
// earlier (the host application's own, or an earlier launch here) is reported once and does not
// fail every later launch.
inline void check_launch(const char* kernel) { check(cudaGetLastError(), kernel); }

// Allows `kernel` its dynamic shared memory on the current device. The attribute is per device: it is
// set when the device changes (a second thread that sees a stale value only sets it once more).
template <class Kernel> inline void set_shared_memory(Kernel kernel, int bytes, std::atomic<int>& configured_device) {
    int device = 0;
    check(cudaGetDevice(&device), "cudaGetDevice");
    if (device == configured_device.load(std::memory_order_relaxed)) return;
    check(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes), "dynamic shared memory");
    configured_device.store(device, std::memory_order_relaxed);
}

// The SMs of the current device.
inline uint32_t device_sm_count() {
    static std::atomic<int> counted_device{-1};
    static std::atomic<uint32_t> count{0};
    int device = 0, sms = 0;
    check(cudaGetDevice(&device), "cudaGetDevice");
    if (device == counted_device.load(std::memory_order_acquire)) return count.load(std::memory_order_relaxed);
    check(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device), "cudaDeviceGetAttribute");
    count.store(static_cast<uint32_t>(sms), std::memory_order_relaxed);
    counted_device.store(device, std::memory_order_release);
    return static_cast<uint32_t>(sms);
}

// ---- kernels that start while the one before them ends -------------------------------------------
// In a step's graph a kernel may be launched as soon as every block of the kernel before it has come this far
// (msx_run turns the edges between kernels into programmatic ones). Each waits here until that one is complete and
// its writes are visible, and only then lets the next one start: whatever a kernel reads or writes in memory comes
// after this call. Kernels whose blocks fill an SM wait first and let the next one start late, with their last loads
// (blocks that stand there early keep the kernels of the side stream from the idle SMs, and gather on those: as early
// as this, the f32 attention made a BERT-tiny step 21 us longer), and only with tensor memory of their own in hand: a block must not wait for tensor
// memory that a block waiting for it has taken.
// Between two kernels of a graph 0.85 us pass, 0.63 so, and a tensor-core kernel's barriers and tensor memory are set
// up under the end of the kernel before.
__device__ __forceinline__ void wait_for_producers() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void after_producers() {
    wait_for_producers();
    let_next_start();
}

// What the launches of a step being captured on this thread say of their kernels, while the runtime asks.
struct CaptureNotes {
    std::set<cudaGraphNode_t> side;      // on the side stream
    std::set<cudaGraphNode_t> in_order;  // better started when the kernel before has ended
};
inline thread_local CaptureNotes* capture_notes = nullptr;
struct NoteCapture {
    explicit NoteCapture(CaptureNotes* notes) { capture_notes = notes; }
    ~NoteCapture() { capture_notes = nullptr; }
    NoteCapture(const NoteCapture&) = delete;
    NoteCapture& operator=(const NoteCapture&) = delete;
};
// The nodes that the next one captured on `s` will follow: after a launch, its kernel.
inline std::vector<cudaGraphNode_t> captured_last(cudaStream_t s) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    const cudaGraphNode_t* last = nullptr;
    size_t count = 0;
    check(cudaStreamGetCaptureInfo_v2(s, &status, nullptr, nullptr, &last, &count), "cudaStreamGetCaptureInfo");
    if (status != cudaStreamCaptureStatusActive) return {};
    return {last, last + count};
}
// The kernel just launched on `s` is one of those.
inline void starts_in_order(cudaStream_t s) {
    if (!capture_notes) return;
    for (cudaGraphNode_t node : captured_last(s)) capture_notes->in_order.insert(node);
}

// A load of what another kernel of the step may have written. The read-only path (__ldg, ld.global.nc, a kernel's `const
// __restrict__` parameter) is for memory that nobody writes while the kernel runs, which a kernel that starts early does not
// know, and the compiler may move such a load in front of the wait above. So: ordinary loads, and no __restrict__ on
// a kernel's parameters (on those of a function in its body it tells the accesses there apart, no more).
template <class T> __device__ __forceinline__ T load_global(const T* p) { return *p; }

// Where a kernel's stores keep the compiler from moving such loads together (they may be to the same memory, for all it
// knows), and registers or unrolled loops ask for that: a pointer made here, behind the wait, and loads that the compiler may place
// anywhere its value is known. For memory that the kernel itself does not write before it has read it.
// (A BERT-tiny step in mixed precision 350 us, 355 with ordinary loads in the layer norms' gradients and the column sums.)
template <class T> struct Settled {
    const T* p;
    __device__ __forceinline__ Settled operator+(uint64_t n) const { return {p + n}; }
    __device__ __forceinline__ explicit operator bool() const { return p != nullptr; }
};
template <class T> __device__ __forceinline__ Settled<T> settled(const T* p) {
    asm volatile("" : "+l"(p)::"memory");
    return {p};
}
template <class V> __device__ __forceinline__ V load_settled(const void* p);
template <> __device__ __forceinline__ uint16_t load_settled<uint16_t>(const void* p) {
    uint16_t v;
    asm("ld.global.u16 %0, [%1];" : "=h"(v) : "l"(p));
    return v;
}
template <> __device__ __forceinline__ uint32_t load_settled<uint32_t>(const void* p) {
    uint32_t v;
    asm("ld.global.b32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
template <> __device__ __forceinline__ uint2 load_settled<uint2>(const void* p) {
    uint2 v;
    asm("ld.global.v2.b32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}
template <> __device__ __forceinline__ uint4 load_settled<uint4>(const void* p) {
    uint4 v;
    asm("ld.global.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

// ---- elements of either storage type ------------------------------------------------------------
// A mixed-precision plan stores activations as bf16; the kernels that touch them are templates on
// the element type and compute in f32 whatever it is. One element, or four consecutive ones (16
// bytes of f32, 8 bytes of bf16; the address a multiple of that).
using bf16 = __nv_bfloat16;
__device__ __forceinline__ float load1(const float* p) { return load_global(p); }
__device__ __forceinline__ float load1(const bf16* p) { return __bfloat162float(*p); }
__device__ __forceinline__ void store1(float* p, float v) { *p = v; }
__device__ __forceinline__ void store1(bf16* p, float v) { *p = __float2bfloat16_rn(v); }
// Two consecutive elements (the address a multiple of their size).
__device__ __forceinline__ float2 load2(const float* p) { return load_global(reinterpret_cast<const float2*>(p)); }
__device__ __forceinline__ float2 load2(const bf16* p) {
    const uint32_t raw = load_global(reinterpret_cast<const uint32_t*>(p));
    return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw));
}
__device__ __forceinline__ void store2(float* p, float2 v) { *reinterpret_cast<float2*>(p) = v; }
__device__ __forceinline__ void store2(bf16* p, float2 v) {
    const __nv_bfloat162 pair = __floats2bfloat162_rn(v.x, v.y);
    *reinterpret_cast<uint32_t*>(p) = *reinterpret_cast<const uint32_t*>(&pair);
}
__device__ __forceinline__ float4 four_halves(const uint2& raw) {
    const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
    const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
    return make_float4(lo.x, lo.y, hi.x, hi.y);
}
__device__ __forceinline__ float4 load4(const float* p) { return load_global(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ float4 load4(const bf16* p) { return four_halves(load_global(reinterpret_cast<const uint2*>(p))); }
__device__ __forceinline__ float load1(Settled<float> s) { return __uint_as_float(load_settled<uint32_t>(s.p)); }
__device__ __forceinline__ float load1(Settled<bf16> s) { return __uint_as_float(static_cast<uint32_t>(load_settled<uint16_t>(s.p)) << 16); }
__device__ __forceinline__ float4 load4(Settled<float> s) {
    const uint4 raw = load_settled<uint4>(s.p);
    return make_float4(__uint_as_float(raw.x), __uint_as_float(raw.y), __uint_as_float(raw.z), __uint_as_float(raw.w));
}
__device__ __forceinline__ float4 load4(Settled<bf16> s) { return four_halves(load_settled<uint2>(s.p)); }
__device__ __forceinline__ void store4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void store4(bf16* p, float4 v) {
    const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
    uint2 raw;
    raw.x = *reinterpret_cast<const uint32_t*>(&lo);
    raw.y = *reinterpret_cast<const uint32_t*>(&hi);
    *reinterpret_cast<uint2*>(p) = raw;
}
// Eight consecutive bf16 elements (16 bytes; the address a multiple of 16).
struct float8 {
    float4 lo, hi;
};
__device__ __forceinline__ float8 eight_halves(const uint4& raw) {
    return {four_halves(make_uint2(raw.x, raw.y)), four_halves(make_uint2(raw.z, raw.w))};
}
__device__ __forceinline__ float8 load8(const bf16* p) { return eight_halves(load_global(reinterpret_cast<const uint4*>(p))); }
__device__ __forceinline__ float8 load8(Settled<bf16> s) { return eight_halves(load_settled<uint4>(s.p)); }
__device__ __forceinline__ void store8(bf16* p, const float8& v) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(v.lo.x, v.lo.y), b = __floats2bfloat162_rn(v.lo.z, v.lo.w);
    const __nv_bfloat162 c = __floats2bfloat162_rn(v.hi.x, v.hi.y), d = __floats2bfloat162_rn(v.hi.z, v.hi.w);
    uint4 raw;
    raw.x = *reinterpret_cast<const uint32_t*>(&a);
    raw.y = *reinterpret_cast<const uint32_t*>(&b);
    raw.z = *reinterpret_cast<const uint32_t*>(&c);
    raw.w = *reinterpret_cast<const uint32_t*>(&d);
    *reinterpret_cast<uint4*>(p) = raw;
}
// `v` as an array of that element type would hold it.
__device__ __forceinline__ float stored_as(float v, const float*) { return v; }
__device__ __forceinline__ float stored_as(float v, const bf16*) { return __bfloat162float(__float2bfloat16_rn(v)); }
// Whether `p` may be read or written four elements at a time.
template <class T> inline bool aligned4(const T* p) { return reinterpret_cast<uintptr_t>(p) % (4 * sizeof(T)) == 0; }

// The activation operands of one launch share one storage type: true when all are bf16.
inline bool all_half(std::initializer_list<bool> halves, const char* kernel) {
    bool any = false, all = true;
    for (bool h : halves) {
        any = any || h;
        all = all && h;
    }
    if (any && !all) throw std::invalid_argument(std::string(kernel) + ": f32 and bf16 activation operands in one launch");
    return all;
}

// ---- GELU, the tanh form evaluated as x / (1 + exp(-2u)) -------------------------------------
// The operation order is the reference's (crates/modelspec-runtime/src/cpu/interpreter.rs:
// 1553-1587); the constants are the nearest f32 to sqrt(2/pi) and 0.044715.
__device__ __forceinline__ float gelu_twice_inner(float x) {
    const float scale = 0.7978845608028654f, cubic = 0.044715f;
    return 2.0f * scale * (x + cubic * x * x * x);
}
__device__ __forceinline__ float logistic(float v) { return 1.0f / (1.0f + expf(0.0f - v)); }
__device__ __forceinline__ float gelu_value(float x) { return x * logistic(gelu_twice_inner(x)); }
__device__ __forceinline__ float gelu_grad_value(float x, float g) {
    const float scale = 0.7978845608028654f, cubic = 0.044715f;
    float v = gelu_twice_inner(x);
    float s = logistic(v), r = logistic(0.0f - v);
    float slope = scale * (1.0f + 3.0f * cubic * x * x);
    return (s + 2.0f * (s * x) * r * slope) * g;
}

// The same two functions where the result is stored as bf16 (mixed-precision plans, which have no
// reference bits to keep): the hardware's base-2 exponential and reciprocal, about 2^-21 relative, far
// inside the 2^-9 of the stored value, r = 1 - s instead of a second exponential, and the polynomials as
// fused multiply-adds: with t = x^2, exp(-2u) = 2^(x (A + B t)) and the gradient's factor is
// s + s r x (C + D t). 7 and 11 instructions an element instead of some 14 and 25: in the drain of a
// product (gemm_bf16.cu) they, not the tensor cores, set the pace (16,384 x 3,072 x 768 with gelu
// 94 -> 90 us, with gelu_grad 129 -> 98).
__device__ __forceinline__ float exp2_fast(float v) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float reciprocal_fast(float v) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}
// 1 / (1 + exp(-2u)) for x and t = x^2.
__device__ __forceinline__ float gelu_logistic_fast(float x, float t) {
    constexpr double twice_scale = 2.0 * 0.7978845608028654, log2e = 1.4426950408889634;
    constexpr float A = static_cast<float>(-twice_scale * log2e), B = static_cast<float>(-twice_scale * 0.044715 * log2e);
    return reciprocal_fast(1.0f + exp2_fast(x * fmaf(B, t, A)));
}
template <class T> __device__ __forceinline__ float gelu_value_for(float x) {
    if constexpr (sizeof(T) == 2) return x * gelu_logistic_fast(x, x * x);
    else return gelu_value(x);
}
template <class T> __device__ __forceinline__ float gelu_grad_value_for(float x, float g) {
    if constexpr (sizeof(T) == 2) {
        constexpr double twice_scale = 2.0 * 0.7978845608028654;
        constexpr float C = static_cast<float>(twice_scale), D = static_cast<float>(3.0 * 0.044715 * twice_scale);
        const float t = x * x, s = gelu_logistic_fast(x, t), r = 1.0f - s;
        return fmaf(s * r, x * fmaf(D, t, C), s) * g;
    } else {
        return gelu_grad_value(x, g);
    }
}

// relu and the two gradients' shared form, as the element kernels compute them.
__device__ __forceinline__ float relu_value(float x) { return x > 0.0f ? x : 0.0f; }
__device__ __forceinline__ float relu_grad_value(float x, float g) { return x > 0.0f ? g : 0.0f; }

// ---- Philox4x32-10, word 0 of the block ------------------------------------------------------
// Counter [c0, c1, c2, c3], key [k0, k1] (Salmon et al., SC 2011); the reference draws a dropout
// decision from word 0 alone (crates/modelspec-runtime/src/train/init.rs:91-112, :160-165).
__device__ __forceinline__ uint32_t philox_word0(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3,
                                                 uint32_t k0, uint32_t k1) {
    const uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u, W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
#pragma unroll
    for (int round = 0; round < 10; ++round) {
        if (round > 0) {
            k0 += W0;
            k1 += W1;
        }
        uint32_t hi0 = __umulhi(M0, c0), lo0 = M0 * c0;
        uint32_t hi1 = __umulhi(M1, c2), lo1 = M1 * c2;
        uint32_t n0 = hi1 ^ c1 ^ k0, n2 = hi0 ^ c3 ^ k1;
        c0 = n0;
        c1 = lo1;
        c2 = n2;
        c3 = lo0;
    }
    return c0;
}

// ---- reductions ------------------------------------------------------------------------------
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sum over a block of up to 1024 threads; every thread gets the result. `shared` holds 33 T.
template <class T> __device__ __forceinline__ T block_sum(T v, T* shared) {
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = (blockDim.x + 31) >> 5;
    v = warp_sum(v);
    __syncthreads();
    if (lane == 0) shared[warp] = v;
    __syncthreads();
    if (warp == 0) {
        T t = lane < warps ? shared[lane] : T(0);
        t = warp_sum(t);
        if (lane == 0) shared[32] = t;
    }
    __syncthreads();
    return shared[32];
}
__device__ __forceinline__ float block_max(float v, float* shared) {
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = (blockDim.x + 31) >> 5;
    v = warp_max(v);
    __syncthreads();
    if (lane == 0) shared[warp] = v;
    __syncthreads();
    if (warp == 0) {
        float t = lane < warps ? shared[lane] : -INFINITY;
        t = warp_max(t);
        if (lane == 0) shared[32] = t;
    }
    __syncthreads();
    return shared[32];
}

// One-launch two-stage reductions: every block publishes its partial result, then calls this; the
// block that arrives last at `counter` (true for all its threads) sees every block's partials and
// finishes the job. The counter goes back to 0 for the next launch. Partials written by other
// blocks must be read with __ldcg (they may sit in another SM's path, never in this SM's L1).
__device__ __forceinline__ bool last_block_arrives(uint32_t* counter, uint32_t expected, bool* shared_flag) {
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0 && threadIdx.y == 0 && threadIdx.z == 0) {
        uint32_t before = atomicAdd(counter, 1u);
        bool last = before + 1u == expected;
        if (last) *counter = 0u;
        *shared_flag = last;
    }
    __syncthreads();
    bool last = *shared_flag;
    if (last) __threadfence();
    return last;
}

}  // namespace k
}  // namespace msx
