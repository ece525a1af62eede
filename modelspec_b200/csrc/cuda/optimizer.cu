// The parameter update: one launch over every parameter tensor of the step.
//
// AdamW is the reference's 16 rounded f32 operations per element, in its order
// (crates/modelspec-core/src/ir/training.rs:925-980):
//   m' = beta1 * m + (1 - beta1) * g
//   v' = beta2 * v + ((1 - beta2) * g) * g
//   p' = p - lr_t * ((m' * c1) / (sqrt(v' * c2) + eps) + weight_decay * p)
// with sqrt and the division correctly rounded and no contraction (the file is compiled with
// -fmad=false), so given the same gradient the new p, m and v are bit-identical to the CPU's.
// The reference's Vulkan path runs one dispatch per parameter
// (crates/modelspec-core/src/ir/kernel.rs:869-894); here a chunk table maps each CTA to 1,024
// or 4,096 elements of one tensor, so 41 tensors are one launch. HBM-bound for a large model (16
// bytes read and 12 written per element: 110 M elements in 455 us, 6.7 TB/s); for a small one the
// launch is one trip to memory and back, so its chunks are short (a float4 a thread): 0.1 to 0.4 M
// elements by SGD took 8.2 us with 4,096-element chunks walked element by element.
#include "common.cuh"
#include "kernels.cuh"

namespace msx {
namespace k {

namespace {

// One block's chunk of one tensor, as elements [start, stop). A whole chunk of 16-byte-aligned tensors
// is VECTORS float4 per thread at a time, every load of a turn issued before its first update; the
// last chunk of a tensor the same, its last elements one by one. An element at a time, each turn of
// a thread waits out a trip to memory: 8 us for a 4,096-element chunk, however small the model.
struct Span {
    UpdateTensor t;
    uint64_t start;
    uint32_t count;
    bool aligned;
};
__device__ __forceinline__ Span span_of(const UpdateTensor* __restrict__ tensors, const uint32_t* __restrict__ chunk_tensor,
                                        const uint32_t* __restrict__ chunk_start, uint32_t chunk) {
    Span s;
    s.start = static_cast<uint64_t>(chunk_start[blockIdx.x]) * chunk;
    s.t = tensors[chunk_tensor[blockIdx.x]];
    s.count = static_cast<uint32_t>(s.t.count - s.start < chunk ? s.t.count - s.start : chunk);
    s.aligned = ((reinterpret_cast<uintptr_t>(s.t.g) | reinterpret_cast<uintptr_t>(s.t.p) | reinterpret_cast<uintptr_t>(s.t.m) |
                  reinterpret_cast<uintptr_t>(s.t.v)) & 15) == 0;
    return s;
}

template <int VECTORS>
__global__ void __launch_bounds__(256) adamw_kernel(const UpdateTensor* tensors,
                                                     const uint32_t* chunk_tensor,
                                                     const uint32_t* chunk_start, uint32_t chunk, AdamWConstants c,
                                                     const float* lr_t, const float* c1,
                                                     const float* c2) {
    after_producers();
    const float lr = lr_t[0], k1 = c1[0], k2 = c2[0];
    const Span s = span_of(tensors, chunk_tensor, chunk_start, chunk);
    const UpdateTensor& t = s.t;
    auto update = [&](float g, float& p, float& m, float& v) {
        float m_next = c.beta1 * m + c.rest1 * g;
        float v_next = c.beta2 * v + (c.rest2 * g) * g;
        float direction = (m_next * k1) / (sqrtf(v_next * k2) + c.eps);
        float step = direction + c.weight_decay * p;
        p = p - lr * step;
        m = m_next;
        v = v_next;
    };
    auto one = [&](uint64_t i) {
        float g = t.g[i], p = t.p[i], m = t.m[i], v = t.v[i];
        update(g, p, m, v);
        t.p[i] = p;
        t.m[i] = m;
        t.v[i] = v;
        if (t.p16 != nullptr) store1(static_cast<bf16*>(t.p16) + i, p);
    };
    if (!s.aligned) {
        for (uint32_t i = threadIdx.x; i < s.count; i += 256) one(s.start + i);
        return;
    }
    const uint32_t whole = s.count / 4;
#pragma unroll 1
    for (uint32_t first = threadIdx.x; first < whole; first += 256 * VECTORS) {
        float4 g[VECTORS], p[VECTORS], m[VECTORS], v[VECTORS];
#pragma unroll
        for (int j = 0; j < VECTORS; ++j) {
            if (first + j * 256 >= whole) break;
            const uint64_t i = s.start + (first + j * 256) * 4;
            g[j] = *reinterpret_cast<const float4*>(t.g + i);
            p[j] = *reinterpret_cast<const float4*>(t.p + i);
            m[j] = *reinterpret_cast<const float4*>(t.m + i);
            v[j] = *reinterpret_cast<const float4*>(t.v + i);
        }
#pragma unroll
        for (int j = 0; j < VECTORS; ++j) {
            if (first + j * 256 >= whole) break;
            const uint64_t i = s.start + (first + j * 256) * 4;
            update(g[j].x, p[j].x, m[j].x, v[j].x);
            update(g[j].y, p[j].y, m[j].y, v[j].y);
            update(g[j].z, p[j].z, m[j].z, v[j].z);
            update(g[j].w, p[j].w, m[j].w, v[j].w);
            *reinterpret_cast<float4*>(t.p + i) = p[j];
            *reinterpret_cast<float4*>(t.m + i) = m[j];
            *reinterpret_cast<float4*>(t.v + i) = v[j];
            // The bf16 working copy the next step's matmuls read (mixed-precision plans).
            if (t.p16 != nullptr) store4(static_cast<bf16*>(t.p16) + i, p[j]);
        }
    }
    if (threadIdx.x < s.count % 4) one(s.start + whole * 4 + threadIdx.x);
}

// The bf16 working copy of a parameter from its f32 master (after an upload).
__global__ void working_copy_kernel(const float* p, bf16* p16, uint64_t n) {
    after_producers();
    const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) store1(p16 + i, p[i]);
}

template <int VECTORS>
__global__ void __launch_bounds__(256) sgd_kernel(const UpdateTensor* tensors,
                                                   const uint32_t* chunk_tensor,
                                                   const uint32_t* chunk_start, uint32_t chunk,
                                                   const float* lr) {
    after_producers();
    const float rate = lr[0];
    const Span s = span_of(tensors, chunk_tensor, chunk_start, chunk);
    const UpdateTensor& t = s.t;
    auto one = [&](uint64_t i) {
        const float p = t.p[i] - rate * t.g[i];
        t.p[i] = p;
        if (t.p16 != nullptr) store1(static_cast<bf16*>(t.p16) + i, p);
    };
    if (!s.aligned) {
        for (uint32_t i = threadIdx.x; i < s.count; i += 256) one(s.start + i);
        return;
    }
    const uint32_t whole = s.count / 4;
#pragma unroll 1
    for (uint32_t first = threadIdx.x; first < whole; first += 256 * VECTORS) {
        float4 g[VECTORS], p[VECTORS];
#pragma unroll
        for (int j = 0; j < VECTORS; ++j) {
            if (first + j * 256 >= whole) break;
            const uint64_t i = s.start + (first + j * 256) * 4;
            g[j] = *reinterpret_cast<const float4*>(t.g + i);
            p[j] = *reinterpret_cast<const float4*>(t.p + i);
        }
#pragma unroll
        for (int j = 0; j < VECTORS; ++j) {
            if (first + j * 256 >= whole) break;
            const uint64_t i = s.start + (first + j * 256) * 4;
            p[j].x = p[j].x - rate * g[j].x;
            p[j].y = p[j].y - rate * g[j].y;
            p[j].z = p[j].z - rate * g[j].z;
            p[j].w = p[j].w - rate * g[j].w;
            *reinterpret_cast<float4*>(t.p + i) = p[j];
            if (t.p16 != nullptr) store4(static_cast<bf16*>(t.p16) + i, p[j]);
        }
    }
    if (threadIdx.x < s.count % 4) one(s.start + whole * 4 + threadIdx.x);
}

}  // namespace

void adamw(cudaStream_t s, const UpdateTensor* d_tensors, const uint32_t* d_chunk_tensor,
           const uint32_t* d_chunk_start, uint32_t chunks, uint32_t chunk, AdamWConstants c, const float* lr_t,
           const float* c1, const float* c2) {
    if (chunks == 0) return;
    if (chunk == kSmallUpdateChunk) adamw_kernel<1><<<chunks, 256, 0, s>>>(d_tensors, d_chunk_tensor, d_chunk_start, chunk, c, lr_t, c1, c2);
    else adamw_kernel<2><<<chunks, 256, 0, s>>>(d_tensors, d_chunk_tensor, d_chunk_start, chunk, c, lr_t, c1, c2);
    check_launch("adamw");
}

void working_copy(cudaStream_t s, const float* p, void* p16, uint64_t n) {
    if (n == 0) return;
    const uint64_t blocks = (n + 255) / 256;
    working_copy_kernel<<<static_cast<uint32_t>(blocks > 148 * 8 ? 148 * 8 : blocks), 256, 0, s>>>(p, static_cast<bf16*>(p16), n);
    check_launch("working_copy");
}

void sgd(cudaStream_t s, const UpdateTensor* d_tensors, const uint32_t* d_chunk_tensor,
         const uint32_t* d_chunk_start, uint32_t chunks, uint32_t chunk, const float* lr) {
    if (chunks == 0) return;
    if (chunk == kSmallUpdateChunk) sgd_kernel<1><<<chunks, 256, 0, s>>>(d_tensors, d_chunk_tensor, d_chunk_start, chunk, lr);
    else sgd_kernel<4><<<chunks, 256, 0, s>>>(d_tensors, d_chunk_tensor, d_chunk_start, chunk, lr);
    check_launch("sgd");
}

}  // namespace k
}  // namespace msx
