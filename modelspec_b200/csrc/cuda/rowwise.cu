// Row kernels: layer_norm and its two gradients, softmax and its gradient, cross_entropy and its
// gradient. One warp per row for hidden-size rows, one block per row for vocabulary-size rows;
// row reductions are warp-shuffle trees, so sums round in another order than the reference's
// ascending-column loops (crates/modelspec-runtime/src/cpu/interpreter.rs:970-1034, :1172-1233,
// :1513-1527): tolerance class, deterministic. The per-element formulas keep the reference's
// operation order. All are HBM-bound; a row is read from L1/L2 on its second and third pass.
#include "common.cuh"
#include "kernels.cuh"

namespace msx {
namespace k {

uint32_t sum_rows_chunks(uint64_t rows);

namespace {

#ifndef MSX_LN_BACKWARD_WIDE_BLOCKS
#define MSX_LN_BACKWARD_WIDE_BLOCKS 296
#endif
#ifndef MSX_LN_BACKWARD_BLOCKS
#define MSX_LN_BACKWARD_BLOCKS 592
#endif
constexpr float kLayerNormEps = 1e-12f;
constexpr int kWarpsPerBlock = 8;

__device__ __forceinline__ void row_moments(const float* __restrict__ row, uint32_t h, int lane,
                                            float* mean, float* rstd) {
    float s = 0.0f;
    for (uint32_t j = lane; j < h; j += 32) s += row[j];
    float m = warp_sum(s) / static_cast<float>(h);
    float q = 0.0f;
    for (uint32_t j = lane; j < h; j += 32) {
        float d = row[j] - m;
        q = fmaf(d, d, q);
    }
    float variance = warp_sum(q) / static_cast<float>(h);
    *mean = m;
    *rstd = 1.0f / sqrtf(variance + kLayerNormEps);
}

__global__ void layer_norm_kernel(const float* x, const float* gamma,
                                  const float* beta, float* out, uint32_t rows,
                                  uint32_t h) {
    after_producers();
    int lane = threadIdx.x & 31;
    uint32_t r = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
    if (r >= rows) return;
    const float* row = x + static_cast<uint64_t>(r) * h;
    float mean, rstd;
    row_moments(row, h, lane, &mean, &rstd);
    float* o = out + static_cast<uint64_t>(r) * h;
    const Settled<float> values = settled(row), by = settled(gamma), plus = settled(beta);
#pragma unroll 4
    for (uint32_t j = lane; j < h; j += 32) o[j] = (load1(values + j) - mean) * rstd * load1(by + j) + load1(plus + j);
}

__global__ void layer_norm_grad_x_kernel(const float* x, const float* gamma,
                                         const float* g, float* out, uint32_t rows,
                                         uint32_t h) {
    after_producers();
    int lane = threadIdx.x & 31;
    uint32_t r = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
    if (r >= rows) return;
    const float* row = x + static_cast<uint64_t>(r) * h;
    const float* grow = g + static_cast<uint64_t>(r) * h;
    float mean, rstd;
    row_moments(row, h, lane, &mean, &rstd);
    float s1 = 0.0f, s2 = 0.0f;
    for (uint32_t j = lane; j < h; j += 32) {
        float gx = grow[j] * gamma[j];
        float xhat = (row[j] - mean) * rstd;
        s1 += gx;
        s2 = fmaf(gx, xhat, s2);
    }
    float width = static_cast<float>(h);
    float mean_gx = warp_sum(s1) / width, mean_gx_xhat = warp_sum(s2) / width;
    float* o = out + static_cast<uint64_t>(r) * h;
    for (uint32_t j = lane; j < h; j += 32) {
        float gx = grow[j] * gamma[j];
        float xhat = (row[j] - mean) * rstd;
        o[j] = rstd * ((gx - mean_gx) - xhat * mean_gx_xhat);
    }
}

__global__ void row_stats_kernel(const float* x, float* stats, uint32_t rows,
                                 uint32_t h) {
    after_producers();
    int lane = threadIdx.x & 31;
    uint32_t r = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
    if (r >= rows) return;
    float mean, rstd;
    row_moments(x + static_cast<uint64_t>(r) * h, h, lane, &mean, &rstd);
    if (lane == 0) {
        stats[2 * r] = mean;
        stats[2 * r + 1] = rstd;
    }
}

// Block (32, 8) over a 32-column tile and a chunk of rows: partial column sums of g * xhat and,
// when wanted, of g.
__global__ void grad_gamma_stage1(const float* x, const float* g,
                                  const float* stats, uint32_t rows, uint32_t h,
                                  uint32_t rows_per_chunk, float* partial_gamma,
                                  float* partial_beta) {
    after_producers();
    __shared__ float sg[8][32], sb[8][32];
    uint32_t c = blockIdx.x * 32 + threadIdx.x;
    uint32_t r0 = blockIdx.y * rows_per_chunk, r1 = min(rows, r0 + rows_per_chunk);
    float acc_g = 0.0f, acc_b = 0.0f;
    if (c < h)
        for (uint32_t r = r0 + threadIdx.y; r < r1; r += 8) {
            float gv = g[static_cast<uint64_t>(r) * h + c];
            float xhat = (x[static_cast<uint64_t>(r) * h + c] - stats[2 * r]) * stats[2 * r + 1];
            acc_g = fmaf(gv, xhat, acc_g);
            acc_b += gv;
        }
    sg[threadIdx.y][threadIdx.x] = acc_g;
    sb[threadIdx.y][threadIdx.x] = acc_b;
    __syncthreads();
    if (threadIdx.y == 0 && c < h) {
        float tg = sg[0][threadIdx.x], tb = sb[0][threadIdx.x];
#pragma unroll
        for (int w = 1; w < 8; ++w) {
            tg += sg[w][threadIdx.x];
            tb += sb[w][threadIdx.x];
        }
        partial_gamma[static_cast<uint64_t>(blockIdx.y) * h + c] = tg;
        if (partial_beta) partial_beta[static_cast<uint64_t>(blockIdx.y) * h + c] = tb;
    }
}

__global__ void grad_gamma_stage2(const float* partial_gamma, const float* partial_beta,
                                  uint32_t chunks, uint32_t h, float* dgamma,
                                  float* dbeta) {
    after_producers();
    uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= h) return;
    float tg = partial_gamma[c];
    for (uint32_t k = 1; k < chunks; ++k) tg += partial_gamma[static_cast<uint64_t>(k) * h + c];
    dgamma[c] = tg;
    if (dbeta) {
        float tb = partial_beta[c];
        for (uint32_t k = 1; k < chunks; ++k) tb += partial_beta[static_cast<uint64_t>(k) * h + c];
        dbeta[c] = tb;
    }
}

constexpr int kRowThreads = 256;

// Max of the row (the first element, replaced only by a greater one: NaN never wins) and the sum
// of exp(x - max), by a block.
template <class T>
__device__ __forceinline__ void block_row_softmax(const T* __restrict__ row, uint32_t v, float* shared,
                                                  float* max, float* total) {
    float m = -INFINITY;
    for (uint32_t c = threadIdx.x; c < v; c += blockDim.x) {
        float x = load1(row + c);
        if (x > m) m = x;
    }
    m = block_max(m, shared);
    float s = 0.0f;
    for (uint32_t c = threadIdx.x; c < v; c += blockDim.x) s += expf(load1(row + c) - m);
    *max = m;
    *total = block_sum(s, shared);
}

__global__ void softmax_kernel(const float* x, float* out, uint32_t k) {
    after_producers();
    __shared__ float shared[33];
    const float* row = x + static_cast<uint64_t>(blockIdx.x) * k;
    float max, total;
    block_row_softmax(row, k, shared, &max, &total);
    float* o = out + static_cast<uint64_t>(blockIdx.x) * k;
    for (uint32_t c = threadIdx.x; c < k; c += blockDim.x) o[c] = expf(row[c] - max) / total;
}

__global__ void softmax_grad_kernel(const float* y, const float* g,
                                    float* out, uint32_t k) {
    after_producers();
    __shared__ float shared[33];
    const float* yr = y + static_cast<uint64_t>(blockIdx.x) * k;
    const float* gr = g + static_cast<uint64_t>(blockIdx.x) * k;
    float acc = 0.0f;
    for (uint32_t c = threadIdx.x; c < k; c += blockDim.x) acc = fmaf(gr[c], yr[c], acc);
    float d = block_sum(acc, shared);
    float* o = out + static_cast<uint64_t>(blockIdx.x) * k;
    for (uint32_t c = threadIdx.x; c < k; c += blockDim.x) o[c] = yr[c] * (gr[c] - d);
}

template <class T>
__global__ void cross_entropy_rows_kernel(const T* logits, const int32_t* labels,
                                          const float* weights, float* row_loss,
                                          uint32_t v, uint32_t ld) {
    after_producers();
    __shared__ float shared[33];
    uint32_t r = blockIdx.x;
    // A row of weight 0 adds w * l = 0 to the loss whatever its logits: skip its passes.
    if (weights[r] == 0.0f) {
        if (threadIdx.x == 0) row_loss[r] = 0.0f;
        return;
    }
    const T* row = logits + static_cast<uint64_t>(r) * ld;
    float max, total;
    block_row_softmax(row, v, shared, &max, &total);
    if (threadIdx.x == 0) {
        int32_t label = labels[r];
        float picked = (label >= 0 && static_cast<uint32_t>(label) < v) ? load1(row + label) : 0.0f;
        row_loss[r] = max + logf(total) - picked;
    }
}

// loss = sum_n w[n] l[n] / sum_n w[n], both sums in f64 (a tree over the block), one rounding.
__global__ void cross_entropy_loss_kernel(const float* row_loss, const float* weights,
                                          uint32_t rows, const float* global_den, float* loss) {
    after_producers();
    __shared__ double shared[33];
    double num = 0.0, den = 0.0;
    for (uint32_t r = threadIdx.x; r < rows; r += blockDim.x) {
        double w = static_cast<double>(weights[r]);
        num = fma(w, static_cast<double>(row_loss[r]), num);
        den += w;
    }
    num = block_sum(num, shared);
    den = block_sum(den, shared);
    // Data parallel: the numerator of this shard over the weight sum of the whole batch.
    if (global_den) den = static_cast<double>(global_den[0]);
    if (threadIdx.x == 0) loss[0] = den == 0.0 ? 0.0f : static_cast<float>(num / den);
}

__global__ void weight_sum_kernel(const float* weights, uint32_t rows, float* out) {
    after_producers();
    __shared__ double shared[33];
    double den = 0.0;
    for (uint32_t r = threadIdx.x; r < rows; r += blockDim.x) den += static_cast<double>(weights[r]);
    den = block_sum(den, shared);
    if (threadIdx.x == 0) out[0] = static_cast<float>(den);
}

__global__ void cross_entropy_grad_kernel(const float* logits, const int32_t* labels,
                                          const float* weights, const float* g,
                                          const float* denominator, float* out,
                                          uint32_t v, uint32_t ld, uint32_t ld_out) {
    after_producers();
    __shared__ float shared[33];
    uint32_t r = blockIdx.x;
    float* o = out + static_cast<uint64_t>(r) * ld_out;
    float den = denominator[0], w = weights[r];
    if (den == 0.0f || w == 0.0f) {
        for (uint32_t c = threadIdx.x; c < v; c += blockDim.x) o[c] = 0.0f;
        return;
    }
    const float* row = logits + static_cast<uint64_t>(r) * ld;
    float max, total;
    block_row_softmax(row, v, shared, &max, &total);
    float scale = g[0] * w / den;
    uint32_t label = static_cast<uint32_t>(labels[r]);
    for (uint32_t c = threadIdx.x; c < v; c += blockDim.x) {
        float target = c == label ? 1.0f : 0.0f;
        o[c] = scale * (expf(row[c] - max) / total - target);
    }
}

// Loss row and gradient row in one visit of the logits row: max, sum of exp, then
// scale * (p - onehot) while the row is still in cache. The same formulas, in the same order, as
// the two separate kernels.
template <class T>
__global__ void cross_entropy_fused_kernel(const T* logits, const int32_t* labels,
                                           const float* weights, const float* g,
                                           const float* denominator, float* row_loss,
                                           T* out, uint32_t v, uint32_t ld, uint32_t ld_out) {
    after_producers();
    __shared__ float shared[33];
    uint32_t r = blockIdx.x;
    T* o = out + static_cast<uint64_t>(r) * ld_out;
    float den = denominator[0], w = weights[r];
    if (w == 0.0f) {
        if (threadIdx.x == 0) row_loss[r] = 0.0f;
        for (uint32_t c = threadIdx.x; c < v; c += blockDim.x) store1(o + c, 0.0f);
        return;
    }
    const T* row = logits + static_cast<uint64_t>(r) * ld;
    float max, total;
    block_row_softmax(row, v, shared, &max, &total);
    uint32_t label = static_cast<uint32_t>(labels[r]);
    if (threadIdx.x == 0) row_loss[r] = max + logf(total) - (label < v ? load1(row + label) : 0.0f);
    if (den == 0.0f) {
        for (uint32_t c = threadIdx.x; c < v; c += blockDim.x) store1(o + c, 0.0f);
        return;
    }
    float scale = g[0] * w / den;
    for (uint32_t c = threadIdx.x; c < v; c += blockDim.x) {
        float target = c == label ? 1.0f : 0.0f;
        store1(o + c, scale * (expf(load1(row + c) - max) / total - target));
    }
}

// The same, for rows of up to 32 * 1024 logits, with the row held in registers: one read of the
// logits from memory (every load of the row in flight at once), one write of the gradient, and
// each exp computed once, by the hardware exponential (relative error about 2^-21, far inside the
// tolerance class every exp-based kernel is in), with one reciprocal of the row sum instead of a
// division per element: 30,522 exps and divisions per row are otherwise as long as the row's
// memory traffic.
// For rows that no 16-byte access can be made on; every other row takes one of the kernels below.
constexpr int kWideThreads = 1024, kWideItems = 32;
template <class T>
__global__ void __launch_bounds__(kWideThreads, 1)
cross_entropy_fused_wide_kernel(const T* logits, const int32_t* labels,
                                const float* weights, const float* g,
                                const float* denominator, float* row_loss,
                                T* out, uint32_t v, uint32_t ld, uint32_t ld_out,
                                uint32_t* counter, float* loss) {
    after_producers();
    // Element i of this thread is column column_of(i): consecutive threads take consecutive columns.
    auto column_of = [](int i, uint32_t tid) { return static_cast<uint32_t>(i) * kWideThreads + tid; };
    __shared__ float shared[33];
    __shared__ double shared64[33];
    __shared__ bool is_last;
    const uint32_t r = blockIdx.x, tid = threadIdx.x, rows = gridDim.x;
    T* o = out + static_cast<uint64_t>(r) * ld_out;
    // The weight sum: given (the whole batch's, data parallel), or summed here by every block in
    // the same order (f64 over the block, one rounding), so that no launch has to precede this one.
    float den;
    if (denominator != nullptr) {
        den = denominator[0];
    } else {
        double sum = 0.0;
        for (uint32_t j = tid; j < rows; j += kWideThreads) sum += static_cast<double>(weights[j]);
        den = static_cast<float>(block_sum(sum, shared64));
    }
    const float w = weights[r];
    float x[kWideItems];
    float total = 0.0f;
    uint32_t label = 0;
    if (w == 0.0f) {
        if (tid == 0) row_loss[r] = 0.0f;
    } else {
        const T* row = logits + static_cast<uint64_t>(r) * ld;
        // Unconditional loads from a clamped column, so that all are in flight together; what lies past v
        // is replaced afterwards.
#pragma unroll
        for (int i = 0; i < kWideItems; ++i) x[i] = load1(row + min(column_of(i, tid), v - 1));
#pragma unroll
        for (int i = 0; i < kWideItems; ++i)
            if (column_of(i, tid) >= v) x[i] = -INFINITY;
        float m = -INFINITY;
#pragma unroll
        for (int i = 0; i < kWideItems; ++i)
            if (x[i] > m) m = x[i];
        m = block_max(m, shared);
        float sum = 0.0f;
#pragma unroll
        for (int i = 0; i < kWideItems; ++i) {
            const uint32_t c = column_of(i, tid);
            if (c < v) {
                x[i] = __expf(x[i] - m);
                sum += x[i];
            }
        }
        total = block_sum(sum, shared);
        label = static_cast<uint32_t>(labels[r]);
        if (tid == 0) row_loss[r] = m + logf(total) - (label < v ? load1(row + label) : 0.0f);
    }
    // The loss, by the last block to get here: sum of w * l over sum of w, f64 sums, one rounding.
    // Only thread 0's row loss has to be visible to that block, so only thread 0 fences, and the
    // gradient stores below are not waited for: they drain while the SM's next block loads.
    if (tid == 0) {
        __threadfence();
        const uint32_t before = atomicAdd(counter, 1u);
        is_last = before + 1u == rows;
        if (is_last) *counter = 0u;
    }
    __syncthreads();
    if (is_last) {
        __threadfence();
        double num = 0.0, den64 = 0.0;
        for (uint32_t j = tid; j < rows; j += kWideThreads) {
            double wj = static_cast<double>(weights[j]);
            num = fma(wj, static_cast<double>(__ldcg(row_loss + j)), num);
            den64 += wj;
        }
        num = block_sum(num, shared64);
        den64 = block_sum(den64, shared64);
        if (denominator != nullptr) den64 = static_cast<double>(denominator[0]);
        if (tid == 0) loss[0] = den64 == 0.0 ? 0.0f : static_cast<float>(num / den64);
    }
    const bool zero = den == 0.0f || w == 0.0f;
    const float scale = zero ? 0.0f : g[0] * w / den;
    const float inverse = zero ? 0.0f : 1.0f / total;
#pragma unroll
    for (int i = 0; i < kWideItems; ++i) {
        const uint32_t c = column_of(i, tid);
        const float target = c == label ? 1.0f : 0.0f;
        x[i] = zero ? 0.0f : scale * (x[i] * inverse - target);
    }
#pragma unroll
    for (int i = 0; i < kWideItems; ++i) {
        const uint32_t c = column_of(i, tid);
        if (c < v) store1(o + c, x[i]);
    }
}

inline uint32_t warp_row_blocks(uint64_t rows) { return static_cast<uint32_t>((rows + kWarpsPerBlock - 1) / kWarpsPerBlock); }

// A row's 16-byte pieces as a thread holds them: f32 values in place, bf16 ones packed as they were read.
__device__ __forceinline__ float4 as_floats(const uint4& v) {
    return make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w));
}
__device__ __forceinline__ float bf16_low(uint32_t pair) { return __uint_as_float(pair << 16); }
__device__ __forceinline__ float bf16_high(uint32_t pair) { return __uint_as_float(pair & 0xffff0000u); }

// The same for rows on 16-byte boundaries: THREADS threads hold a row in GROUPS pieces of 16 bytes each, ROWS
// such rows a block (more than one only as a warp a row, which then needs no barrier for its row).
//
// Bound for long rows by their one read and one write, for short ones by the chain of dependent steps of a
// row. So one barrier serves the row's maximum and the weight sum, one the row's sum, each warp adds the
// warps' shares up for itself, and the atomic that finds the last block is not waited for before the
// gradient is written. bf16 pieces stay packed (half the registers: two blocks of 512 threads an SM hold
// rows of 32,768, so that one block's loads and stores run under the other's reductions), and their
// exponentials are taken twice rather than kept as f32.
// A launch (with what launching costs): 64 x 10 f32 12.6 -> 6.5 us, 96 x 1,009 f32 12.6 -> 6.5, 384 x 5,003 bf16
// 24.9 -> 10.6, 832 x 30,522 bf16 47.6 -> 32.4, 2,880 x 30,522 bf16 177 -> 107 (a 1,024-thread block a row before).
template <int THREADS, int ROWS, int GROUPS, int BLOCKS, class T>
__global__ void __launch_bounds__(THREADS * ROWS, BLOCKS)
cross_entropy_row_kernel(const T* logits, const int32_t* labels, const float* weights,
                         const float* g, const float* denominator, float* row_loss,
                         T* out, uint32_t rows, uint32_t v, uint32_t ld, uint32_t ld_out, uint32_t* counter,
                         float* loss) {
    after_producers();
    static_assert(ROWS == 1 || THREADS == 32);
    constexpr bool HALF = sizeof(T) == 2;
    constexpr uint32_t E = 16 / sizeof(T), ALL = THREADS * ROWS, WARPS = ALL / 32;
    __shared__ float shared_max[WARPS], shared_sum[WARPS];
    __shared__ double shared_weight[WARPS];
    __shared__ bool is_last;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, t = ROWS > 1 ? lane : tid;
    const uint32_t r = blockIdx.x * ROWS + (ROWS > 1 ? warp : 0);
    auto column_of = [t](int k) { return (static_cast<uint32_t>(k) * THREADS + t) * E; };
    const bool here = r < rows;
    const float w = here ? weights[r] : 0.0f;
    const uint32_t label = here ? static_cast<uint32_t>(labels[r]) : 0u;
    const T* row = logits + static_cast<uint64_t>(r) * ld;
    // Unconditional loads from a clamped column (the pitch covers the whole piece of the last valid column), so
    // that all are in flight together. A row of weight 0 is not read.
    uint4 x[GROUPS];
    float picked = 0.0f;
    if (w != 0.0f) {
        const uint32_t last = (v - 1) / E * E;
#pragma unroll
        for (int k = 0; k < GROUPS; ++k) x[k] = load_global(reinterpret_cast<const uint4*>(row + min(column_of(k), last)));
        if (t == 0 && label < v) picked = load1(row + label);
    }
    // The weight sum: given (the whole batch's, data parallel), or summed here by every block in the same
    // order (f64, one rounding), so that no launch has to precede this one.
    double weight = 0.0;
    if (denominator == nullptr)
        for (uint32_t j = tid; j < rows; j += ALL) weight += static_cast<double>(weights[j]);
    float m = -INFINITY;
    if (w != 0.0f) {
        if constexpr (HALF) {
            const uint32_t none = 0xff80ff80u;  // a pair of -inf
            __nv_bfloat162 best = *reinterpret_cast<const __nv_bfloat162*>(&none);
#pragma unroll
            for (int k = 0; k < GROUPS; ++k) {
                uint32_t* pair = &x[k].x;
                const uint32_t c = column_of(k);
                if (c + E > v) {
#pragma unroll
                    for (uint32_t i = 0; i < 4; ++i) {
                        if (c + 2 * i >= v) pair[i] = none;
                        else if (c + 2 * i + 1 >= v) pair[i] = (pair[i] & 0xffffu) | (none & 0xffff0000u);
                    }
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) best = __hmax2(best, *reinterpret_cast<const __nv_bfloat162*>(&pair[i]));
            }
            const uint32_t both = *reinterpret_cast<const uint32_t*>(&best);
            m = fmaxf(bf16_low(both), bf16_high(both));
        } else {
#pragma unroll
            for (int k = 0; k < GROUPS; ++k) {
                uint32_t* one = &x[k].x;
#pragma unroll
                for (uint32_t i = 0; i < 4; ++i) {
                    if (column_of(k) + i >= v) one[i] = 0xff800000u;
                    m = fmaxf(m, __uint_as_float(one[i]));
                }
            }
        }
        m = warp_max(m);
    }
    weight = warp_sum(weight);
    if (lane == 0) {
        shared_weight[warp] = weight;
        if (ROWS == 1) shared_max[warp] = m;
    }
    __syncthreads();
    if (ROWS == 1) m = warp_max(lane < WARPS ? shared_max[lane] : -INFINITY);
    float total = 0.0f;
    if (w != 0.0f) {
        // exp(-inf) is 0: the columns past the row's end add nothing.
#pragma unroll
        for (int k = 0; k < GROUPS; ++k) {
            if constexpr (HALF) {
                const uint32_t* pair = &x[k].x;
                float part = 0.0f;
#pragma unroll
                for (int i = 0; i < 4; ++i) part += __expf(bf16_low(pair[i]) - m) + __expf(bf16_high(pair[i]) - m);
                total += part;
            } else {
                const float4 f = as_floats(x[k]);
                const float4 e = make_float4(__expf(f.x - m), __expf(f.y - m), __expf(f.z - m), __expf(f.w - m));
                total += (e.x + e.y) + (e.z + e.w);
                x[k] = make_uint4(__float_as_uint(e.x), __float_as_uint(e.y), __float_as_uint(e.z), __float_as_uint(e.w));
            }
        }
        total = warp_sum(total);
    }
    if (ROWS == 1 && WARPS > 1) {
        if (lane == 0) shared_sum[warp] = total;
        __syncthreads();
        total = warp_sum(lane < WARPS ? shared_sum[lane] : 0.0f);
    }
    weight = denominator != nullptr ? static_cast<double>(denominator[0]) : warp_sum(lane < WARPS ? shared_weight[lane] : 0.0);
    const float den = static_cast<float>(weight);
    if (t == 0 && here) row_loss[r] = w == 0.0f ? 0.0f : m + logf(total) - picked;
    // Which block finishes the loss: only the row losses have to be visible to it, so only their writers
    // fence, and the answer is not needed before the gradient's stores are on their way.
    uint32_t before = 0;
    if (ROWS > 1) {
        if (lane == 0) __threadfence();
        __syncthreads();
    } else if (tid == 0) {
        __threadfence();
    }
    if (tid == 0) before = atomicAdd(counter, 1u);
    const bool zero = den == 0.0f || w == 0.0f;
    const float scale = zero ? 0.0f : g[0] * w / den, inverse = zero ? 0.0f : 1.0f / total, both = scale * inverse;
    T* o = out + static_cast<uint64_t>(r) * ld_out;
#pragma unroll
    for (int k = 0; k < GROUPS; ++k) {
        const uint32_t c = column_of(k);
        float e[E];
#pragma unroll
        for (uint32_t i = 0; i < E; ++i) {
            const uint32_t bits = (&x[k].x)[HALF ? i / 2 : i];
            e[i] = !HALF ? __uint_as_float(bits) : __expf((i % 2 ? bf16_high(bits) : bf16_low(bits)) - m);
        }
        // scale (p - 1) at the label, scale p elsewhere.
        const bool has_label = label - c < E;
        const uint32_t at = label - c;
#pragma unroll
        for (uint32_t i = 0; i < E; ++i) {
            if (has_label && i == at) e[i] = zero ? 0.0f : scale * (e[i] * inverse - 1.0f);
            else e[i] = zero ? 0.0f : e[i] * both;
        }
        if (here && c < v) {
            // Columns past v inside the pitch are padding nobody reads: the whole piece is written.
            if constexpr (HALF) store8(reinterpret_cast<bf16*>(o) + c, {make_float4(e[0], e[1], e[2], e[3]), make_float4(e[4], e[5], e[6], e[7])});
            else store4(o + c, make_float4(e[0], e[1], e[2], e[3]));
        }
    }
    if (tid == 0) {
        is_last = before + 1u == gridDim.x;
        if (is_last) *counter = 0u;
    }
    __syncthreads();
    if (!is_last) return;
    // The loss: sum of w * l over sum of w, f64 sums, one rounding.
    __threadfence();
    double num = 0.0;
    for (uint32_t j = tid; j < rows; j += ALL) num = fma(static_cast<double>(weights[j]), static_cast<double>(__ldcg(row_loss + j)), num);
    num = warp_sum(num);
    if (lane == 0) shared_weight[warp] = num;
    __syncthreads();
    num = warp_sum(lane < WARPS ? shared_weight[lane] : 0.0);
    if (tid == 0) loss[0] = weight == 0.0 ? 0.0f : static_cast<float>(num / weight);
}

// The same for f32 rows of more than 16,384 logits, as two blocks per SM: 512 threads hold 32 elements each in
// registers and up to 32 more in shared memory (64 KB a block), so that one block's loads and
// stores run under the other's reductions and exponentials. Rows of more than 32,768 take 1,024 threads. Elements bound for shared memory go
// there straight from global memory (cp.async, 16 bytes), all in flight with the register loads;
// every thread reads back only what it copied itself.
constexpr int kSplitRegisterItems = 32, kSplitSharedItems = 32;
template <int kSplitThreads>
__global__ void __launch_bounds__(kSplitThreads, 1024 / kSplitThreads)
cross_entropy_fused_split_kernel(const float* logits, const int32_t* labels,
                                 const float* weights, const float* g,
                                 const float* denominator, float* row_loss,
                                 float* out, uint32_t v, uint32_t ld, uint32_t ld_out,
                                 uint32_t* counter, float* loss) {
    after_producers();
    // Group k of this thread is the four columns from (k * threads + tid) * 4 on: groups 0..7 live in
    // registers, groups 8..15 in shared memory.
    extern __shared__ float4 parked[];  // [kSplitSharedItems / 4][kSplitThreads]
    __shared__ float shared[33];
    __shared__ double shared64[33];
    __shared__ bool is_last;
    constexpr int kRegisterGroups = kSplitRegisterItems / 4, kSharedGroups = kSplitSharedItems / 4;
    const uint32_t r = blockIdx.x, tid = threadIdx.x, rows = gridDim.x;
    auto column_of = [tid](int group) { return (static_cast<uint32_t>(group) * kSplitThreads + tid) * 4; };
    float* o = out + static_cast<uint64_t>(r) * ld_out;
    float den;
    if (denominator != nullptr) {
        den = denominator[0];
    } else {
        double sum = 0.0;
        for (uint32_t j = tid; j < rows; j += kSplitThreads) sum += static_cast<double>(weights[j]);
        den = static_cast<float>(block_sum(sum, shared64));
    }
    const float w = weights[r];
    float4 x[kRegisterGroups];
    float total = 0.0f;
    uint32_t label = 0;
    // How many of the parked groups hold columns of the row at all (the same for every thread of
    // a warp but the one the row ends in, whose later lanes have one fewer).
    int parked_groups = 0;
#pragma unroll
    for (int k = 0; k < kSharedGroups; ++k)
        if (column_of(kRegisterGroups + k) < v) parked_groups = k + 1;
    if (w == 0.0f) {
        if (tid == 0) row_loss[r] = 0.0f;
    } else {
        const float* row = logits + static_cast<uint64_t>(r) * ld;
        const uint32_t last = (v - 1) & ~3u;
#pragma unroll
        for (int k = 0; k < kSharedGroups; ++k)
            if (k < parked_groups) {
                const uint32_t to = static_cast<uint32_t>(__cvta_generic_to_shared(&parked[k * kSplitThreads + tid]));
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(row + column_of(kRegisterGroups + k)) : "memory");
            }
        asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll
        for (int k = 0; k < kRegisterGroups; ++k) x[k] = load_global(reinterpret_cast<const float4*>(row + min(column_of(k), last)));
        auto mask = [v](float4 f, uint32_t c) {
            if (c >= v) f.x = -INFINITY;
            if (c + 1 >= v) f.y = -INFINITY;
            if (c + 2 >= v) f.z = -INFINITY;
            if (c + 3 >= v) f.w = -INFINITY;
            return f;
        };
        float m = -INFINITY;
#pragma unroll
        for (int k = 0; k < kRegisterGroups; ++k) {
            x[k] = mask(x[k], column_of(k));
            m = fmaxf(fmaxf(m, fmaxf(x[k].x, x[k].y)), fmaxf(x[k].z, x[k].w));
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
        for (int k = 0; k < kSharedGroups; ++k)
            if (k < parked_groups) {
                const float4 f = mask(parked[k * kSplitThreads + tid], column_of(kRegisterGroups + k));
                parked[k * kSplitThreads + tid] = f;
                m = fmaxf(fmaxf(m, fmaxf(f.x, f.y)), fmaxf(f.z, f.w));
            }
        m = block_max(m, shared);
        // exp(-inf) is 0: the masked columns add nothing and need no test of their own.
        auto exponentials = [m](float4 f) { return make_float4(__expf(f.x - m), __expf(f.y - m), __expf(f.z - m), __expf(f.w - m)); };
        float sum = 0.0f;
#pragma unroll
        for (int k = 0; k < kRegisterGroups; ++k) {
            x[k] = exponentials(x[k]);
            sum += (x[k].x + x[k].y) + (x[k].z + x[k].w);
        }
#pragma unroll
        for (int k = 0; k < kSharedGroups; ++k)
            if (k < parked_groups) {
                const float4 f = exponentials(parked[k * kSplitThreads + tid]);
                parked[k * kSplitThreads + tid] = f;
                sum += (f.x + f.y) + (f.z + f.w);
            }
        total = block_sum(sum, shared);
        label = static_cast<uint32_t>(labels[r]);
        if (tid == 0) row_loss[r] = m + logf(total) - (label < v ? row[label] : 0.0f);
    }
    if (tid == 0) {
        __threadfence();
        const uint32_t before = atomicAdd(counter, 1u);
        is_last = before + 1u == rows;
        if (is_last) *counter = 0u;
    }
    __syncthreads();
    if (is_last) {
        __threadfence();
        double num = 0.0, den64 = 0.0;
        for (uint32_t j = tid; j < rows; j += kSplitThreads) {
            double wj = static_cast<double>(weights[j]);
            num = fma(wj, static_cast<double>(__ldcg(row_loss + j)), num);
            den64 += wj;
        }
        num = block_sum(num, shared64);
        den64 = block_sum(den64, shared64);
        if (denominator != nullptr) den64 = static_cast<double>(denominator[0]);
        if (tid == 0) loss[0] = den64 == 0.0 ? 0.0f : static_cast<float>(num / den64);
    }
    const bool zero = den == 0.0f || w == 0.0f;
    const float scale = zero ? 0.0f : g[0] * w / den;
    const float inverse = zero ? 0.0f : 1.0f / total;
    auto gradient = [=](float4 f, uint32_t c) {
        if (zero) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        return make_float4(scale * (f.x * inverse - (c == label ? 1.0f : 0.0f)), scale * (f.y * inverse - (c + 1 == label ? 1.0f : 0.0f)),
                           scale * (f.z * inverse - (c + 2 == label ? 1.0f : 0.0f)), scale * (f.w * inverse - (c + 3 == label ? 1.0f : 0.0f)));
    };
    // Columns past v inside the pitch are padding nobody reads: the whole float4 is written.
#pragma unroll
    for (int k = 0; k < kRegisterGroups; ++k) {
        const uint32_t c = column_of(k);
        if (c < v) *reinterpret_cast<float4*>(o + c) = gradient(x[k], c);
    }
#pragma unroll
    for (int k = 0; k < kSharedGroups; ++k)
        if (k < parked_groups) {
            const uint32_t c = column_of(kRegisterGroups + k);
            *reinterpret_cast<float4*>(o + c) = gradient(zero ? make_float4(0.0f, 0.0f, 0.0f, 0.0f) : parked[k * kSplitThreads + tid], c);
        }
}

// How a warp holds a row in registers: lane l keeps ITEMS values, V consecutive columns per turn of
// 32 V columns. V = 1 (one 4-byte load per value; the f32 layout) or V = 2 (a bf16 pair per 4-byte
// load, so that a warp's load still covers 128 contiguous bytes).
template <int V> __device__ __forceinline__ uint32_t column_of(int i, uint32_t lane) {
    return static_cast<uint32_t>(i / V) * (32u * V) + lane * V + static_cast<uint32_t>(i % V);
}
// The row's values from clamped columns (what a column past h reads is discarded by the caller):
// unconditional, so that every load of a row is in flight before the first use.
template <int ITEMS, int V, class T>
__device__ __forceinline__ void load_row(const T* __restrict__ row, uint32_t lane, uint32_t h, float (&to)[ITEMS]) {
    if constexpr (V == 1) {
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) to[i] = load1(row + min(i * 32 + lane, h - 1));
    } else {
        static_assert(ITEMS % 2 == 0, "pairs");
#pragma unroll
        for (int j = 0; j < ITEMS / 2; ++j) {
            const float2 f = load2(row + min(j * 64 + lane * 2, h - 2));
            to[2 * j] = f.x;
            to[2 * j + 1] = f.y;
        }
    }
}
template <int ITEMS, int V, class T>
__device__ __forceinline__ void store_row(T* __restrict__ row, uint32_t lane, uint32_t h, const float (&from)[ITEMS]) {
    if constexpr (V == 1) {
#pragma unroll
        for (int i = 0; i < ITEMS; ++i)
            if (i * 32 + lane < h) store1(row + i * 32 + lane, from[i]);
    } else {
#pragma unroll
        for (int j = 0; j < ITEMS / 2; ++j)
            if (j * 64 + lane * 2 < h) store2(row + j * 64 + lane * 2, make_float2(from[2 * j], from[2 * j + 1]));  // h is even
    }
}

// The same as it was read, pairs of bf16 packed: rows that a kernel holds while others are on their way.
template <int ITEMS, int V, class T> struct RawRow {
    static constexpr bool HALF = sizeof(T) == 2;
    static_assert(V == 1 || HALF);
    uint32_t e[V == 2 ? ITEMS / 2 : ITEMS];
    __device__ __forceinline__ void load(Settled<T> row, uint32_t lane, uint32_t h) {
        if constexpr (V == 2) {
#pragma unroll
            for (int j = 0; j < ITEMS / 2; ++j) e[j] = load_settled<uint32_t>((row + min(j * 64 + lane * 2, h - 2)).p);
        } else {
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) {
                if constexpr (HALF) e[i] = load_settled<uint16_t>((row + min(i * 32 + lane, h - 1)).p);
                else e[i] = load_settled<uint32_t>((row + min(i * 32 + lane, h - 1)).p);
            }
        }
    }
    __device__ __forceinline__ float operator[](int i) const {
        if constexpr (V == 2) return i % 2 ? bf16_high(e[i / 2]) : bf16_low(e[i / 2]);
        else return HALF ? bf16_low(e[i]) : __uint_as_float(e[i]);
    }
};

// The keep decisions of one row as the warp holds it (bit i of `mask` = item i of this lane) to
// and from their stored form: word w of the row holds columns 32 w .. 32 w + 31, bit = column
// modulo 32. The row has a multiple of 32 columns, at most 1,024: one word per lane.
__device__ __forceinline__ uint32_t spread16(uint32_t x) {  // bit b of the low half to bit 2 b
    x = (x | (x << 8)) & 0x00FF00FFu;
    x = (x | (x << 4)) & 0x0F0F0F0Fu;
    x = (x | (x << 2)) & 0x33333333u;
    x = (x | (x << 1)) & 0x55555555u;
    return x;
}
template <int ITEMS, int V>
__device__ __forceinline__ void save_keep_bits(uint32_t* __restrict__ row_words, uint32_t lane, uint32_t h, uint32_t mask) {
    uint32_t mine = 0;
    if constexpr (V == 1) {
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const uint32_t word = __ballot_sync(0xffffffffu, (mask >> i) & 1u);  // columns 32 i + lane
            if (lane == static_cast<uint32_t>(i)) mine = word;
        }
    } else {
#pragma unroll
        for (int j = 0; j < ITEMS / 2; ++j) {
            // Lane l holds columns 64 j + 2 l and + 1: lanes 0-15 fill word 2 j, lanes 16-31 word 2 j + 1.
            const uint32_t even = __ballot_sync(0xffffffffu, (mask >> (2 * j)) & 1u), odd = __ballot_sync(0xffffffffu, (mask >> (2 * j + 1)) & 1u);
            if (lane == static_cast<uint32_t>(2 * j)) mine = spread16(even & 0xffffu) | (spread16(odd & 0xffffu) << 1);
            if (lane == static_cast<uint32_t>(2 * j + 1)) mine = spread16(even >> 16) | (spread16(odd >> 16) << 1);
        }
    }
    if (lane < h / 32) row_words[lane] = mine;
}
template <int ITEMS, int V>
__device__ __forceinline__ uint32_t spread_keep_bits(uint32_t mine, uint32_t lane) {
    uint32_t mask = 0;
    if constexpr (V == 1) {
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) mask |= ((__shfl_sync(0xffffffffu, mine, i) >> lane) & 1u) << i;
    } else {
#pragma unroll
        for (int j = 0; j < ITEMS / 2; ++j) {
            const uint32_t word = __shfl_sync(0xffffffffu, mine, 2 * j + static_cast<int>(lane >> 4));
            mask |= ((word >> (2 * (lane & 15u))) & 3u) << (2 * j);
        }
    }
    return mask;
}
// This lane's word of a row's stored decisions (0 where they are drawn).
__device__ __forceinline__ uint32_t stored_keep_word(const DropoutDraw& draw, uint64_t row_at, uint32_t lane, uint32_t h) {
    return draw.token != nullptr && draw.stored && draw.bits != nullptr && lane < h / 32 ? load_global(draw.bits + row_at / 32 + lane) : 0u;
}
// The keep decisions of a row for one site: read when an earlier launch of the step stored them,
// else drawn (element index_base + row h + column of Philox stream 4) and stored when asked.
template <int ITEMS, int V>
__device__ __forceinline__ uint32_t keep_mask(const DropoutDraw& draw, uint64_t row_at, uint32_t lane, uint32_t h, uint32_t stored_word) {
    uint32_t* const row_words = draw.bits ? draw.bits + row_at / 32 : nullptr;
    if (draw.stored && row_words != nullptr) return spread_keep_bits<ITEMS, V>(stored_word, lane);
    const uint32_t id_lo = static_cast<uint32_t>(draw.token[0]), id_hi = static_cast<uint32_t>(draw.token[1]);
    uint32_t mask = 0;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const uint32_t w0 = philox_word0(static_cast<uint32_t>(draw.index_base + row_at + column_of<V>(i, lane)), 4u, id_lo, id_hi,
                                         static_cast<uint32_t>(draw.seed), static_cast<uint32_t>(draw.seed >> 32));
        mask |= (w0 >= draw.threshold ? 1u : 0u) << i;
    }
    if (row_words != nullptr) save_keep_bits<ITEMS, V>(row_words, lane, h, mask);
    return mask;
}

// dropout(x) + residual, then layer_norm of the sum, one warp per row with the row in registers:
// the three launches of a transformer sublayer's tail as one. Every element goes through the same
// rounded operations as the separate kernels (the Philox draw of element index_base + r h + c, the
// scaled or zeroed value, one addition, the layer norm of the stored sum). Each part is optional:
// without a draw on x the sum is x + residual; without gamma the launch ends with the sum; with a
// draw on the result, dropout of the layer norm is written to out_dropped (and out may be null);
// sum_out may be null when only the layer norm is wanted.
// EXACT: the row is ITEMS x 32 wide, so that no column has to be tested. The test of every value, a
// branch around a load or a store each, cost more than the arithmetic (16,384 bf16 rows of 768: 75 -> 59 us, of which some 40 are the Philox rounds).
// The Philox rounds are what it waits for: of rows of 768, three blocks to an SM (80 registers) keep the
// integer units busier than the two of 92 (68 -> 59 us).
template <int ITEMS, int V, bool EXACT, class T>
__global__ void __launch_bounds__(256, !EXACT ? 1 : ITEMS >= 32 ? 2 : ITEMS >= 24 ? 3 : 4) dropout_add_layer_norm_kernel(
    const T* x, const T* residual, DropoutDraw x_draw, const float* gamma,
    const float* beta, T* sum_out, T* out, DropoutDraw out_draw,
    T* out_dropped, uint32_t rows, uint32_t width_given, bool gelu_first) {
    after_producers();
    const uint32_t h = EXACT ? 32u * ITEMS : width_given;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t r = blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
    if (r >= rows) return;
    const uint64_t base = static_cast<uint64_t>(r) * h;
    // The loads first, so that all are in flight before the Philox rounds of the first element start.
    float v[ITEMS], xs[ITEMS];
    load_row<ITEMS, V>(x + base, lane, h, xs);
    if (residual != nullptr) load_row<ITEMS, V>(residual + base, lane, h, v);
    const uint32_t x_word = stored_keep_word(x_draw, base, lane, h), out_word = stored_keep_word(out_draw, base, lane, h);
    constexpr bool HELD_GAMMA = ITEMS <= 8;  // (wider rows have no registers left for it)
    float gam[HELD_GAMMA ? ITEMS : 1], bet[HELD_GAMMA ? ITEMS : 1];
    if constexpr (HELD_GAMMA) {
        if (gamma != nullptr) {
            load_row<ITEMS, V>(gamma, lane, h, gam);
            load_row<ITEMS, V>(beta, lane, h, bet);
        }
    }
    // gelu(x) in the place of the sum (the head's transform: dense, gelu, layer norm).
    if (gelu_first) {
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) xs[i] = gelu_value_for<T>(xs[i]);
    }
    if (x_draw.token != nullptr) {
        const uint32_t keep = keep_mask<ITEMS, V>(x_draw, base, lane, h, x_word);
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) xs[i] = (keep >> i) & 1u ? xs[i] * x_draw.scale : 0.0f;
    }
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const uint32_t c = column_of<V>(i, lane);
        v[i] = c < h ? (residual != nullptr ? v[i] + xs[i] : xs[i]) : 0.0f;
        // What is stored is what the layer norm below reads: the sum as its storage type holds it.
        v[i] = stored_as(v[i], static_cast<const T*>(nullptr));
    }
    if (sum_out != nullptr) store_row<ITEMS, V>(sum_out + base, lane, h, v);
    if (gamma == nullptr) return;
    const float width = static_cast<float>(h);
    float sum = 0.0f;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i)
        if (column_of<V>(i, lane) < h) sum += v[i];
    const float mean = warp_sum(sum) / width;
    float q = 0.0f;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i)
        if (column_of<V>(i, lane) < h) {
            float d = v[i] - mean;
            q = fmaf(d, d, q);
        }
    const float rstd = 1.0f / sqrtf(warp_sum(q) / width + kLayerNormEps);
    const uint32_t keep_out = out_dropped != nullptr ? keep_mask<ITEMS, V>(out_draw, base, lane, h, out_word) : 0u;
    float dropped[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const uint32_t c = column_of<V>(i, lane);
        const uint32_t cc = min(c, h - 1);
        const float y = HELD_GAMMA ? (v[i] - mean) * rstd * gam[HELD_GAMMA ? i : 0] + bet[HELD_GAMMA ? i : 0] : (v[i] - mean) * rstd * gamma[cc] + beta[cc];
        v[i] = y;
        dropped[i] = (out_dropped != nullptr && c < h && ((keep_out >> i) & 1u)) ? y * out_draw.scale : 0.0f;
    }
    if (out != nullptr) store_row<ITEMS, V>(out + base, lane, h, v);
    if (out_dropped != nullptr) store_row<ITEMS, V>(out_dropped + base, lane, h, dropped);
}

// layer_norm_grad_x, layer_norm_grad_gamma and the beta gradient in one launch. A block takes a
// chunk of rows, a warp one row at a time with the row of x and of g in registers (ITEMS values
// per lane): row moments, then the dx row, then this row's terms of the column sums. Warp sums of
// a chunk are added in warp order, chunk sums by the last block to finish: thread (lane, w) adds
// chunks w, w + 8, ... in ascending order and the eight sums are added in ascending w. Every
// output is a fixed expression of the inputs: deterministic, tolerance class against a
// sequential column sum. dx (with gamma), dgamma and dbeta may each be null.
// Rows of 512 or more elements (ITEMS >= 16) keep their column sums in shared memory instead of
// registers (the same additions in the same order), and gamma is read where it is used: with the
// sums and gamma in registers a thread needs about 250 of them, one block of 8 warps fills an SM's
// register file, and the loads of a row have nothing to hide behind.
// EXACT: the row is ITEMS x 32 wide, so that no column has to be tested and the loads of gamma and the
// updates of the column sums go out together (16,384 bf16 rows of 768 with an addend and a dropped
// copy: 71 -> 44 us).
// Blocks to an SM: four where 64 registers hold a row (4,096 bf16 rows of 128 in one wave: a BERT-tiny step 5 us less), else
// two (as four, f32 rows of 128 spill: a BERT-tiny step 4 us more).
template <int ITEMS, int V, bool EXACT, class T>
__global__ void __launch_bounds__(256, ITEMS <= 2 || (ITEMS <= 4 && EXACT && sizeof(T) == 2) ? 4 : 2) layer_norm_backward_kernel(
    const T* x, const float* gamma, const T* g, const T* g1,
    const T* g2, const T* g3, T* dx,
    float* partial, uint32_t* counter, float* dgamma, float* dbeta,
    uint32_t want, uint32_t rows, uint32_t width_given, uint32_t rows_per_chunk, DropoutDraw adjoint_draw, DropoutDraw dx_draw,
    T* dx_dropped, const T* pre_activation) {
    after_producers();
    const Settled<T> x_rows = settled(x), g_rows = settled(g), pre_rows = settled(pre_activation), added_rows[3] = {settled(g1), settled(g2), settled(g3)};
    constexpr bool WIDE = ITEMS >= 16;
    const uint32_t h = EXACT ? 32u * ITEMS : width_given;
    extern __shared__ float backward_sums[];  // 8 * 32 * ITEMS floats, twice that for wide rows
    float* const buf = backward_sums;
    float* const buf_b = backward_sums + (WIDE ? 8 * 32 * ITEMS : 0);
    __shared__ bool is_last;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, chunks = gridDim.x;
    const uint32_t r0 = blockIdx.x * rows_per_chunk, r1 = min(rows, r0 + rows_per_chunk);
    const float width = static_cast<float>(h);
    // dx is formed when it is stored or when what is stored is a function of it.
    const bool want_dx = dx != nullptr || dx_dropped != nullptr;
    constexpr int HELD = WIDE ? 1 : ITEMS;
    float acc_g[HELD], acc_b[HELD], gam[HELD];
    // This thread's column sums when they live in shared memory: value i at [i * 32].
    float* const sum_g = buf + warp * ITEMS * 32 + lane;
    float* const sum_b = buf_b + (WIDE ? warp * ITEMS * 32 + lane : 0);
    if constexpr (WIDE) {
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            sum_g[i * 32] = 0.0f;
            sum_b[i * 32] = 0.0f;
        }
    } else {
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            acc_g[i] = 0.0f;
            acc_b[i] = 0.0f;
            uint32_t c = column_of<V>(i, lane);
            gam[i] = (want_dx && c < h) ? gamma[c] : 0.0f;
        }
    }
    for (uint32_t r = r0 + warp; r < r1; r += 8) {
        // All loads of a row are issued before any is used: unconditional, from clamped columns (what a column
        // past h reads is discarded below), the addends of the adjoint, the stored decisions and the
        // pre-activations with the rest. A load behind a use of another one would wait for that
        // (an addend or a pre-activation each a trip to the L2; inside a step 2,200 bf16 rows of 200 take 2.4 us less so,
        // 4,096 f32 rows of 256 2.3). Wide f32 rows have registers for two arrays: their addends follow, out of the L2.
        const uint64_t row_at = static_cast<uint64_t>(r) * h;
        constexpr int AHEAD = !WIDE ? 3 : sizeof(T) == 2 && V == 2 ? 1 : 0;  // addends held while x and g are on their way
        const uint32_t adjoint_word = stored_keep_word(adjoint_draw, row_at, lane, h), dx_word = stored_keep_word(dx_draw, row_at, lane, h);
        const T* const addends[3] = {g1, g2, g3};
        float xv[ITEMS], gv[ITEMS];
        RawRow<!WIDE ? ITEMS : 2, V, T> pre_raw;
        {
            RawRow<ITEMS, V, T> x_raw, g_raw, more[AHEAD > 0 ? AHEAD : 1];
            x_raw.load(x_rows + row_at, lane, h);
            g_raw.load(g_rows + row_at, lane, h);
#pragma unroll
            for (int a = 0; a < AHEAD; ++a)
                if (added_rows[a]) more[a].load(added_rows[a] + row_at, lane, h);
            if constexpr (!WIDE) {
                if (pre_rows) pre_raw.load(pre_rows + row_at, lane, h);
            }
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) {
                xv[i] = x_raw[i];
                gv[i] = g_raw[i];
            }
            // The adjoint as a sum the program spells as a chain of Adds: ((g + g1) + g2) + g3.
#pragma unroll
            for (int a = 0; a < AHEAD; ++a) {
                if (addends[a] == nullptr) continue;
#pragma unroll
                for (int i = 0; i < ITEMS; ++i) gv[i] = gv[i] + more[a][i];
            }
        }
        if constexpr (WIDE) {
            // The warp's next row on its way into the L2, 128 bytes a lane.
            if (r + 8 < r1 && lane * 128u < h * sizeof(T)) {
                const uint64_t next = row_at + 8ull * h;
                for (const T* from : {x, g, g1, g2, g3})
                    if (from != nullptr) asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char*>(from + next) + lane * 128u));
            }
        }
#pragma unroll
        for (int a = AHEAD; a < 3; ++a) {
            if (addends[a] == nullptr) continue;
            float t[ITEMS];
            load_row<ITEMS, V>(addends[a] + row_at, lane, h, t);
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) gv[i] = gv[i] + t[i];
        }
        // An adjoint that the program passes through dropout_grad first: the draw of element
        // (r, c), on the sum.
        if (adjoint_draw.token != nullptr) {
            const uint32_t keep = keep_mask<ITEMS, V>(adjoint_draw, row_at, lane, h, adjoint_word);
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) gv[i] = (keep >> i) & 1u ? gv[i] * adjoint_draw.scale : 0.0f;
        }
#pragma unroll
        for (int i = 0; i < ITEMS; ++i)
            if (column_of<V>(i, lane) >= h) {
                xv[i] = 0.0f;
                gv[i] = 0.0f;
            }
        float sum = 0.0f;
#pragma unroll
        for (int i = 0; i < ITEMS; ++i)
            if (column_of<V>(i, lane) < h) sum += xv[i];
        const float mean = warp_sum(sum) / width;
        float q = 0.0f;
#pragma unroll
        for (int i = 0; i < ITEMS; ++i)
            if (column_of<V>(i, lane) < h) {
                float d = xv[i] - mean;
                q = fmaf(d, d, q);
            }
        const float rstd = 1.0f / sqrtf(warp_sum(q) / width + kLayerNormEps);
        float s1 = 0.0f, s2 = 0.0f;
        // Gamma of a wide row: loaded together where registers are left for it, else where it is used.
        constexpr bool ROW_GAMMA = WIDE && ITEMS <= 24;
        float row_gamma[ROW_GAMMA ? ITEMS : 1];
        if constexpr (ROW_GAMMA) {
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) row_gamma[i] = 0.0f;
            if (want_dx) load_row<ITEMS, V>(gamma, lane, h, row_gamma);
        }
        auto gamma_of = [&](int i) -> float {
            if constexpr (!WIDE) return gam[i];
            else if constexpr (ROW_GAMMA) return row_gamma[i];
            else return want_dx ? load_global(gamma + column_of<V>(i, lane)) : 0.0f;
        };
#pragma unroll
        for (int i = 0; i < ITEMS; ++i)
            if (column_of<V>(i, lane) < h) {
                float xhat = (xv[i] - mean) * rstd;
                if constexpr (WIDE) {
                    sum_g[i * 32] = fmaf(gv[i], xhat, sum_g[i * 32]);
                    sum_b[i * 32] += gv[i];
                } else {
                    acc_g[i] = fmaf(gv[i], xhat, acc_g[i]);
                    acc_b[i] += gv[i];
                }
                float gx = gv[i] * gamma_of(i);
                s1 += gx;
                s2 = fmaf(gx, xhat, s2);
                // The dx row below is a function of these two: kept in the registers of x and g.
                xv[i] = xhat;
                gv[i] = gx;
            }
        if (want_dx) {
            const float mean_gx = warp_sum(s1) / width, mean_gx_xhat = warp_sum(s2) / width;
            // The pre-activations of a gelu_grad on dx: loaded together, before the first is used.
            float pre[ITEMS];
            if (pre_activation != nullptr) {
                if constexpr (!WIDE) {
#pragma unroll
                    for (int i = 0; i < ITEMS; ++i) pre[i] = pre_raw[i];
                } else {
                    load_row<ITEMS, V>(pre_activation + row_at, lane, h, pre);
                }
            }
            float second[ITEMS];
            const uint32_t keep_dx = (pre_activation == nullptr && dx_dropped != nullptr) ? keep_mask<ITEMS, V>(dx_draw, row_at, lane, h, dx_word) : 0u;
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) {
                const uint32_t c = column_of<V>(i, lane);
                const float gx = gv[i], xhat = xv[i];
                const float value = rstd * ((gx - mean_gx) - xhat * mean_gx_xhat);
                xv[i] = value;  // the dx row, in the registers of the x row
                second[i] = 0.0f;
                // A function of dx for the reader that wants that: gelu_grad (the dense layer
                // before a gelu and this layer norm), or dropout_grad (the projection before
                // this sublayer's dropout).
                if (pre_activation != nullptr) {
                    second[i] = gelu_grad_value_for<T>(pre[i], value);
                } else if (dx_dropped != nullptr && c < h) {
                    second[i] = (keep_dx >> i) & 1u ? value * dx_draw.scale : 0.0f;
                }
            }
            if (dx != nullptr) store_row<ITEMS, V>(dx + row_at, lane, h, xv);
            if (dx_dropped != nullptr) store_row<ITEMS, V>(dx_dropped + row_at, lane, h, second);
        }
    }
    if (want == 0) return;
    float* partial_gamma = partial + static_cast<uint64_t>(blockIdx.x) * h;
    float* partial_beta = partial + static_cast<uint64_t>(chunks + blockIdx.x) * h;
#pragma unroll
    for (int pass = 0; pass < 2; ++pass) {
        if ((want & (1u << pass)) == 0) continue;
        __syncthreads();
        if constexpr (!WIDE) {
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) buf[(warp * ITEMS + i) * 32 + lane] = pass == 0 ? acc_g[i] : acc_b[i];
        }
        __syncthreads();
        const float* const sums = (WIDE && pass == 1) ? buf_b : buf;
        for (uint32_t c = threadIdx.x; c < h; c += 256) {
            // Column c is value i of lane l (the inverse of column_of).
            const uint32_t turn = c / (32u * V), within = c % (32u * V);
            const uint32_t i = turn * V + within % V, l = within / V;
            float total = sums[i * 32 + l];
#pragma unroll
            for (int w = 1; w < 8; ++w) total += sums[(w * ITEMS + i) * 32 + l];
            (pass == 0 ? partial_gamma : partial_beta)[c] = total;
        }
    }
    if (counter == nullptr) return;  // the chunk sums are added later, by finalize_sums
    if (!last_block_arrives(counter, chunks, &is_last)) return;
    for (int pass = 0; pass < 2; ++pass) {
        float* out = pass == 0 ? dgamma : dbeta;
        if ((want & (1u << pass)) == 0) continue;
        const float* from = partial + static_cast<uint64_t>(pass) * chunks * h;
        for (uint32_t c0 = 0; c0 < h; c0 += 32) {
            uint32_t c = c0 + lane;
            float total = 0.0f;
            if (c < h)
                for (uint32_t k = warp; k < chunks; k += 8) total += __ldcg(from + static_cast<uint64_t>(k) * h + c);
            __syncthreads();
            buf[warp * 32 + lane] = total;
            __syncthreads();
            if (warp == 0 && c < h) {
                float t = buf[lane];
#pragma unroll
                for (int w = 1; w < 8; ++w) t += buf[w * 32 + lane];
                out[c] = t;
            }
        }
    }
}

// The one-read kernels. Rows on 16-byte boundaries: a warp a row up to 1,024 logits (a row's maximum and sum without a
// barrier), then the fewest threads that hold the row in 32 registers each, so that more rows share an SM (f32 beyond 16,384: half of it in shared memory). Other rows: 1,024 threads, an element a load.
constexpr uint64_t kWideRow = static_cast<uint64_t>(kWideThreads) * kWideItems, kLongestRow = 65536;
template <class T>
void launch_cross_entropy_one_read(cudaStream_t s, const T* logits, const int32_t* labels, const float* weights, const float* g,
                                   const float* den, float* row_loss, T* grad, uint32_t vv, uint32_t l1, uint32_t l2, uint32_t* counter,
                                   float* loss, uint32_t rows, bool vec) {
    constexpr bool HALF = sizeof(T) == 2;
    if (!vec) {
        cross_entropy_fused_wide_kernel<<<rows, kWideThreads, 0, s>>>(logits, labels, weights, g, den, row_loss, grad, vv, l1, l2, counter, loss);
        return;
    }
    constexpr int G = HALF ? 4 : 8;  // pieces of 16 bytes that hold 32 elements
    auto rows_in_registers = [&](auto kernel, uint32_t threads, uint32_t rows_a_block) {
        kernel<<<(rows + rows_a_block - 1) / rows_a_block, threads * rows_a_block, 0, s>>>(logits, labels, weights, g, den, row_loss, grad, rows, vv,
                                                                                           l1, l2, counter, loss);
    };
    if (vv <= 128) rows_in_registers(cross_entropy_row_kernel<32, 4, 1, 1, T>, 32, 4);
    else if (vv <= 1024) rows_in_registers(cross_entropy_row_kernel<32, 4, G, 1, T>, 32, 4);
    else if (vv <= 4096) rows_in_registers(cross_entropy_row_kernel<128, 1, G, 1, T>, 128, 1);
    else if (vv <= 8192) rows_in_registers(cross_entropy_row_kernel<256, 1, G, 1, T>, 256, 1);
    else if (vv <= 16384) rows_in_registers(cross_entropy_row_kernel<512, 1, G, 2, T>, 512, 1);
    else if constexpr (HALF) {
        if (vv <= 32768) rows_in_registers(cross_entropy_row_kernel<512, 1, 8, 2, T>, 512, 1);
        else rows_in_registers(cross_entropy_row_kernel<1024, 1, 8, 1, T>, 1024, 1);
    } else {
        auto split = [&](auto kernel, int threads, std::atomic<int>& configured_device) {
            const int bytes = kSplitSharedItems * threads * 4;
            set_shared_memory(kernel, bytes, configured_device);
            kernel<<<rows, threads, bytes, s>>>(logits, labels, weights, g, den, row_loss, grad, vv, l1, l2, counter, loss);
        };
        static std::atomic<int> half_device{-1}, whole_device{-1};
        if (vv <= 32768) split(cross_entropy_fused_split_kernel<512>, 512, half_device);
        else split(cross_entropy_fused_split_kernel<1024>, 1024, whole_device);
    }
}

uint32_t backward_chunks(uint64_t rows, uint64_t h) {
    // Four blocks per SM: a warp walks its rows one after another, each row a chain of loads and
    // three warp reductions, so it is the number of warps in flight that hides that latency (4,096
    // rows of 128: a row a warp, 8.4 us; three blocks per SM left a quarter of the warps a second
    // row, 10.5 us). Rows
    // of more than 256 elements keep their column sums in shared memory, two blocks per SM: one wave
    // of 296 blocks instead of a full wave and a half one.
    const uint64_t blocks = h > 256 ? MSX_LN_BACKWARD_WIDE_BLOCKS : MSX_LN_BACKWARD_BLOCKS;
    uint64_t per = (rows + blocks - 1) / blocks;
    if (per < 8) per = 8;
    uint64_t chunks = (rows + per - 1) / per;
    return static_cast<uint32_t>(chunks < 1 ? 1 : chunks);
}

}  // namespace

void layer_norm(cudaStream_t s, const float* x, const float* gamma, const float* beta, float* out,
                uint64_t rows, uint64_t h) {
    if (rows == 0) return;
    layer_norm_kernel<<<warp_row_blocks(rows), kWarpsPerBlock * 32, 0, s>>>(x, gamma, beta, out,
                                                                            static_cast<uint32_t>(rows), static_cast<uint32_t>(h));
    check_launch("layer_norm");
}

void layer_norm_grad_x(cudaStream_t s, const float* x, const float* gamma, const float* g, float* out,
                       uint64_t rows, uint64_t h) {
    if (rows == 0) return;
    layer_norm_grad_x_kernel<<<warp_row_blocks(rows), kWarpsPerBlock * 32, 0, s>>>(
        x, gamma, g, out, static_cast<uint32_t>(rows), static_cast<uint32_t>(h));
    check_launch("layer_norm_grad_x");
}

uint64_t layer_norm_grad_gamma_scratch_floats(uint64_t rows, uint64_t h) {
    return 2 * rows + 2 * sum_rows_chunks(rows) * h;
}

void layer_norm_grad_gamma(cudaStream_t s, const float* x, const float* g, float* scratch, float* dgamma,
                           float* dbeta, uint64_t rows, uint64_t h) {
    if (h == 0) return;
    uint32_t chunks = sum_rows_chunks(rows);
    uint32_t rows_per_chunk = static_cast<uint32_t>((rows + chunks - 1) / chunks);
    float* stats = scratch;
    float* partial_gamma = scratch + 2 * rows;
    float* partial_beta = partial_gamma + static_cast<uint64_t>(chunks) * h;
    if (rows > 0) {
        row_stats_kernel<<<warp_row_blocks(rows), kWarpsPerBlock * 32, 0, s>>>(x, stats, static_cast<uint32_t>(rows),
                                                                                static_cast<uint32_t>(h));
        check_launch("layer_norm_grad_gamma");
    }
    dim3 grid(static_cast<uint32_t>((h + 31) / 32), chunks);
    grad_gamma_stage1<<<grid, dim3(32, 8), 0, s>>>(x, g, stats, static_cast<uint32_t>(rows), static_cast<uint32_t>(h),
                                                   rows_per_chunk, partial_gamma, dbeta ? partial_beta : nullptr);
    check_launch("layer_norm_grad_gamma");
    grad_gamma_stage2<<<static_cast<uint32_t>((h + 127) / 128), 128, 0, s>>>(partial_gamma, partial_beta, chunks,
                                                                              static_cast<uint32_t>(h), dgamma, dbeta);
    check_launch("layer_norm_grad_gamma");
}

namespace {
template <class T>
void launch_add_layer_norm(cudaStream_t s, const T* x, const T* residual, const DropoutDraw& first, const float* gamma, const float* beta,
                           T* sum_out, T* out, const DropoutDraw& second, T* out_dropped, uint64_t rows, uint64_t h, bool gelu_first) {
    const uint32_t items = static_cast<uint32_t>((h + 31) / 32), blocks = static_cast<uint32_t>((rows + kWarpsPerBlock - 1) / kWarpsPerBlock);
    const uint32_t r = static_cast<uint32_t>(rows), hh = static_cast<uint32_t>(h);
    // bf16 rows of even width are held as pairs (4-byte loads); everything else one value per load.
    constexpr int PAIR = sizeof(T) == 2 ? 2 : 1;
    const bool pairs = PAIR == 2 && h % 2 == 0 && items >= 2;
#define MSX_DROPOUT_LN_ONE(N, W, E) dropout_add_layer_norm_kernel<N, W, E><<<blocks, 256, 0, s>>>(x, residual, first, gamma, beta, sum_out, out, second, out_dropped, r, hh, gelu_first)
#define MSX_DROPOUT_LN(N) do { \
        if (h == 32 * N) MSX_DROPOUT_LN_ONE(N, (N % 2 == 0 ? PAIR : 1), true); \
        else if (pairs) MSX_DROPOUT_LN_ONE(N, (N % 2 == 0 ? PAIR : 1), false); \
        else MSX_DROPOUT_LN_ONE(N, 1, false); } while (0)
    if (items <= 1) MSX_DROPOUT_LN(1);
    else if (items <= 2) MSX_DROPOUT_LN(2);
    else if (items <= 4) MSX_DROPOUT_LN(4);
    else if (items <= 8) MSX_DROPOUT_LN(8);
    else if (items <= 16) MSX_DROPOUT_LN(16);
    else if (items <= 24) MSX_DROPOUT_LN(24);
    else MSX_DROPOUT_LN(32);
#undef MSX_DROPOUT_LN
#undef MSX_DROPOUT_LN_ONE
    check_launch("add_layer_norm");
}
template <class T> const T* typed(In a) { return static_cast<const T*>(a.p); }
template <class T> T* typed(Out a) { return static_cast<T*>(a.p); }
}  // namespace

void add_layer_norm(cudaStream_t s, In x, In residual, const DropoutDraw* x_draw, const float* gamma,
                    const float* beta, Out sum_out, Out out, const DropoutDraw* out_draw, Out out_dropped, uint64_t rows,
                    uint64_t h, bool gelu_first) {
    if (rows == 0 || h == 0) return;
    const DropoutDraw none = {};
    const DropoutDraw first = x_draw ? *x_draw : none, second = out_draw ? *out_draw : none;
    if (out_draw == nullptr || gamma == nullptr) out_dropped = Out();
    // The element type of the launch is that of x; the optional operands that are present share it.
    const bool half = x.half;
    for (bool other : {residual ? residual.half : half, sum_out ? sum_out.half : half, out ? out.half : half, out_dropped ? out_dropped.half : half})
        if (other != half) throw std::invalid_argument("add_layer_norm: f32 and bf16 activation operands in one launch");
    if (half)
        launch_add_layer_norm(s, typed<bf16>(x), typed<bf16>(residual), first, gamma, beta, typed<bf16>(sum_out), typed<bf16>(out), second,
                              typed<bf16>(out_dropped), rows, h, gelu_first);
    else
        launch_add_layer_norm(s, typed<float>(x), typed<float>(residual), first, gamma, beta, typed<float>(sum_out), typed<float>(out), second,
                              typed<float>(out_dropped), rows, h, gelu_first);
}

void dropout_add_layer_norm(cudaStream_t s, In x, In residual, const int32_t* token, uint64_t seed,
                            uint32_t threshold, float scale, uint64_t index_base, const float* gamma, const float* beta,
                            Out sum_out, Out out, uint64_t rows, uint64_t h) {
    DropoutDraw draw;
    draw.token = token;
    draw.seed = seed;
    draw.threshold = threshold;
    draw.scale = scale;
    draw.index_base = index_base;
    add_layer_norm(s, x, residual, &draw, gamma, beta, sum_out, out, nullptr, Out(), rows, h, false);
}

bool layer_norm_backward_supported(uint64_t h) { return h >= 1 && h <= 1024; }
uint32_t layer_norm_backward_chunks(uint64_t rows, uint64_t h) { return backward_chunks(rows, h); }
uint64_t layer_norm_backward_scratch_floats(uint64_t rows, uint64_t h) { return 2ull * backward_chunks(rows, h) * h; }

namespace {
template <class T>
void launch_layer_norm_backward(cudaStream_t s, const T* x, const float* gamma, const T* g, T* dx, float* scratch, uint32_t* counter,
                                float* dgamma, float* dbeta, uint64_t rows, uint64_t h, const T* g1, const T* g2, const T* g3,
                                const DropoutDraw& in_draw, const DropoutDraw& out_draw, T* dx_dropped, const T* pre_activation) {
    uint32_t chunks = backward_chunks(rows, h);
    uint32_t per = static_cast<uint32_t>((rows + chunks - 1) / chunks);
    uint32_t items = static_cast<uint32_t>((h + 31) / 32);
    uint32_t r = static_cast<uint32_t>(rows), hh = static_cast<uint32_t>(h);
    uint32_t want = (dgamma ? 1u : 0u) | (dbeta ? 2u : 0u);
    constexpr int PAIR = sizeof(T) == 2 ? 2 : 1;
    const bool pairs = PAIR == 2 && h % 2 == 0 && items >= 2;
    // Shared memory of the column sums: one array of 8 x 32 x N floats, two for rows of 512 or more.
#define MSX_LN_BACKWARD_ONE(N, W, E) do { \
        auto kernel = layer_norm_backward_kernel<N, W, E, T>; \
        constexpr uint32_t bytes = (N >= 16 ? 2u : 1u) * 8u * 32u * N * 4u; \
        if (bytes > 40000u) { \
            static std::atomic<int> configured_device{-1}; \
            set_shared_memory(kernel, static_cast<int>(bytes), configured_device); \
        } \
        kernel<<<chunks, 256, bytes, s>>>(x, gamma, g, g1, g2, g3, dx, scratch, counter, dgamma, dbeta, want, r, hh, per, in_draw, out_draw, dx_dropped, pre_activation); } while (0)
#define MSX_LN_BACKWARD(N) do { \
        if (h == 32 * N) MSX_LN_BACKWARD_ONE(N, (N % 2 == 0 ? PAIR : 1), true); \
        else if (pairs) MSX_LN_BACKWARD_ONE(N, (N % 2 == 0 ? PAIR : 1), false); \
        else MSX_LN_BACKWARD_ONE(N, 1, false); } while (0)
    if (items <= 1) MSX_LN_BACKWARD(1);
    else if (items <= 2) MSX_LN_BACKWARD(2);
    else if (items <= 4) MSX_LN_BACKWARD(4);
    else if (items <= 8) MSX_LN_BACKWARD(8);
    else if (items <= 16) MSX_LN_BACKWARD(16);
    else if (items <= 24) MSX_LN_BACKWARD(24);
    else MSX_LN_BACKWARD(32);
#undef MSX_LN_BACKWARD
#undef MSX_LN_BACKWARD_ONE
    check_launch("layer_norm_backward");
}
}  // namespace

void layer_norm_backward(cudaStream_t s, In x, const float* gamma, In g, Out dx, float* scratch,
                         uint32_t* counter, float* dgamma, float* dbeta, uint64_t rows, uint64_t h, In g1, In g2,
                         In g3, const DropoutDraw* adjoint_draw, const DropoutDraw* dx_draw, Out dx_dropped,
                         In pre_activation) {
    if (h == 0) return;
    const DropoutDraw none = {};
    const DropoutDraw in_draw = adjoint_draw ? *adjoint_draw : none, out_draw = dx_draw ? *dx_draw : none;
    if (dx_draw == nullptr && !pre_activation) dx_dropped = Out();
    if (!dx_dropped) pre_activation = In();
    const bool half = x.half;
    for (bool other : {g.half, g1 ? g1.half : half, g2 ? g2.half : half, g3 ? g3.half : half, dx ? dx.half : half,
                       dx_dropped ? dx_dropped.half : half, pre_activation ? pre_activation.half : half})
        if (other != half) throw std::invalid_argument("layer_norm_backward: f32 and bf16 activation operands in one launch");
    if (half)
        launch_layer_norm_backward(s, typed<bf16>(x), gamma, typed<bf16>(g), typed<bf16>(dx), scratch, counter, dgamma, dbeta, rows, h,
                                   typed<bf16>(g1), typed<bf16>(g2), typed<bf16>(g3), in_draw, out_draw, typed<bf16>(dx_dropped),
                                   typed<bf16>(pre_activation));
    else
        launch_layer_norm_backward(s, typed<float>(x), gamma, typed<float>(g), typed<float>(dx), scratch, counter, dgamma, dbeta, rows, h,
                                   typed<float>(g1), typed<float>(g2), typed<float>(g3), in_draw, out_draw, typed<float>(dx_dropped),
                                   typed<float>(pre_activation));
}

void softmax(cudaStream_t s, const float* x, float* out, uint64_t rows, uint64_t k) {
    if (rows == 0) return;
    softmax_kernel<<<static_cast<uint32_t>(rows), kRowThreads, 0, s>>>(x, out, static_cast<uint32_t>(k));
    check_launch("softmax");
}

void softmax_grad(cudaStream_t s, const float* y, const float* g, float* out, uint64_t rows, uint64_t k) {
    if (rows == 0) return;
    softmax_grad_kernel<<<static_cast<uint32_t>(rows), kRowThreads, 0, s>>>(y, g, out, static_cast<uint32_t>(k));
    check_launch("softmax_grad");
}

void weight_sum(cudaStream_t s, const float* weights, uint64_t rows, float* out) {
    weight_sum_kernel<<<1, 1024, 0, s>>>(weights, static_cast<uint32_t>(rows), out);
    check_launch("weight_sum");
}

void cross_entropy(cudaStream_t s, In logits, const int32_t* labels, const float* weights,
                   float* row_loss, const float* global_den, float* loss, uint64_t rows, uint64_t v, uint64_t ld) {
    if (ld == 0) ld = v;
    if (rows > 0) {
        if (logits.half)
            cross_entropy_rows_kernel<<<static_cast<uint32_t>(rows), kRowThreads, 0, s>>>(typed<bf16>(logits), labels, weights, row_loss,
                                                                                          static_cast<uint32_t>(v), static_cast<uint32_t>(ld));
        else
            cross_entropy_rows_kernel<<<static_cast<uint32_t>(rows), kRowThreads, 0, s>>>(typed<float>(logits), labels, weights, row_loss,
                                                                                          static_cast<uint32_t>(v), static_cast<uint32_t>(ld));
        check_launch("cross_entropy");
    }
    cross_entropy_loss_kernel<<<1, 1024, 0, s>>>(row_loss, weights, static_cast<uint32_t>(rows), global_den, loss);
    check_launch("cross_entropy");
}

namespace {
template <class T>
void launch_cross_entropy_with_grad(cudaStream_t s, const T* logits, const int32_t* labels, const float* weights, const float* g,
                                    bool denominator_ready, float* denominator, float* row_loss, float* loss, T* grad, uint64_t rows,
                                    uint64_t v, uint32_t* counter, uint64_t ld, uint64_t ld_grad) {
    const uint32_t vv = static_cast<uint32_t>(v), l1 = static_cast<uint32_t>(ld), l2 = static_cast<uint32_t>(ld_grad);
    constexpr uint64_t E = 16 / sizeof(T);
    const bool vec = ld % E == 0 && ld_grad % E == 0 && reinterpret_cast<uintptr_t>(logits) % 16 == 0 && reinterpret_cast<uintptr_t>(grad) % 16 == 0;
    if (rows > 0 && counter != nullptr && v > 0 && v <= (vec ? kLongestRow : kWideRow)) {
        const float* den = denominator_ready ? denominator : nullptr;
        launch_cross_entropy_one_read(s, logits, labels, weights, g, den, row_loss, grad, vv, l1, l2, counter, loss,
                                      static_cast<uint32_t>(rows), vec);
        check_launch("cross_entropy_with_grad");
        return;
    }
    if (!denominator_ready) {
        weight_sum_kernel<<<1, 1024, 0, s>>>(weights, static_cast<uint32_t>(rows), denominator);
        check_launch("cross_entropy_with_grad");
    }
    if (rows > 0) {
        cross_entropy_fused_kernel<<<static_cast<uint32_t>(rows), kRowThreads, 0, s>>>(logits, labels, weights, g, denominator, row_loss,
                                                                                       grad, vv, l1, l2);
        check_launch("cross_entropy_with_grad");
    }
    cross_entropy_loss_kernel<<<1, 1024, 0, s>>>(row_loss, weights, static_cast<uint32_t>(rows), denominator_ready ? denominator : nullptr, loss);
    check_launch("cross_entropy_with_grad");
}
}  // namespace

void cross_entropy_with_grad(cudaStream_t s, In logits, const int32_t* labels, const float* weights,
                             const float* g, bool denominator_ready, float* denominator, float* row_loss, float* loss,
                             Out grad, uint64_t rows, uint64_t v, uint32_t* counter, uint64_t ld, uint64_t ld_grad) {
    if (ld == 0) ld = v;
    if (ld_grad == 0) ld_grad = v;
    if (all_half({logits.half, grad.half}, "cross_entropy_with_grad"))
        launch_cross_entropy_with_grad(s, typed<bf16>(logits), labels, weights, g, denominator_ready, denominator, row_loss, loss,
                                       typed<bf16>(grad), rows, v, counter, ld, ld_grad);
    else
        launch_cross_entropy_with_grad(s, typed<float>(logits), labels, weights, g, denominator_ready, denominator, row_loss, loss,
                                       typed<float>(grad), rows, v, counter, ld, ld_grad);
}

void cross_entropy_grad(cudaStream_t s, const float* logits, const int32_t* labels, const float* weights,
                        const float* g, bool denominator_ready, float* denominator, float* out, uint64_t rows,
                        uint64_t v, uint64_t ld, uint64_t ld_out) {
    if (rows == 0) return;
    if (ld == 0) ld = v;
    if (ld_out == 0) ld_out = v;
    if (!denominator_ready) {
        weight_sum_kernel<<<1, 1024, 0, s>>>(weights, static_cast<uint32_t>(rows), denominator);
        check_launch("cross_entropy_grad");
    }
    cross_entropy_grad_kernel<<<static_cast<uint32_t>(rows), kRowThreads, 0, s>>>(logits, labels, weights, g, denominator, out,
                                                                                  static_cast<uint32_t>(v), static_cast<uint32_t>(ld),
                                                                                  static_cast<uint32_t>(ld_out));
    check_launch("cross_entropy_grad");
}

}  // namespace k
}  // namespace msx
