// Attention and its gradients on the tensor cores: each contraction is one batched tcgen05
// matmul over every (sequence, head) (gemm_tf32.cu, or gemm_tc.cu for widths off 16 bytes; 3xTF32), with two
// row kernels between them.
//
//   forward   S = Q_h K_h^T            -> P = masked softmax(S / sqrt(d))   -> O_h = P V_h
//   backward  P as the forward left it (or computed again as above);  dP = G_h V_h^T;  dS = scale P (dP - rowsum(P dP));
//             dV_h = P^T G_h;  dQ_h = dS K_h;  dK_h = dS^T Q_h
//
// Heads are addressed in place (row pitch H, head offset a * d), so nothing is gathered or
// transposed. The score matrices [B, A, L, S] live in scratch between the launches: 4 MB per
// layer at 32 x 2 heads x 128 x 128, which stays in the 126 MB L2 between producer and consumer.
// A masked key gets probability 0, so it adds exact zeros to every sum and its dK and dV rows
// are +0, as in the reference (crates/modelspec-runtime/src/cpu/interpreter.rs:1035-1119).
// Tolerance class: 3xTF32 products, warp-tree row sums, device expf.
#include "common.cuh"
#include "kernels.cuh"

namespace msx {
namespace k {

namespace {

// One warp per score row, the row in registers (ITEMS x 32 keys or fewer): a score is read once and a
// probability written once, with every load of a row in flight together. Rows on 16 bytes (V = 4) are read
// and written four keys a lane.
constexpr uint32_t ROW_BLOCK_WARPS = 8;

// p = softmax over the unmasked keys of acc * scale, in place.
template <int ITEMS, int V>
__global__ void __launch_bounds__(32 * ROW_BLOCK_WARPS) masked_softmax_kernel(float* scores, const float* mask, uint32_t rows,
                                                                              uint32_t rows_per_sequence, uint32_t s, float scale) {
    after_producers();
    const uint32_t row = blockIdx.x * ROW_BLOCK_WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (row >= rows) return;
    float* p = scores + static_cast<uint64_t>(row) * s;
    const float* m = mask + static_cast<uint64_t>(row / rows_per_sequence) * s;
    auto key_of = [lane](int i) { return static_cast<uint32_t>(i / V * 32 * V + i % V) + lane * V; };  // of item i
    float x[ITEMS];
    uint32_t counts = 0;
#pragma unroll
    for (int i = 0; i < ITEMS; i += V) {
        const uint32_t j = min(key_of(i), s - V);
        float4 mask4;
        if constexpr (V == 4) {
            const float4 x4 = *reinterpret_cast<const float4*>(p + j);
            x[i] = x4.x; x[i + 1] = x4.y; x[i + 2] = x4.z; x[i + 3] = x4.w;
            mask4 = make_float4(load_global(m + j), load_global(m + j + 1), load_global(m + j + 2), load_global(m + j + 3));
            if (key_of(i) < s) counts |= ((mask4.x != 0.0f ? 1u : 0u) | (mask4.y != 0.0f ? 2u : 0u) | (mask4.z != 0.0f ? 4u : 0u) | (mask4.w != 0.0f ? 8u : 0u)) << i;
        } else {
            x[i] = p[j];
            counts |= (key_of(i) < s && load_global(m + j) != 0.0f ? 1u : 0u) << i;
        }
    }
    float best = -INFINITY;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i)
        if ((counts >> i) & 1u) best = fmaxf(best, x[i] * scale);
    best = warp_max(best);
    float total = 0.0f;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        x[i] = (counts >> i) & 1u ? expf(x[i] * scale - best) : 0.0f;
        total += x[i];
    }
    total = warp_sum(total);
    // x / total, rounded once: with the rounded reciprocal, the quotient corrected by its exact remainder is the
    // nearest one (Markstein, IBM J. Res. Dev. 34, 1990, theorem 8.2; total is between 1 and the number of keys. A
    // quotient too small for its remainder to be exact is off by less than the smallest normal number).
    const float inverse = 1.0f / total;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const float first = x[i] * inverse;
        x[i] = fmaf(fmaf(-first, total, x[i]), inverse, first);
    }
#pragma unroll
    for (int i = 0; i < ITEMS; i += V) {
        if (key_of(i) >= s) continue;
        if constexpr (V == 4) *reinterpret_cast<float4*>(p + key_of(i)) = make_float4(x[i], x[i + 1], x[i + 2], x[i + 3]);
        else p[key_of(i)] = x[i];
    }
}

// dS = scale * P * (dP - sum_j P dP), written over dP.
template <int ITEMS>
__global__ void __launch_bounds__(32 * ROW_BLOCK_WARPS) score_grad_kernel(const float* p, float* dp, uint32_t rows, uint32_t s,
                                                                          float scale) {
    after_producers();
    const uint32_t row = blockIdx.x * ROW_BLOCK_WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (row >= rows) return;
    const float* pr = p + static_cast<uint64_t>(row) * s;
    float* dr = dp + static_cast<uint64_t>(row) * s;
    float x[ITEMS], d[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const uint32_t j = min(lane + 32 * i, s - 1);
        x[i] = load_global(pr + j);
        d[i] = dr[j];
    }
    float dot = 0.0f;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i)
        if (lane + 32 * i < s) dot = fmaf(x[i], d[i], dot);
    dot = warp_sum(dot);
#pragma unroll
    for (int i = 0; i < ITEMS; ++i)
        if (lane + 32 * i < s) dr[lane + 32 * i] = x[i] * (d[i] - dot) * scale;
}

struct Heads {
    uint32_t b, l, s, a, d, h;
    float scale;
    BatchedOperand q(const float* x) const { return {x, h, static_cast<uint64_t>(l) * h, d, false}; }   // [L, d] of a head, row pitch H
    BatchedOperand kv(const float* x) const { return {x, h, static_cast<uint64_t>(s) * h, d, false}; }  // [S, d]
    BatchedOperand scores(const float* x) const { return {x, s, static_cast<uint64_t>(a) * l * s, static_cast<uint64_t>(l) * s, false}; }
    uint32_t rows() const { return b * a * l; }
};

Heads heads_of(AttentionShape sh) {
    Heads hd;
    hd.b = sh.batch; hd.l = sh.q_len; hd.s = sh.k_len; hd.a = sh.heads; hd.d = sh.head_dim; hd.h = sh.heads * sh.head_dim;
    hd.scale = 1.0f / sqrtf(static_cast<float>(sh.head_dim));
    return hd;
}

BatchedOperand transposed(BatchedOperand o) {
    o.transposed = true;
    return o;
}

void product(cudaStream_t s, const BatchedProduct& one, uint64_t m, uint64_t n, uint64_t k, const Heads& hd, uint32_t* status) {
    matmul_tc_batched(s, &one, 1, m, n, k, hd.b, hd.a, status);
}

void probabilities(cudaStream_t s, const float* q, const float* k, const float* mask, float* p, const Heads& hd, uint32_t* status) {
    // S[i, j] = sum_c q[i, c] k[j, c]: B is the keys stored [n, k].
    product(s, {hd.q(q), transposed(hd.kv(k)), hd.scores(p)}, hd.l, hd.s, hd.d, hd, status);
    uint32_t rows = hd.rows();
    const bool wide = hd.s % 4 == 0 && reinterpret_cast<uintptr_t>(p) % 16 == 0;
    const dim3 grid((rows + ROW_BLOCK_WARPS - 1) / ROW_BLOCK_WARPS), block(32 * ROW_BLOCK_WARPS);
    if (wide && hd.s <= 128) masked_softmax_kernel<4, 4><<<grid, block, 0, s>>>(p, mask, rows, hd.a * hd.l, hd.s, hd.scale);
    else if (wide && hd.s <= 256) masked_softmax_kernel<8, 4><<<grid, block, 0, s>>>(p, mask, rows, hd.a * hd.l, hd.s, hd.scale);
    else if (wide) masked_softmax_kernel<16, 4><<<grid, block, 0, s>>>(p, mask, rows, hd.a * hd.l, hd.s, hd.scale);
    else if (hd.s <= 64) masked_softmax_kernel<2, 1><<<grid, block, 0, s>>>(p, mask, rows, hd.a * hd.l, hd.s, hd.scale);
    else if (hd.s <= 128) masked_softmax_kernel<4, 1><<<grid, block, 0, s>>>(p, mask, rows, hd.a * hd.l, hd.s, hd.scale);
    else if (hd.s <= 256) masked_softmax_kernel<8, 1><<<grid, block, 0, s>>>(p, mask, rows, hd.a * hd.l, hd.s, hd.scale);
    else masked_softmax_kernel<16, 1><<<grid, block, 0, s>>>(p, mask, rows, hd.a * hd.l, hd.s, hd.scale);
    check_launch("attention masked_softmax");
}

}  // namespace

uint64_t attention_tc_scratch_floats(AttentionShape sh) {
    return static_cast<uint64_t>(sh.batch) * sh.heads * sh.q_len * sh.k_len;
}

void attention_tc_forward(cudaStream_t s, const float* q, const float* k, const float* v, const float* mask, float* out,
                          float* p, AttentionShape sh, uint32_t* status) {
    if (sh.batch == 0 || sh.q_len == 0) return;
    Heads hd = heads_of(sh);
    probabilities(s, q, k, mask, p, hd, status);
    // O[i, c] = sum_j P[i, j] v[j, c]
    product(s, {hd.scores(p), hd.kv(v), hd.q(out)}, hd.l, hd.d, hd.s, hd, status);
}

void attention_tc_backward(cudaStream_t s, const float* q, const float* k, const float* v, const float* mask, const float* g,
                           float* dq, float* dk, float* dv, float* p, float* dp, AttentionShape sh, uint32_t* status, bool p_ready) {
    if (sh.batch == 0 || sh.q_len == 0) return;
    Heads hd = heads_of(sh);
    if (!p_ready) probabilities(s, q, k, mask, p, hd, status);
    // dV[j, c] = sum_i P[i, j] g[i, c] and dK[j, c] = sum_i dS[i, j] q[i, c], one launch: A is P or dS
    // stored [k, m].
    auto key_gradients = [&] {
        BatchedProduct both[2];
        uint32_t count = 0;
        if (dv) both[count++] = {transposed(hd.scores(p)), hd.q(g), hd.kv(dv)};
        if (dk) both[count++] = {transposed(hd.scores(dp)), hd.q(q), hd.kv(dk)};
        if (count) matmul_tc_batched(s, both, count, hd.s, hd.d, hd.l, hd.b, hd.a, status);
    };
    if (!dq && !dk) {
        key_gradients();
        return;
    }
    // dP[i, j] = sum_c g[i, c] v[j, c]
    product(s, {hd.q(g), transposed(hd.kv(v)), hd.scores(dp)}, hd.l, hd.s, hd.d, hd, status);
    uint32_t rows = hd.rows();
    const dim3 grid((rows + ROW_BLOCK_WARPS - 1) / ROW_BLOCK_WARPS), block(32 * ROW_BLOCK_WARPS);
    if (hd.s <= 64) score_grad_kernel<2><<<grid, block, 0, s>>>(p, dp, rows, hd.s, hd.scale);
    else if (hd.s <= 128) score_grad_kernel<4><<<grid, block, 0, s>>>(p, dp, rows, hd.s, hd.scale);
    else if (hd.s <= 256) score_grad_kernel<8><<<grid, block, 0, s>>>(p, dp, rows, hd.s, hd.scale);
    else score_grad_kernel<16><<<grid, block, 0, s>>>(p, dp, rows, hd.s, hd.scale);
    check_launch("attention score_grad");
    key_gradients();
    // dQ[i, c] = sum_j dS[i, j] k[j, c]
    if (dq) product(s, {hd.scores(dp), hd.kv(k), hd.q(dq)}, hd.l, hd.d, hd.s, hd, status);
}

// ---- mixed precision ----------------------------------------------------------------------------
// The same launches for a plan that stores activations as bf16: the products run on the bf16
// kernel (gemm_bf16.cu), scores and their adjoints are written in f32 (a scratch matrix that only
// the row kernel after it reads), and the row kernels store the probabilities and the score
// gradients as bf16 for the products that follow.

namespace {

// One warp per score row: p = softmax over the unmasked keys of scores * scale, stored as bf16.
__global__ void masked_softmax_half_kernel(const float* scores, const float* mask, bf16* p,
                                           uint32_t rows, uint32_t rows_per_sequence, uint32_t s, float scale) {
    after_producers();
    uint32_t row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= rows) return;
    int lane = threadIdx.x & 31;
    const float* x = scores + static_cast<uint64_t>(row) * s;
    bf16* out = p + static_cast<uint64_t>(row) * s;
    const float* m = mask + static_cast<uint64_t>(row / rows_per_sequence) * s;
    float best = -INFINITY;
    for (uint32_t j = lane; j < s; j += 32)
        if (m[j] != 0.0f) best = fmaxf(best, x[j] * scale);
    best = warp_max(best);
    float total = 0.0f;
    for (uint32_t j = lane; j < s; j += 32) total += m[j] != 0.0f ? expf(x[j] * scale - best) : 0.0f;
    total = warp_sum(total);
    for (uint32_t j = lane; j < s; j += 32) out[j] = __float2bfloat16_rn(m[j] != 0.0f ? expf(x[j] * scale - best) / total : 0.0f);
}

// dS = scale * P * (dP - sum_j P dP), stored as bf16.
__global__ void score_grad_half_kernel(const bf16* p, const float* dp, bf16* ds, uint32_t rows,
                                       uint32_t s, float scale) {
    after_producers();
    uint32_t row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= rows) return;
    int lane = threadIdx.x & 31;
    const bf16* pr = p + static_cast<uint64_t>(row) * s;
    const float* dr = dp + static_cast<uint64_t>(row) * s;
    bf16* out = ds + static_cast<uint64_t>(row) * s;
    float dot = 0.0f;
    for (uint32_t j = lane; j < s; j += 32) dot = fmaf(__bfloat162float(pr[j]), dr[j], dot);
    dot = warp_sum(dot);
    for (uint32_t j = lane; j < s; j += 32) out[j] = __float2bfloat16_rn(__bfloat162float(pr[j]) * (dr[j] - dot) * scale);
}

struct HalfHeads {
    Heads hd;
    HalfMatrix q(const void* x, bool transposed = false) const { return {x, hd.h, static_cast<uint64_t>(hd.l) * hd.h, hd.d, transposed}; }
    HalfMatrix kv(const void* x, bool transposed = false) const { return {x, hd.h, static_cast<uint64_t>(hd.s) * hd.h, hd.d, transposed}; }
    HalfMatrix scores(const void* x, bool transposed = false) const {
        return {x, hd.s, static_cast<uint64_t>(hd.a) * hd.l * hd.s, static_cast<uint64_t>(hd.l) * hd.s, transposed};
    }
    HalfResult to_q(void* x) const { return {x, true, hd.h, static_cast<uint64_t>(hd.l) * hd.h, hd.d}; }
    HalfResult to_kv(void* x) const { return {x, true, hd.h, static_cast<uint64_t>(hd.s) * hd.h, hd.d}; }
    HalfResult to_scores(float* x) const { return {x, false, hd.s, static_cast<uint64_t>(hd.a) * hd.l * hd.s, static_cast<uint64_t>(hd.l) * hd.s}; }
};

void half_probabilities(cudaStream_t s, const void* q, const void* k, const float* mask, void* p, float* scores, const HalfHeads& hh,
                        uint32_t* status) {
    const Heads& hd = hh.hd;
    // S[i, j] = sum_c q[i, c] k[j, c]: B is the keys stored [n, k].
    matmul_bf16(s, hh.q(q), hh.kv(k, true), hh.to_scores(scores), hd.l, hd.s, hd.d, hd.b, hd.a, nullptr, nullptr, status);
    const uint32_t rows = hd.rows();
    masked_softmax_half_kernel<<<(rows + 7) / 8, 256, 0, s>>>(scores, mask, static_cast<bf16*>(p), rows, hd.a * hd.l, hd.s, hd.scale);
    check_launch("attention masked_softmax");
}

}  // namespace

void attention_bf16_forward(cudaStream_t s, const void* q, const void* k, const void* v, const float* mask, void* out, void* p,
                            float* scores, AttentionShape sh, uint32_t* status) {
    if (sh.batch == 0 || sh.q_len == 0) return;
    const HalfHeads hh = {heads_of(sh)};
    const Heads& hd = hh.hd;
    half_probabilities(s, q, k, mask, p, scores, hh, status);
    // O[i, c] = sum_j P[i, j] v[j, c]
    matmul_bf16(s, hh.scores(p), hh.kv(v), hh.to_q(out), hd.l, hd.d, hd.s, hd.b, hd.a, nullptr, nullptr, status);
}

void attention_bf16_backward(cudaStream_t s, const void* q, const void* k, const void* v, const float* mask, const void* g, void* dq,
                             void* dk, void* dv, void* p, void* ds, float* scores, AttentionShape sh, uint32_t* status, bool p_ready) {
    if (sh.batch == 0 || sh.q_len == 0) return;
    const HalfHeads hh = {heads_of(sh)};
    const Heads& hd = hh.hd;
    if (!p_ready) half_probabilities(s, q, k, mask, p, scores, hh, status);
    // dV[j, c] = sum_i P[i, j] g[i, c]: A is P stored [k, m].
    if (dv) matmul_bf16(s, hh.scores(p, true), hh.q(g), hh.to_kv(dv), hd.s, hd.d, hd.l, hd.b, hd.a, nullptr, nullptr, status);
    if (!dq && !dk) return;
    // dP[i, j] = sum_c g[i, c] v[j, c], in f32.
    matmul_bf16(s, hh.q(g), hh.kv(v, true), hh.to_scores(scores), hd.l, hd.s, hd.d, hd.b, hd.a, nullptr, nullptr, status);
    const uint32_t rows = hd.rows();
    score_grad_half_kernel<<<(rows + 7) / 8, 256, 0, s>>>(static_cast<const bf16*>(p), scores, static_cast<bf16*>(ds), rows, hd.s, hd.scale);
    check_launch("attention score_grad");
    // dQ[i, c] = sum_j dS[i, j] k[j, c];  dK[j, c] = sum_i dS[i, j] q[i, c]
    if (dq) matmul_bf16(s, hh.scores(ds), hh.kv(k), hh.to_q(dq), hd.l, hd.d, hd.s, hd.b, hd.a, nullptr, nullptr, status);
    if (dk) matmul_bf16(s, hh.scores(ds, true), hh.q(q), hh.to_kv(dk), hd.s, hd.d, hd.l, hd.b, hd.a, nullptr, nullptr, status);
}

}  // namespace k
}  // namespace msx
