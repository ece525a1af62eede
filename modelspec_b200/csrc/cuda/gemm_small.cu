// Small f32 products on the FMA units: what the tensor-core tiles of gemm_tf32.cu and gemm_tc.cu cost
// before their first and after their last product (barriers, tensor memory, a TMA round trip, the
// split, the drain: 5 to 6 us a launch) is more than the whole product here. Tolerance class; every
// term is a fused multiply-add in f32, so a sum is closer to the exact one than a split-TF32 one.
//
// Bound by latency: one trip to memory, the FMA chain, one trip back. A CTA computes one 32 x 32 tile of
// C (small tiles spread a small product over the most SMs) with 8 groups of 64 threads, 4 x 4 results
// each, that share out the k slabs (16 deep) among themselves and add their sums at the end through
// shared memory, in ascending group order: a group's slabs, not k, are what a CTA waits for, 1.2 us for
// each one after the first. A long k is shared out further among the 2 to 8 CTAs of a cluster, which add
// their tiles through distributed shared memory: no workspace and no second launch.
// 1,024 x 128 x 128 takes 3.6 us (5.5 on the tensor-core tiles it replaces), 385 x 99 x 99 3.5 (6.0);
// beyond about four tiles an SM shared-memory reads bound it (20 to 24 TFLOP/s) and the tensor cores win.
// Any size, storage form and alignment; rows whose four-element pieces lie on 16-byte boundaries are
// read 16 bytes at a time.
#include "common.cuh"
#include "kernels.cuh"

namespace msx {
namespace k {

namespace {

constexpr int KS = 16;                       // k slab
constexpr int BM = 32, BN = 32, TM = 4, G = 8;
constexpr int MAX_PRODUCTS = 4, MAX_JOBS = 24;

struct Problem {
    const float* a;
    const float* b;
    float* c;           // the result, or the split-k workspace [splits][m][n]
    const float* bias;  // or null
    uint32_t m, n, k, lda, ldb, ldc;
    uint32_t splits;    // of k into partial results
    uint32_t first_block;
    uint32_t a_vec, b_vec;
    float* beside;      // the epilogue's second matrix, of C's rows
};
template <int COUNT> struct Problems {
    uint32_t count;
    uint32_t cluster;  // CTAs that share one tile's k; splits are then 1
    Epilogue epilogue;
    Problem p[COUNT];
};

// Four consecutive elements at p + index, `valid` of which exist.
__device__ __forceinline__ float4 load_four(const float* __restrict__ p, uint64_t index, uint32_t valid, bool vec) {
    if (valid == 4 && vec) return load_global(reinterpret_cast<const float4*>(p + index));
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (valid > 0) v.x = load_global(p + index);
    if (valid > 1) v.y = load_global(p + index + 1);
    if (valid > 2) v.z = load_global(p + index + 2);
    if (valid > 3) v.w = load_global(p + index + 3);
    return v;
}
__device__ __forceinline__ uint32_t inside(uint32_t start, uint32_t limit) { return start >= limit ? 0u : (limit - start >= 4u ? 4u : limit - start); }

constexpr int GROUP = BM / TM * (BN / 4);  // threads of a group: TM x 4 results each
constexpr int THREADS = GROUP * G;
constexpr int A_PITCH = BM + 4, B_PITCH = BN + 4;
constexpr int SLAB = KS * (A_PITCH + B_PITCH);  // floats
constexpr int SHARED_BYTES = G * 2 * SLAB * 4;
static_assert(BM * BN / THREADS <= 2 && BM * BN % THREADS == 0, "a thread's elements");
constexpr int A_FOURS = BM * KS / 4 / GROUP, B_FOURS = BN * KS / 4 / GROUP;
static_assert(G * BM * BN <= G * 2 * SLAB, "the groups' sums take the slabs' place");

__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// ACT: with an epilogue (an instantiation of its own: its code in every product cost a transformer block's step 2.7 %).
template <bool A_T, bool B_T, int COUNT, bool ACT>
__global__ void __launch_bounds__(THREADS) matmul_small_kernel(const __grid_constant__ Problems<COUNT> problems) {
    after_producers();
    extern __shared__ __align__(16) float shared[];
    uint32_t which = 0;
    while (which + 1 < problems.count && problems.p[which + 1].first_block <= blockIdx.x) ++which;
    const Problem& p = problems.p[which];
    const float* __restrict__ const a = p.a;
    const float* __restrict__ const b = p.b;
    const uint32_t m = p.m, n = p.n, k = p.k, lda = p.lda, ldb = p.ldb;
    const bool a_vec = p.a_vec != 0, b_vec = p.b_vec != 0;
    const uint32_t cluster = problems.cluster;
    uint32_t at = blockIdx.x - p.first_block;
    const uint32_t rank = at % cluster;
    at /= cluster;
    const uint32_t across = (n + BN - 1) / BN, down = (m + BM - 1) / BM;
    const uint32_t n0 = (at % across) * BN;
    at /= across;
    const uint32_t m0 = (at % down) * BM, split = at / down;

    const uint32_t group = threadIdx.x / GROUP, t = threadIdx.x % GROUP;
    float* const mine = shared + group * 2 * SLAB;
    // Slabs are dealt out over the splits or the CTAs of the cluster and, within one, over the groups.
    const uint32_t slabs = (k + KS - 1) / KS, first = (split + rank) * G + group, stride = p.splits * cluster * G;
    float4 av[A_FOURS], bv[B_FOURS];
    auto fetch = [&](uint32_t slab) {
        const uint32_t k0 = slab * KS;
#pragma unroll
        for (int i = 0; i < A_FOURS; ++i) {
            const uint32_t q = t + i * GROUP;
            if (A_T) {  // stored [k, m]: four m of one k
                const uint32_t kk = k0 + q / (BM / 4), row = m0 + q % (BM / 4) * 4;
                av[i] = load_four(a, static_cast<uint64_t>(kk) * lda + row, kk < k ? inside(row, m) : 0u, a_vec);
            } else {    // stored [m, k]: four k of one row
                const uint32_t row = m0 + q / (KS / 4), kk = k0 + q % (KS / 4) * 4;
                av[i] = load_four(a, static_cast<uint64_t>(row) * lda + kk, row < m ? inside(kk, k) : 0u, a_vec);
            }
        }
#pragma unroll
        for (int i = 0; i < B_FOURS; ++i) {
            const uint32_t q = t + i * GROUP;
            if (B_T) {  // stored [n, k]
                const uint32_t col = n0 + q / (KS / 4), kk = k0 + q % (KS / 4) * 4;
                bv[i] = load_four(b, static_cast<uint64_t>(col) * ldb + kk, col < n ? inside(kk, k) : 0u, b_vec);
            } else {    // stored [k, n]
                const uint32_t kk = k0 + q / (BN / 4), col = n0 + q % (BN / 4) * 4;
                bv[i] = load_four(b, static_cast<uint64_t>(kk) * ldb + col, kk < k ? inside(col, n) : 0u, b_vec);
            }
        }
    };
    auto deposit = [&](float* to) {
        float* const as = to;
        float* const bs = to + KS * A_PITCH;
#pragma unroll
        for (int i = 0; i < A_FOURS; ++i) {
            const uint32_t q = t + i * GROUP;
            if (A_T) {
                *reinterpret_cast<float4*>(as + q / (BM / 4) * A_PITCH + q % (BM / 4) * 4) = av[i];
            } else {
                float* at_k = as + q % (KS / 4) * 4 * A_PITCH + q / (KS / 4);
                at_k[0] = av[i].x; at_k[A_PITCH] = av[i].y; at_k[2 * A_PITCH] = av[i].z; at_k[3 * A_PITCH] = av[i].w;
            }
        }
#pragma unroll
        for (int i = 0; i < B_FOURS; ++i) {
            const uint32_t q = t + i * GROUP;
            if (B_T) {
                float* at_k = bs + q % (KS / 4) * 4 * B_PITCH + q / (KS / 4);
                at_k[0] = bv[i].x; at_k[B_PITCH] = bv[i].y; at_k[2 * B_PITCH] = bv[i].z; at_k[3 * B_PITCH] = bv[i].w;
            } else {
                *reinterpret_cast<float4*>(bs + q / (BN / 4) * B_PITCH + q % (BN / 4) * 4) = bv[i];
            }
        }
    };
    auto group_barrier = [&] { asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(GROUP) : "memory"); };

    // The arguments of the activations whose gradient this thread's elements take: fetched with the first slabs (behind
    // the sums they would be a trip to memory of their own).
    constexpr uint32_t OWN = BM * BN / THREADS;
    const Epilogue epilogue = ACT ? problems.epilogue : Epilogue::None;
    float argument[ACT ? OWN : 1];
    if constexpr (ACT) {
        if (epilogue == Epilogue::GeluGrad || epilogue == Epilogue::ReluGrad) {
            const uint32_t share = BM * BN / cluster, end = (rank + 1) * share;
#pragma unroll
            for (uint32_t i = 0; i < OWN; ++i) {
                const uint32_t e = rank * share + threadIdx.x + i * THREADS, row = m0 + e / BN, col = n0 + e % BN;
                argument[i] = e < end && row < m && col < n ? load_global(p.beside + static_cast<uint64_t>(row) * p.ldc + col) : 0.0f;
            }
        }
    }

    const uint32_t tm = t / (BN / 4) * TM, tn = t % (BN / 4) * 4;
    float acc[TM][4];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    if (first < slabs) fetch(first);
    uint32_t half = 0;
    for (uint32_t slab = first; slab < slabs; slab += stride, half ^= 1u) {
        float* const to = mine + half * SLAB;
        deposit(to);
        group_barrier();  // (the slab before last, in this half, was read before the barrier before this one)
        if (slab + stride < slabs) fetch(slab + stride);
        const float* const as = to + tm;
        const float* const bs = to + KS * A_PITCH + tn;
#pragma unroll
        for (int kk = 0; kk < KS; ++kk) {
            float av4[TM];
#pragma unroll
            for (int i = 0; i < TM; i += 4) *reinterpret_cast<float4*>(av4 + i) = *reinterpret_cast<const float4*>(as + kk * A_PITCH + i);
            const float4 bv4 = *reinterpret_cast<const float4*>(bs + kk * B_PITCH);
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                acc[i][0] = fmaf(av4[i], bv4.x, acc[i][0]);
                acc[i][1] = fmaf(av4[i], bv4.y, acc[i][1]);
                acc[i][2] = fmaf(av4[i], bv4.z, acc[i][2]);
                acc[i][3] = fmaf(av4[i], bv4.w, acc[i][3]);
            }
        }
    }
    __syncthreads();
    float* const sums = shared + group * BM * BN;
#pragma unroll
    for (int i = 0; i < TM; ++i) *reinterpret_cast<float4*>(sums + (tm + i) * BN + tn) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    __syncthreads();
    float* __restrict__ const out = p.c + static_cast<uint64_t>(split) * m * p.ldc;
    const float* __restrict__ const bias = p.bias;
    auto sum_of = [&](uint32_t e) {
        float v = shared[e];
#pragma unroll
        for (int g = 1; g < G; ++g) v += shared[g * BM * BN + e];
        return v;
    };
    // Element e of the tile, the thread's i-th.
    auto store = [&](uint32_t e, uint32_t i, float v) {
        const uint32_t row = m0 + e / BN, col = n0 + e % BN;
        if (row >= m || col >= n) return;
        const uint64_t at = static_cast<uint64_t>(row) * p.ldc + col;
        v = bias ? v + load_global(bias + col) : v;
        if constexpr (ACT) {
            const float x = argument[OWN == 2 ? i & 1u : i];
            if (epilogue == Epilogue::GeluGrad) v = gelu_grad_value(x, v);
            else if (epilogue == Epilogue::ReluGrad) v = relu_grad_value(x, v);
            else p.beside[at] = epilogue == Epilogue::Gelu ? gelu_value(v) : relu_value(v);
        }
        out[at] = v;
    };
    if (cluster == 1) {
#pragma unroll
        for (uint32_t i = 0; i < OWN; ++i) store(threadIdx.x + i * THREADS, i, sum_of(threadIdx.x + i * THREADS));
        return;
    }
    // Each CTA of the cluster adds its groups, then its share of the tile over the CTAs in ascending order.
    float total[BM * BN / THREADS];
#pragma unroll
    for (int i = 0; i < BM * BN / THREADS; ++i) total[i] = sum_of(threadIdx.x + i * THREADS);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < BM * BN / THREADS; ++i) shared[threadIdx.x + i * THREADS] = total[i];
    cluster_barrier();
    const uint32_t share = BM * BN / cluster;
    uint32_t i = 0;
    for (uint32_t e = rank * share + threadIdx.x; e < (rank + 1) * share; e += THREADS, ++i) {
        float v = 0.f;
        for (uint32_t r = 0; r < cluster; ++r) {
            float term;
            asm volatile("{\n\t.reg .b32 far;\n\tmapa.shared::cluster.u32 far, %1, %2;\n\tld.shared::cluster.f32 %0, [far];\n\t}"
                         : "=f"(term) : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(shared + e))), "r"(r) : "memory");
            v = r == 0 ? term : v + term;
        }
        store(e, i, v);
    }
    cluster_barrier();  // no CTA goes away while another reads its tile
}

template <bool A_T, bool B_T, bool ACT, int COUNT> void launch(cudaStream_t s, const Problems<COUNT>& problems, uint32_t blocks) {
    auto kernel = matmul_small_kernel<A_T, B_T, COUNT, ACT>;
    static std::atomic<int> configured_device{-1};
    set_shared_memory(kernel, SHARED_BYTES, configured_device);
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(blocks);
    config.blockDim = dim3(THREADS);
    config.dynamicSmemBytes = SHARED_BYTES;
    config.stream = s;
    cudaLaunchAttribute cluster = {};
    cluster.id = cudaLaunchAttributeClusterDimension;
    cluster.val.clusterDim.x = problems.cluster;
    cluster.val.clusterDim.y = cluster.val.clusterDim.z = 1;
    if (problems.cluster > 1) {
        config.attrs = &cluster;
        config.numAttrs = 1;
    }
    check(cudaLaunchKernelEx(&config, kernel, problems), "matmul_small");
    starts_in_order(s);  // (its small blocks would gather on the few SMs that are idle early)
}
template <int COUNT> void launch_form(cudaStream_t s, bool a_t, bool b_t, const Problems<COUNT>& problems, uint32_t blocks) {
    if constexpr (COUNT == MAX_PRODUCTS) {
        if (problems.epilogue != Epilogue::None) {
            if (a_t && b_t) launch<true, true, true>(s, problems, blocks);
            else if (a_t) launch<true, false, true>(s, problems, blocks);
            else if (b_t) launch<false, true, true>(s, problems, blocks);
            else launch<false, false, true>(s, problems, blocks);
            return;
        }
    }
    if (a_t && b_t) launch<true, true, false>(s, problems, blocks);
    else if (a_t) launch<true, false, false>(s, problems, blocks);
    else if (b_t) launch<false, true, false>(s, problems, blocks);
    else launch<false, false, false>(s, problems, blocks);
}

bool aligned16(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

Problem problem_of(const float* a, const float* b, float* c, const float* bias, uint64_t m, uint64_t n, uint64_t k, uint64_t lda, uint64_t ldb, uint64_t ldc,
                   uint32_t splits, uint32_t first_block) {
    Problem p = {a, b, c, bias, static_cast<uint32_t>(m), static_cast<uint32_t>(n), static_cast<uint32_t>(k), static_cast<uint32_t>(lda),
                 static_cast<uint32_t>(ldb), static_cast<uint32_t>(ldc), splits, first_block, 0, 0, nullptr};
    p.a_vec = aligned16(a) && lda % 4 == 0;
    p.b_vec = aligned16(b) && ldb % 4 == 0;
    return p;
}
uint32_t blocks_of(uint64_t m, uint64_t n) { return static_cast<uint32_t>(((m + BM - 1) / BM) * ((n + BN - 1) / BN)); }

}  // namespace

void matmul_small(cudaStream_t s, const MatmulTcPlan& p, const MatmulOperands* products, uint32_t count, bool a_t, bool b_t, uint64_t m, uint64_t n, uint64_t k,
                  MatmulPitches pitches, Epilogue epilogue, float* beside) {
    Problems<MAX_PRODUCTS> problems = {};
    problems.cluster = p.cluster;
    problems.epilogue = epilogue;
    uint32_t blocks = 0;
    for (uint32_t g = 0; g < count; ++g) {
        problems.p[problems.count++] = problem_of(products[g].a, products[g].b, products[g].c, products[g].bias, m, n, k, pitches.a ? pitches.a : (a_t ? m : k),
                                                  pitches.b ? pitches.b : (b_t ? k : n), pitches.c ? pitches.c : n, 1, blocks);
        problems.p[g].beside = beside;
        blocks += blocks_of(m, n) * p.cluster;
    }
    launch_form(s, a_t, b_t, problems, blocks);
}

void matmul_small_jobs(cudaStream_t s, const MatmulJob* jobs, uint32_t count, bool a_t, bool b_t) {
    Problems<MAX_JOBS> problems = {};
    problems.cluster = 1;
    uint32_t blocks = 0;
    for (uint32_t j = 0; j < count; ++j) {
        const MatmulJob& job = jobs[j];
        const uint32_t splits = matmul_tc_job_plan(job.m, job.n, job.k).splits;
        problems.p[problems.count++] = problem_of(job.a, job.b, splits > 1 ? job.workspace : job.c, nullptr, job.m, job.n, job.k, a_t ? job.m : job.k,
                                                  b_t ? job.k : job.n, job.n, splits, blocks);
        blocks += blocks_of(job.m, job.n) * splits;
    }
    launch_form(s, a_t, b_t, problems, blocks);
}

}  // namespace k
}  // namespace msx
