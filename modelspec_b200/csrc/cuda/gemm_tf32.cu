// f32 products on the 5th-generation tensor cores for operands TMA can address (bases on 16 bytes,
// row pitches multiples of 16 bytes): tcgen05.mma kind::tf32 on split operands, accumulators in tensor
// memory, tolerance class.
//
// Each f32 operand x is the sum of hi = its top 11 significant bits and lo = x - hi (exact; the tensor
// core keeps 11 significant bits of it), and a product is summed as hi*hi + hi*lo + lo*hi in f32
// accumulators; lo*lo, below 2^-20 of a product, is left out. A tf32 operand is read as the upper 19
// bits of its 32-bit word, so the raw f32 block, as TMA leaves it in shared memory, is the hi operand
// itself, and only the lo block has to be made: the same bytes at the same offsets of a second tile.
//
// What bounds it. Per 8-deep k slice the three MMAs of 128 x N x 8 read 128 + N rows of 32 bytes each
// out of shared memory, 8 KB at N = 128: 64 of the 67 cycles the MMA takes at the tf32 rate, which
// leaves no bandwidth for loading and splitting. (The tile that split both halves into tiles of
// their own took 1,460 to 1,800 cycles a 128 x 128 x 32 block, 140 to 178 TFLOP/s at BERT-base's
// shapes.) Two CTAs of a cluster therefore pair up for large products: one tcgen05.mma of 256 x 256 x 8
// (cta_group::2) reads from each SM its own 128 rows of A and 128 of the 256 columns of B, half the
// bytes per product, and every operand crosses the L2 half as often. Small products, where what counts
// is how soon the last CTA is done, take 128-row tiles 128, 64 or 32 wide in CTAs of their own.
//
// A CTA is persistent and walks the launch's units (tiles x k splits x products):
//   lo warps     two to a stage: wait for its raw block, write the lo block beside it, tell the MMA warp;
//   MMA warp     (of the pair's first CTA) issues the MMAs into one of two accumulators;
//   TMA warp     loads all the CTA's k blocks as one sequence;
//   drain warps  empty the other accumulator: 32 lanes x 32 columns at a time into a slab of their own,
//                which a TMA store writes to C.
// The tensor core's f32 accumulation truncates: a sum of N MMAs comes out low by about N 2^-24 of its
// terms' magnitude (3 10^-4 of a sum of 16,384 positive products). So the sums of a tile leave tensor
// memory every 24 k blocks and go on in C, the first by a TMA store and the later ones by TMA's f32
// reduction in the L2 (each after the one before it has landed, so in one order), and on the tiles of
// one CTA the two cross products, whose terms are 2^-11 of the others', have an accumulator of their own.
//
// Stages are handed over by mbarriers; every wait is bounded and, when it runs out, raises bit 1 of the
// status word, makes every role leave its loop, frees the tensor memory and returns.
#include <atomic>

#include "common.cuh"
#include "kernels.cuh"
#include "tcgen05.cuh"

namespace msx {
namespace k {

namespace {

constexpr int BK = 32;
constexpr int GROUP_THREADS = 64;  // of the warps that make one stage's lo blocks
constexpr int MAX_PRODUCTS = 4, MAX_JOBS = 24;
// k blocks summed in tensor memory before the sum goes to C (768 deep: 6 10^-6 of a product's norm on the
// paired tiles, however deep the product). The sums into C cost a weight gradient 768 x 3,072 x 16,384
// nothing (309 us; 312 with 64 blocks, 322 with 256) and 3,072 x 768 x 16,384 up to 5 % (328 us; 321 and
// 308), for errors of 6 10^-6 (1.5 10^-5 and 5.9 10^-5) of their norm.
constexpr uint32_t SEGMENT = 24;

template <int CG, int BN> struct Tile {
    static constexpr int BN_CTA = BN / CG;  // columns of B a CTA holds
    static constexpr uint32_t A_BYTES = 128 * BK * 4, B_BYTES = BN_CTA * BK * 4;
    static constexpr uint32_t RAW_BYTES = A_BYTES + B_BYTES, STAGE_BYTES = 2 * RAW_BYTES;  // raw A, lo A, raw B, lo B
    static constexpr int STAGES = BN_CTA == 128 ? 3 : (BN_CTA == 64 ? 4 : 5);
    static constexpr int DRAIN_WARPS = BN == 32 ? 4 : 8;          // one or two per lane quarter
    static constexpr int CHUNKS = BN / 32 / (DRAIN_WARPS / 4);    // of 32 columns, per drain warp and tile
    static constexpr int LO_WARPS = STAGES * GROUP_THREADS / 32, MMA_WARP = LO_WARPS, TMA_WARP = LO_WARPS + 1;
    static constexpr int FIRST_DRAIN_WARP = (LO_WARPS + 2 + 3) / 4 * 4;  // drain warp w reads lane quarter w % 4
    static constexpr int THREADS = 32 * (FIRST_DRAIN_WARP + DRAIN_WARPS);
    static constexpr uint32_t SLAB_BYTES = 32 * 128;
    static constexpr uint32_t BIAS_BYTES = 2 * BN * 4;
    static constexpr uint32_t TOTAL = STAGES * STAGE_BYTES + DRAIN_WARPS * SLAB_BYTES + BIAS_BYTES + 256 /* barriers */;
    // A tile of one CTA multiplies raw A by raw and lo B together (they lie side by side, 2 BN columns of
    // one operand), lo A by raw B into the lo half, and the drain adds the two halves: two MMAs a k slice
    // instead of three, where an MMA takes its 90 cycles however narrow it is.
    static constexpr bool STACKED = CG == 1;
    static constexpr uint32_t ACC_COLUMNS = STACKED ? 2 * BN : BN, TMEM_COLUMNS = 2 * ACC_COLUMNS;
    static_assert(TOTAL <= 232448, "shared memory of a CTA");
};

struct Job {
    float* c;  // the result, or the job's split-k workspace
    uint32_t m, n, kblocks, first_unit;
    tc::Divisor splits;
    tc::TileWalk walk;
};
struct Args {
    uint32_t units = 0, m = 0, n = 0, ldc = 0;
    tc::TileWalk walk;
    tc::Divisor splits;
    uint32_t kblocks = 0;                       // of one product
    uint32_t chain = 1;                         // > 1: that many products are summed into one result
    tc::Divisor batch{1}, batch_inner{1};       // matrices of each product, (outer, inner) of them (k unsplit)
    uint32_t c_tma = 1, c_vec = 1, c_padded = 0;  // C by TMA stores; else 16-byte stores; padding between n and ldc may be overwritten
    float* c[MAX_PRODUCTS] = {};                // C, or the split-k workspace [splits][m][n]
    const float* bias[MAX_PRODUCTS] = {};       // null for none
    uint32_t* status = nullptr;
};
struct Maps {
    CUtensorMap a[MAX_PRODUCTS], b[MAX_PRODUCTS], c[MAX_PRODUCTS];
};
// Products of different shapes and one storage form in one launch.
struct JobArgs : Args {
    uint32_t job_count = 0;
    Job jobs[MAX_JOBS] = {};
};
struct JobMaps {
    CUtensorMap a[MAX_JOBS], b[MAX_JOBS], c[MAX_JOBS];
};

// Unit `u` of a launch: its tile, then the split, the matrix of a batch, and the product or job.
struct Unit {
    uint32_t m0, n0, split, splits, product, kblocks, z_inner, z_outer;
    uint32_t m, n, ldc;
    float* c;
    const float* bias;
};
__device__ __forceinline__ Unit unit_of(const Args& args, uint32_t u) {
    Unit w;
    w.m = args.m; w.n = args.n; w.ldc = args.ldc; w.splits = args.splits.d;
    u = args.walk.take(u, &w.m0, &w.n0);
    const uint32_t after_split = args.splits.quotient(u);
    w.split = u - after_split * args.splits.d;
    w.product = args.batch.quotient(after_split);
    const uint32_t z = after_split - w.product * args.batch.d;
    w.z_outer = args.batch_inner.quotient(z);
    w.z_inner = z - w.z_outer * args.batch_inner.d;
    w.c = args.c[w.product];
    w.bias = args.bias[w.product];
    w.kblocks = args.chain > 1 ? args.kblocks * args.chain : args.splits.quotient(args.kblocks - w.split + w.splits - 1);
    return w;
}
__device__ __forceinline__ Unit unit_of(const JobArgs& args, uint32_t u) {
    uint32_t j = 0;
    while (j + 1 < args.job_count && args.jobs[j + 1].first_unit <= u) ++j;
    const Job& job = args.jobs[j];
    Unit w;
    w.m = job.m; w.n = w.ldc = job.n; w.splits = job.splits.d;
    w.split = job.walk.take(u - job.first_unit, &w.m0, &w.n0);
    w.product = j;
    w.z_inner = w.z_outer = 0;
    w.c = job.c;
    w.bias = nullptr;
    w.kblocks = job.splits.quotient(job.kblocks - w.split + w.splits - 1);
    return w;
}

// `reuse`: 1 keeps the A operand in the tensor core's collector buffer for the next MMA, 2 takes it from
// there (a sixth of the shared-memory reads of a k slice, 1 % of a large product).
template <int CG, int REUSE> __device__ __forceinline__ void mma_tf32(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
#define MSX_MMA(group, collector)                                                                                                          \
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::" group ".kind::tf32" collector " [%0], %1, %2, %3, p;\n\t}" \
                 ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory")
    if constexpr (CG == 1) MSX_MMA("1", "");
    else if constexpr (REUSE == 1) MSX_MMA("2", ".collector::a::fill");
    else if constexpr (REUSE == 2) MSX_MMA("2", ".collector::a::lastuse");
    else MSX_MMA("2", "");
#undef MSX_MMA
}
__device__ __forceinline__ void store_add(const CUtensorMap* map, uint32_t src, uint32_t x, uint32_t row, uint32_t inner, uint32_t outer) {
    asm volatile("cp.reduce.async.bulk.tensor.4d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
                 ::"l"(map), "r"(src), "r"(x), "r"(row), "r"(inner), "r"(outer) : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}

// The part of x below its top 11 significant bits, exactly.
__device__ __forceinline__ float lo_of(float x) { return x - __uint_as_float(__float_as_uint(x) & 0xffffe000u); }

template <int CG, int BN, bool A_T, bool B_T, class A, class M>
__global__ void __launch_bounds__(Tile<CG, BN>::THREADS, 1) tf32_kernel(const __grid_constant__ A args, const __grid_constant__ M maps) {
    using T = Tile<CG, BN>;
    constexpr int STAGES = T::STAGES;
    extern __shared__ __align__(1024) char smem[];  // tiles on 1,024 bytes: the swizzle pattern is a function of address bits
    char* const slabs = smem + STAGES * T::STAGE_BYTES;
    float* const bias_tile = reinterpret_cast<float*>(slabs + T::DRAIN_WARPS * T::SLAB_BYTES);  // two of BN columns
    uint64_t* const bars = reinterpret_cast<uint64_t*>(bias_tile + 2 * BN);
    uint64_t* const raw_full = bars;             // a stage's raw block has landed (each CTA its own)
    uint64_t* const lo_full = raw_full + STAGES; // its lo block is written, in both CTAs (the first CTA's counts)
    uint64_t* const empty = lo_full + STAGES;    // the MMAs that read it are done
    uint64_t* const acc_full = empty + STAGES;
    uint64_t* const acc_empty = acc_full + 2;    // the first CTA's counts
    uint32_t* const tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    volatile uint32_t* const abort_flag = tmem_slot + 1;

    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = tc::cta_rank<CG>();
    const uint32_t first_unit = blockIdx.x / CG, step = gridDim.x / CG, units = args.units;

    if (tid == 0) {
        for (int s = 0; s < STAGES; ++s) {
            tc::mbar_init(tc::smem_u32(&raw_full[s]), 1);
            tc::mbar_init(tc::smem_u32(&lo_full[s]), CG * GROUP_THREADS / 32);
            tc::mbar_init(tc::smem_u32(&empty[s]), 1);
        }
        for (int b = 0; b < 2; ++b) {
            tc::mbar_init(tc::smem_u32(&acc_full[b]), 1);
            tc::mbar_init(tc::smem_u32(&acc_empty[b]), CG * T::DRAIN_WARPS);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == T::TMA_WARP && lane == 0 && first_unit < units) {
        const uint32_t product = unit_of(args, first_unit).product;
        tc::prefetch_map(&maps.a[product]);
        tc::prefetch_map(&maps.b[product]);
        tc::prefetch_map(&maps.c[product]);
    }
    if (warp == T::MMA_WARP) {
        tc::tmem_alloc<CG>(tc::smem_u32(tmem_slot), T::TMEM_COLUMNS);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if constexpr (CG == 2) tc::cluster_barrier();  // the other CTA's barriers exist before anything arrives on them
    else __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    wait_for_producers();

    if (warp < T::LO_WARPS) {
        // ---- lo blocks: the word at an offset of the lo tile belongs to the word at the same offset of the
        // raw tile, whatever the layout, so the tiles are walked straight through. A group of warps to each
        // stage: a block is a chain of about a thousand cycles (wait, read, write, the proxy fence, the
        // arrival) that more warps on one block do not shorten, so blocks are worked on side by side.
        uint32_t total = 0;
        for (uint32_t u = first_unit; u < units; u += step) total += unit_of(args, u).kblocks;
        const uint32_t stage = tid / GROUP_THREADS, in_group = tid % GROUP_THREADS;
        bool alive = true;
        uint32_t parity = 0;
        for (uint32_t g = stage; g < total && alive; g += STAGES, parity ^= 1u) {
            char* const at = smem + stage * T::STAGE_BYTES + in_group * 16;
            alive = tc::warp_wait<1>(tc::smem_u32(&raw_full[stage]), parity, abort_flag, args.status);
            if (!alive) break;
            constexpr int PER_THREAD = T::RAW_BYTES / 16 / GROUP_THREADS, OF_A = T::A_BYTES / 16 / GROUP_THREADS;
            constexpr int BATCH = PER_THREAD % 8 == 0 ? 8 : 10;
            static_assert(PER_THREAD % BATCH == 0, "whole batches");
            // Where chunk i of this thread lies: raw A, then (behind lo A) raw B; its lo half an operand further.
            auto raw_at = [](int i) -> uint32_t { return i * (GROUP_THREADS * 16u) + (i < OF_A ? 0u : T::A_BYTES); };
            auto lo_at = [&](int i) -> uint32_t { return raw_at(i) + (i < OF_A ? T::A_BYTES : T::B_BYTES); };
#pragma unroll
            for (int first = 0; first < PER_THREAD; first += BATCH) {
                float4 v[BATCH];
#pragma unroll
                for (int i = 0; i < BATCH; ++i) v[i] = *reinterpret_cast<const float4*>(at + raw_at(first + i));
#pragma unroll
                for (int i = 0; i < BATCH; ++i)
                    *reinterpret_cast<float4*>(at + lo_at(first + i)) = make_float4(lo_of(v[i].x), lo_of(v[i].y), lo_of(v[i].z), lo_of(v[i].w));
            }
            // Visible to the tensor core's async-proxy reads before the MMA warp is told.
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) tc::arrive_first<CG>(tc::smem_u32(&lo_full[stage]));
        }
    } else if (warp == T::MMA_WARP) {
        // ---- the MMA warp (the pair's first CTA) -------------------------------------------------------
        // Instruction descriptor: f32 accumulator, tf32 A and B, their majors, N >> 3, M >> 4. Matrix
        // descriptors as in tcgen05.cuh; an operand stored with k along its rows is K-major in the 128-byte
        // swizzle of 16-byte chunks (8-row groups 1,024 bytes apart), one stored with k down its columns
        // MN-major in the swizzle of 32-byte chunks, the one layout MN-major 32-bit operands have (4-row
        // groups 512 bytes, panels of 32 elements 4,096 bytes apart).
        if (CG == 1 || rank == 0) {
            const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((A_T ? 1u : 0u) << 15) | ((B_T ? 0u : 1u) << 16) |
                                   (static_cast<uint32_t>((128 * CG) >> 4) << 24);
            const uint32_t idesc_bn = idesc | (static_cast<uint32_t>(BN >> 3) << 17), idesc_acc = idesc | (T::ACC_COLUMNS >> 3) << 17;
            constexpr uint32_t a_lbo = A_T ? BK * 128u : 16u, b_lbo = B_T ? 16u : BK * 128u;
            constexpr uint32_t a_sbo = A_T ? 512u : 1024u, b_sbo = B_T ? 1024u : 512u;
            constexpr uint32_t a_type = A_T ? 1u : 2u, b_type = B_T ? 2u : 1u;
            constexpr uint32_t a_high = ((a_sbo >> 4) & 0x3FFFu) | (1u << 14) | (a_type << 29);
            constexpr uint32_t b_high = ((b_sbo >> 4) & 0x3FFFu) | (1u << 14) | (b_type << 29);
            constexpr uint32_t a_low = ((a_lbo >> 4) & 0x3FFFu) << 16, b_low = ((b_lbo >> 4) & 0x3FFFu) << 16;
            const uint32_t tiles16 = (tc::smem_u32(smem) & 0x3FFFFu) >> 4;
            auto desc = [](uint32_t high, uint32_t low) { return (static_cast<uint64_t>(high) << 32) | low; };
            bool alive = true;
            uint32_t stage = 0, parity = 0, turn = 0;
            for (uint32_t u = first_unit; u < units && alive; u += step) {
                const uint32_t kblocks = unit_of(args, u).kblocks;
                for (uint32_t kb = 0; kb < kblocks && alive; ++kb) {
                    const uint32_t in_segment = kb % SEGMENT, acc = turn & 1u;
                    if (in_segment == 0) {
                        alive = tc::warp_wait<CG>(tc::smem_u32(&acc_empty[acc]), ((turn >> 1) & 1u) ^ 1u, abort_flag, args.status);
                        if (!alive) break;
                    }
                    alive = tc::warp_wait<CG>(tc::smem_u32(&lo_full[stage]), parity, abort_flag, args.status);
                    if (!alive) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (lane == 0) {
                        const uint32_t a16 = a_low + tiles16 + stage * (T::STAGE_BYTES >> 4);
                        const uint32_t b16 = b_low + tiles16 + ((stage * T::STAGE_BYTES + 2 * T::A_BYTES) >> 4);
                        const uint32_t to = tmem_base + acc * T::ACC_COLUMNS;
#pragma unroll
                        for (uint32_t ks = 0; ks < BK / 8; ++ks) {
                            const uint32_t a_at = (A_T ? ks * 1024u : ks * 32u) >> 4, b_at = (B_T ? ks * 32u : ks * 1024u) >> 4;
                            const uint64_t a_hi = desc(a_high, a16 + a_at), a_lo = desc(a_high, a16 + (T::A_BYTES >> 4) + a_at);
                            const uint64_t b_hi = desc(b_high, b16 + b_at), b_lo = desc(b_high, b16 + (T::B_BYTES >> 4) + b_at);
                            if constexpr (T::STACKED) {
                                mma_tf32<CG, 0>(to, a_hi, b_hi, idesc_acc, (in_segment | ks) != 0u);  // raw and lo B
                                mma_tf32<CG, 0>(to + BN, a_lo, b_hi, idesc_bn, 1u);
                            } else {
                                mma_tf32<CG, 1>(to, a_hi, b_hi, idesc_bn, (in_segment | ks) != 0u);
                                mma_tf32<CG, 2>(to, a_hi, b_lo, idesc_bn, 1u);
                                mma_tf32<CG, 0>(to, a_lo, b_hi, idesc_bn, 1u);
                            }
                        }
                        tc::commit<CG>(tc::smem_u32(&empty[stage]));
                        if (in_segment + 1 == SEGMENT || kb + 1 == kblocks) tc::commit<CG>(tc::smem_u32(&acc_full[acc]));
                    }
                    if (in_segment + 1 == SEGMENT || kb + 1 == kblocks) ++turn;
                    if (++stage == STAGES) { stage = 0; parity ^= 1u; }
                    __syncwarp();
                }
            }
        }
    } else if (warp == T::TMA_WARP) {
        // ---- the TMA warp: the raw k blocks of every unit of this CTA, in order -----------------------------
        bool alive = true;
        uint32_t stage = 0, parity = 1;  // the parity a free stage shows
        uint32_t issued = 0;
        for (uint32_t u = first_unit; u < units && alive; u += step) {
            const Unit w = unit_of(args, u);
            const uint32_t m0 = w.m0 + rank * 128u, n0 = w.n0 + rank * T::BN_CTA;
            uint32_t product = w.product, k_at = w.split;  // k block of the product
            for (uint32_t kb = 0; kb < w.kblocks && alive; ++kb, ++issued) {
                alive = tc::warp_wait<CG>(tc::smem_u32(&empty[stage]), parity, abort_flag, args.status);
                if (!alive) break;
                if (lane == 0) {
                    const uint32_t bar = tc::smem_u32(&raw_full[stage]);
                    const uint32_t to_a = tc::smem_u32(smem + stage * T::STAGE_BYTES), to_b = to_a + 2 * T::A_BYTES;
                    const uint32_t k0 = k_at * BK;
                    auto load = [&](uint32_t to, const CUtensorMap* map, uint32_t x, uint32_t row) { tc::load_tile<1>(to, map, bar, x, row, w.z_inner, w.z_outer); };
                    tc::mbar_expect_tx(bar, T::RAW_BYTES);
                    if (A_T) {  // stored [k, m]: four boxes of 32 m by 32 k
#pragma unroll
                        for (uint32_t p = 0; p < 4; ++p) load(to_a + p * 4096u, &maps.a[product], m0 + 32u * p, k0);
                    } else {    // stored [m, k]: one box of 32 k by 128 m
                        load(to_a, &maps.a[product], k0, m0);
                    }
                    if (B_T) {  // stored [n, k]
                        load(to_b, &maps.b[product], k0, n0);
                    } else {    // stored [k, n]
#pragma unroll
                        for (uint32_t p = 0; p < T::BN_CTA / 32; ++p) load(to_b + p * 4096u, &maps.b[product], n0 + 32u * p, k0);
                    }
                }
                if (++stage == STAGES) { stage = 0; parity ^= 1u; }
                k_at += w.splits;
                if (args.chain > 1 && k_at == args.kblocks) { k_at = 0; ++product; }
                __syncwarp();
            }
        }
        let_next_start();  // what is left of this kernel are its last products and their way out
        // A role gave up: the loads still in flight land (a bounded wait each) before the CTA, and
        // with it their shared-memory destination, goes away.
        if (*abort_flag && lane == 0) {
            for (uint32_t back = 0; back < static_cast<uint32_t>(STAGES) && back < issued; ++back) {
                const uint32_t i = issued - 1 - back;
                for (uint32_t spin = 0; spin < tc::WAIT_LIMIT; ++spin)
                    if (tc::mbar_try_wait(tc::smem_u32(&raw_full[i % STAGES]), (i / STAGES) & 1u)) break;
            }
        }
    } else if (warp >= T::FIRST_DRAIN_WARP) {
        // ---- the drain warps ---------------------------------------------------------------------------------
        // A warp reads its lane quarter (the lanes a warp may read are 32 (warp % 4) ..), its share of the
        // columns 32 at a time; the sums with the bias go row by row into its slab of 32 rows x 128 bytes in
        // the 128-byte swizzle, which one TMA store writes (what lies outside C is not written), or, where C
        // cannot be a TMA target, the warp itself as 128-byte row segments.
        const uint32_t quarter = warp & 3u, part = (warp - T::FIRST_DRAIN_WARP) >> 2;
        char* const slab = slabs + (warp - T::FIRST_DRAIN_WARP) * T::SLAB_BYTES;
        const uint32_t first_col = part * T::CHUNKS * 32u;
        bool alive = true;
        uint32_t turn = 0;
        for (uint32_t u = first_unit; u < units && alive; u += step)
        for (uint32_t segment = 0, left = unit_of(args, u).kblocks; left > 0 && alive; left -= left < SEGMENT ? left : SEGMENT, ++segment, ++turn) {
            const Unit w = unit_of(args, u);
            const uint32_t acc = turn & 1u;
            // The bias of the warp's columns, fetched before the wait for the tile (a load issued in the drain
            // would queue behind all the SM has in flight) and put where every lane reads all of it. The
            // buffer is free: its last tile is two turns back, and this tile was begun only when all warps
            // were done with that one.
            float4 bias4 = make_float4(0.f, 0.f, 0.f, 0.f);
            const uint32_t bias_at = w.n0 + first_col + 4 * lane;
            if (w.bias && segment == 0 && lane < T::CHUNKS * 8u) {
                if (bias_at + 4 <= w.n && reinterpret_cast<uintptr_t>(w.bias) % 16 == 0) {
                    bias4 = load_global(reinterpret_cast<const float4*>(w.bias + bias_at));
                } else {
                    if (bias_at < w.n) bias4.x = load_global(w.bias + bias_at);
                    if (bias_at + 1 < w.n) bias4.y = load_global(w.bias + bias_at + 1);
                    if (bias_at + 2 < w.n) bias4.z = load_global(w.bias + bias_at + 2);
                    if (bias_at + 3 < w.n) bias4.w = load_global(w.bias + bias_at + 3);
                }
            }
            alive = tc::warp_wait<CG>(tc::smem_u32(&acc_full[acc]), (turn >> 1) & 1u, abort_flag, args.status);
            if (!alive) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            float* const my_bias = bias_tile + acc * BN + first_col;
            if (lane < T::CHUNKS * 8u) *reinterpret_cast<float4*>(my_bias + 4 * lane) = bias4;
            __syncwarp();
            const uint32_t first_row = w.m0 + rank * 128u + quarter * 32u;
            float* __restrict__ const out = w.c + static_cast<uint64_t>(w.split) * w.m * w.ldc;
            const uint32_t taddr = tmem_base + ((quarter * 32u) << 16) + acc * T::ACC_COLUMNS + first_col;
            // Two sets of registers: the next chunk, or the chunk's second half.
            uint32_t r[2][32];
            if (!T::STACKED) tc::tmem_load32(taddr, r[0]);
#pragma unroll
            for (int chunk = 0; chunk < T::CHUNKS; ++chunk) {
                if (T::STACKED) {
                    tc::tmem_load32(taddr + chunk * 32u, r[0]);
                    tc::tmem_load32(taddr + BN + chunk * 32u, r[1]);
                }
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (!T::STACKED && chunk + 1 < T::CHUNKS) tc::tmem_load32(taddr + (chunk + 1) * 32u, r[(chunk + 1) & 1]);
                const uint32_t gn0 = w.n0 + first_col + chunk * 32u;
                if (gn0 >= w.n) continue;  // the same for the whole warp
                // The store that last read the slab has finished reading it, and, for a later segment, written
                // what this one adds to.
                if (args.c_tma) {
                    if (lane == 0) {
                        if (segment == 0) tc::tma_store_wait_read<0>();
                        else asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
                    }
                    __syncwarp();
                }
                const uint32_t(&from)[32] = r[T::STACKED ? 0 : chunk & 1];
                auto sum = [&](uint32_t j) {
                    return T::STACKED ? __uint_as_float(from[j]) + __uint_as_float(r[1][j]) : __uint_as_float(from[j]);
                };
#pragma unroll
                for (uint32_t j = 0; j < 32; j += 4) {
                    // One addition an element: the bias, or the `x + 0` that turns a -0 sum of zero products
                    // into the +0 a skipped term gives (as a bias of +0 does).
                    const float4 add = *reinterpret_cast<const float4*>(my_bias + chunk * 32 + j);
                    float4 v;
                    v.x = sum(j) + add.x;
                    v.y = sum(j + 1) + add.y;
                    v.z = sum(j + 2) + add.z;
                    v.w = sum(j + 3) + add.w;
                    *reinterpret_cast<float4*>(slab + tc::swizzled_chunk(lane, j >> 2)) = v;
                }
                if (args.c_tma) {
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0 && first_row < w.m) {
                        const uint32_t inner = w.splits > 1 ? w.split : w.z_inner;
                        if (segment == 0) tc::store_tile(&maps.c[w.product], tc::smem_u32(slab), gn0, first_row, inner, w.z_outer);
                        else store_add(&maps.c[w.product], tc::smem_u32(slab), gn0, first_row, inner, w.z_outer);
                    }
                    continue;
                }
                __syncwarp();
                const uint32_t c4 = (lane & 7u) * 4, gn = gn0 + c4;
#pragma unroll
                for (uint32_t pass = 0; pass < 8; ++pass) {
                    const uint32_t row = pass * 4 + (lane >> 3), gm = first_row + row;
                    if (gm >= w.m || gn >= w.n) continue;
                    float4 v = *reinterpret_cast<const float4*>(slab + tc::swizzled_chunk(row, lane & 7u));
                    float* dst = out + static_cast<uint64_t>(gm) * w.ldc + gn;
                    if (segment > 0) {  // (the lane wrote these elements itself)
                        v.x += dst[0];
                        if (gn + 1 < w.n) v.y += dst[1];
                        if (gn + 2 < w.n) v.z += dst[2];
                        if (gn + 3 < w.n) v.w += dst[3];
                    }
                    // Inside the pitch a whole float4 may be written: what lies past n is padding.
                    if (args.c_vec && (gn + 4 <= w.n || (args.c_padded && gn + 4 <= w.ldc))) {
                        *reinterpret_cast<float4*>(dst) = v;
                    } else {
                        if (gn < w.n) dst[0] = v.x;
                        if (gn + 1 < w.n) dst[1] = v.y;
                        if (gn + 2 < w.n) dst[2] = v.z;
                        if (gn + 3 < w.n) dst[3] = v.w;
                    }
                }
                __syncwarp();
            }
            // The warp's share of the accumulator and of the bias has been read.
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) tc::arrive_first<CG>(tc::smem_u32(&acc_empty[acc]));
        }
        // The slab must outlive the store that reads it.
        if (args.c_tma && lane == 0) tc::tma_store_wait_read<0>();
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncwarp();
    if constexpr (CG == 2) tc::cluster_barrier();  // the pair's remote arrivals have landed before either CTA goes away
    else __syncthreads();
    if (warp == T::MMA_WARP) {
        tc::tmem_dealloc<CG>(tmem_base, T::TMEM_COLUMNS);
    }
}

template <int CG, int BN, bool A_T, bool B_T, class A, class M> void launch(cudaStream_t s, const A& args, const M& maps) {
    using T = Tile<CG, BN>;
    auto kernel = tf32_kernel<CG, BN, A_T, B_T, A, M>;
    static std::atomic<int> configured_device{-1};
    set_shared_memory(kernel, static_cast<int>(T::TOTAL), configured_device);
    // One CTA per SM, alone or in pairs, each walking its share of the units.
    const uint32_t most = device_sm_count() / CG;
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3((args.units < most ? args.units : most) * CG);
    config.blockDim = dim3(T::THREADS);
    config.dynamicSmemBytes = T::TOTAL;
    config.stream = s;
    cudaLaunchAttribute pair = {};
    pair.id = cudaLaunchAttributeClusterDimension;
    pair.val.clusterDim.x = CG;
    pair.val.clusterDim.y = pair.val.clusterDim.z = 1;
    if (CG > 1) {
        config.attrs = &pair;
        config.numAttrs = 1;
    }
    check(cudaLaunchKernelEx(&config, kernel, args, maps), "matmul_tf32");
}

template <int CG, int BN, class A, class M> void launch_form(cudaStream_t s, bool a_t, bool b_t, const A& args, const M& maps) {
    if (a_t && b_t) launch<CG, BN, true, true>(s, args, maps);
    else if (a_t) launch<CG, BN, true, false>(s, args, maps);
    else if (b_t) launch<CG, BN, false, true>(s, args, maps);
    else launch<CG, BN, false, false>(s, args, maps);
}

bool aligned16(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

// Where the matrices of a batch lie: `inner` of them stride_inner apart, `outer` such rows stride_outer apart.
struct Batch {
    uint64_t inner, stride_inner, outer, stride_outer;
};
// A matrix of `rows` rows of `cols` floats, `pitch` apart, or a batch of them as two more coordinates,
// as a tensor map of boxes of 32 floats by `box_rows` rows.
CUtensorMap encode(const float* base, uint64_t cols, uint64_t rows, uint64_t pitch, const Batch& z, uint32_t box_rows, bool chunks_of_32) {
    // A dimension of one element may carry any stride.
    const uint64_t whole = pitch * rows;
    const cuuint64_t size[4] = {cols, rows, z.inner, z.outer};
    const cuuint64_t stride[3] = {pitch * 4, (z.inner > 1 ? z.stride_inner : whole) * 4, (z.outer > 1 ? z.stride_outer : whole) * 4};
    const cuuint32_t box[4] = {32, box_rows, 1, 1}, element[4] = {1, 1, 1, 1};
    CUtensorMap map;
    const CUresult r = tc::encode_tiled()(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float*>(base), size, stride, box, element,
                                          CU_TENSOR_MAP_INTERLEAVE_NONE, chunks_of_32 ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B,
                                          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) throw std::invalid_argument("matmul_tf32: cuTensorMapEncodeTiled refused a matrix (" + std::to_string(static_cast<int>(r)) + ")");
    return map;
}
constexpr Batch ONE = {1, 0, 1, 0};
Batch splits_of(uint64_t splits, uint64_t m, uint64_t n) { return {splits, m * n, 1, 0}; }  // the split-k workspace
// The tensor maps of one product's operands: boxes of 32 floats by the CTA's rows for an operand stored
// with k along its rows, 32 by 32 in the swizzle of 32-byte chunks for one with k down its columns.
template <class M> void encode_operands(M& maps, uint32_t at, const float* a, uint32_t lda, const float* b, uint32_t ldb, bool a_t, bool b_t, uint64_t m, uint64_t n,
                                        uint64_t k, uint32_t b_rows, const Batch& of_a = ONE, const Batch& of_b = ONE) {
    maps.a[at] = a_t ? encode(a, m, k, lda, of_a, 32, true) : encode(a, k, m, lda, of_a, 128, false);
    maps.b[at] = b_t ? encode(b, k, n, ldb, of_b, b_rows, false) : encode(b, n, k, ldb, of_b, 32, true);
}
bool tma_addressable(const float* base, uint64_t pitch) { return aligned16(base) && pitch % 4 == 0; }
bool tma_addressable(const BatchedOperand& x) { return tma_addressable(x.base, x.pitch) && x.stride_outer % 4 == 0 && x.stride_inner % 4 == 0; }

void launch_plan(cudaStream_t s, const MatmulTcPlan& p, bool a_t, bool b_t, const Args& args, const Maps& maps) {
    if (p.bm == 256) launch_form<2, 256>(s, a_t, b_t, args, maps);
    else if (p.bn == 128) launch_form<1, 128>(s, a_t, b_t, args, maps);
    else if (p.bn == 64) launch_form<1, 64>(s, a_t, b_t, args, maps);
    else launch_form<1, 32>(s, a_t, b_t, args, maps);
}

}  // namespace

void matmul_tf32(cudaStream_t s, const MatmulTcPlan& p, const MatmulOperands* products, uint32_t count, bool a_t, bool b_t, uint64_t m, uint64_t n, uint64_t k,
                 uint32_t chain, MatmulPitches pitches, uint32_t* status) {
    Args args;
    Maps maps = {};
    const bool partial = p.splits > 1;
    const uint32_t lda = pitches.a ? pitches.a : static_cast<uint32_t>(a_t ? m : k), ldb = pitches.b ? pitches.b : static_cast<uint32_t>(b_t ? k : n);
    args.m = static_cast<uint32_t>(m);
    args.n = static_cast<uint32_t>(n);
    // Partial tiles of a split k are dense; the pitch of C applies to the CTAs that write C itself.
    args.ldc = pitches.c && !partial ? pitches.c : static_cast<uint32_t>(n);
    args.splits = tc::Divisor(p.splits);
    args.walk = tc::TileWalk(m, n, p.bm, p.bn);
    args.kblocks = static_cast<uint32_t>((k + BK - 1) / BK);
    args.chain = chain;
    args.status = status;
    args.c_padded = pitches.c != 0 && !partial;
    args.c_vec = args.ldc % 4 == 0;
    const uint32_t results = chain > 1 ? 1 : count, group = p.bm / 128;
    for (uint32_t g = 0; g < count; ++g) {
        encode_operands(maps, g, products[g].a, lda, products[g].b, ldb, a_t, b_t, m, n, k, p.bn / group);
        if (g >= results) continue;
        args.c[g] = partial ? products[g].workspace : products[g].c;
        args.bias[g] = partial ? nullptr : products[g].bias;
        args.c_vec = args.c_vec && aligned16(args.c[g]);
        args.c_tma = args.c_tma && tma_addressable(args.c[g], args.ldc);
    }
    for (uint32_t g = 0; g < results && args.c_tma; ++g) maps.c[g] = encode(args.c[g], n, m, args.ldc, splits_of(p.splits, m, n), 32, false);
    args.units = args.walk.count() * p.splits * results;
    launch_plan(s, p, a_t, b_t, args, maps);
}

bool matmul_tf32_batched(cudaStream_t s, const BatchedProduct* products, uint32_t count, uint64_t m, uint64_t n, uint64_t k, uint32_t outer, uint32_t inner,
                         uint32_t* status) {
    if (k == 0) return false;
    for (uint32_t g = 0; g < count; ++g)
        for (const BatchedOperand* x : {&products[g].a, &products[g].b, &products[g].c})
            if (!tma_addressable(*x)) return false;
    const uint64_t problems = static_cast<uint64_t>(outer) * inner;
    // One product whose 64 x 32 tiles all find an SM of their own is about a microsecond sooner on those, or as soon
    // (eleven attentions of 16 to 144 such tiles a product, forward: 2 to 16 heads of 128 queries x 128 keys x 64 18.6 ->
    // 16.6 us, 12 of 100 x 100 x 40 the same, the others of 32 to 512 keys within 1 us either way); from two tiles to an SM on, or with two products
    // to share a launch, these tiles win (64 such heads: forward 16.3 -> 14.9 us, backward 29.9 -> 21.0;
    // 384 heads of 512 x 512 x 64: forward 745 -> 414 us, backward 1,151 -> 643).
    if (count == 1 && (m + 63) / 64 * ((n + 31) / 32) * problems <= device_sm_count()) return false;
    const MatmulTcPlan p = matmul_tc_plan(m, n, k, problems, count, true, 1, true);
    Args args;
    Maps maps = {};
    args.m = static_cast<uint32_t>(m);
    args.n = static_cast<uint32_t>(n);
    args.ldc = products[0].c.pitch;
    args.splits = tc::Divisor(1);
    args.batch = tc::Divisor(static_cast<uint32_t>(problems));
    args.batch_inner = tc::Divisor(inner);
    args.walk = tc::TileWalk(m, n, p.bm, p.bn);
    args.kblocks = static_cast<uint32_t>((k + BK - 1) / BK);
    args.status = status;
    const bool a_t = products[0].a.transposed, b_t = products[0].b.transposed;
    for (uint32_t g = 0; g < count; ++g) {
        const BatchedProduct& q = products[g];
        auto batch = [&](const BatchedOperand& x) { return Batch{inner, x.stride_inner, outer, x.stride_outer}; };
        encode_operands(maps, g, q.a.base, q.a.pitch, q.b.base, q.b.pitch, a_t, b_t, m, n, k, p.bn / (p.bm / 128), batch(q.a), batch(q.b));
        maps.c[g] = encode(q.c.base, n, m, q.c.pitch, batch(q.c), 32, false);
        args.c[g] = const_cast<float*>(q.c.base);
    }
    args.units = static_cast<uint32_t>(args.walk.count() * problems * count);
    launch_plan(s, p, a_t, b_t, args, maps);
    return true;
}

bool matmul_tf32_jobs(cudaStream_t s, const MatmulJob* jobs, uint32_t count, bool a_t, bool b_t, uint32_t* status) {
    JobArgs args;
    JobMaps maps = {};
    args.status = status;
    for (uint32_t j = 0; j < count; ++j) {
        const MatmulJob& job = jobs[j];
        const MatmulTcPlan p = matmul_tc_job_plan(job.m, job.n, job.k);
        const bool partial = p.splits > 1;
        float* const c = partial ? job.workspace : job.c;
        const uint32_t lda = static_cast<uint32_t>(a_t ? job.m : job.k), ldb = static_cast<uint32_t>(b_t ? job.k : job.n);
        if (job.k == 0 || !tma_addressable(job.a, lda) || !tma_addressable(job.b, ldb) || !tma_addressable(c, job.n)) return false;
        Job& to = args.jobs[args.job_count++];
        to.c = c;
        to.m = static_cast<uint32_t>(job.m);
        to.n = static_cast<uint32_t>(job.n);
        to.splits = tc::Divisor(p.splits);
        to.walk = tc::TileWalk(job.m, job.n, 128, 128);
        to.kblocks = static_cast<uint32_t>((job.k + BK - 1) / BK);
        to.first_unit = args.units;
        args.units += to.walk.count() * p.splits;
        encode_operands(maps, j, job.a, lda, job.b, ldb, a_t, b_t, job.m, job.n, job.k, 128);
        maps.c[j] = encode(c, job.n, job.m, job.n, splits_of(p.splits, job.m, job.n), 32, false);
    }
    launch_form<1, 128>(s, a_t, b_t, args, maps);
    return true;
}

}  // namespace k
}  // namespace msx
