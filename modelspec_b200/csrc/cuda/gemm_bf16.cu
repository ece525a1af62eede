// matmul on bf16 operands for mixed-precision plans: tcgen05.mma (kind::f16, bf16 inputs) fed by TMA,
// f32 accumulation in tensor memory.
//
// The reference has no 16-bit type (crates/modelspec-core/src/ir/tensor.rs:38-51: f32 and i32); a
// plan made with MSX_PLAN_BF16 stores activations and the working copy of every weight as bf16
// and runs every product here. An operand needs no conversion on its way to the tensor core, so
// unlike the split-TF32 kernels no thread touches the tiles between global memory and the MMA.
//
// What bounds it. A large product is bound by the tensor cores once its operands reach them: two CTAs of
// a cluster pair up on 256 x 256 tiles (cta_group::2), each holding its 128 rows of A and 128 of the 256
// columns of B, so that a k block of 64 costs an SM 32 KB of loads and shared memory for 512 cycles of
// MMAs (a 128 x 256 tile of one CTA: 48 KB). A small one is bound by its launch's chain of latencies
// (set-up, TMA round trip, drain, 4 to 5 us together), which products of one shape that are ready
// together share (`products`), as do weight gradients of different shapes (jobs); products that are summed
// are one with a longer k (`chain`). What follows a product element by element is applied as its tile
// drains: the bias, gelu (stored beside its argument), the gradient of gelu.
//
// A CTA is persistent and walks the launch's units (tiles x k splits x batch x products):
//   warp 0      one thread issues the TMA loads of a k block (64 deep) into the next free stage;
//   warp 1      (of the pair's first CTA) issues the MMAs into one of two accumulators;
//   warps 4..   drain the other accumulator: 32 lanes x 32 columns at a time, bias, epilogue, conversion,
//               into slabs of 32 rows x 128 bytes of their own, which TMA stores write to C.
//
// Storage forms: an operand is K-major when k is its contiguous index (A stored [m, k], B stored
// [n, k]) and MN-major otherwise (A stored [k, m], B stored [k, n]). Both are read in place: a
// K-major tile is rows of 128 bytes (64 k), an MN-major tile is panels of 64 m (or n) by 64 k
// rows of 128 bytes; the shared-memory descriptors name the layout, so NN, NT, TN and TT need no
// transposed copy. Batched products (attention heads) address (sequence, head) through two more
// tensor-map coordinates. Every tensor map covers this GPU's own memory only, and every load is a
// plain one to the issuing CTA.
//
// Every wait is bounded and, when it runs out, raises bit 1 of the status word, makes every role leave
// its loop, lets the copies in flight land, frees the tensor memory and returns.
#include <atomic>
#include <cmath>

#include "common.cuh"
#include "kernels.cuh"
#include "tcgen05.cuh"

namespace msx {
namespace k {

namespace {

using namespace tc;

constexpr int BK = 64;
constexpr int FIRST_DRAIN_WARP = 4;
constexpr uint32_t PANEL_BYTES = 64 * BK * 2;  // an MN-major panel: 64 k rows of 64 elements
constexpr uint32_t SLAB_BYTES = 32 * 128;
constexpr int MAX_PRODUCTS = 4, MAX_JOBS = 24;

template <int CG, int BN> struct Tile {
    static constexpr int BN_CTA = BN / CG;  // columns of B a CTA holds
    static constexpr uint32_t A_BYTES = 128 * BK * 2, B_BYTES = BN_CTA * BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
    static constexpr int STAGES = BN_CTA == 128 ? 5 : 6;
    static constexpr int DRAIN_WARPS = BN == 64 ? 4 : 8;         // one or two per lane quarter
    static constexpr int COLUMNS = BN / (DRAIN_WARPS / 4);       // of a drain warp
    static constexpr int THREADS = 32 * (FIRST_DRAIN_WARP + DRAIN_WARPS);
    static constexpr uint32_t TOTAL = STAGES * STAGE_BYTES + DRAIN_WARPS * 2 * SLAB_BYTES + 2 * BN * 4 /* bias */ + 256 /* barriers */;
    static constexpr uint32_t TMEM_COLUMNS = 2 * BN;
    static_assert(TOTAL <= 232448, "shared memory of a CTA");
};

struct Job {
    void* c;  // the result (f32), or the job's split-k workspace
    uint32_t m, n, splits, kblocks, per_split, first_unit;
    TileWalk walk;
};
struct Args {
    uint32_t units = 0, m = 0, n = 0, ldc = 0;
    TileWalk walk;
    Divisor splits;
    uint32_t kblocks = 0, per_split = 0;  // of one product; contiguous k blocks of a split
    uint32_t chain = 1;                   // > 1: that many products are summed into one result
    Divisor batch, batch_inner;           // matrices per operand, and the faster of their two indices
    uint64_t c_outer = 0, c_inner = 0;    // elements between the C matrices of consecutive batch indices
    uint32_t out_half = 0;                // C is bf16 (never the workspace)
    uint32_t c_tma = 1;                   // C by TMA stores
    void* c[MAX_PRODUCTS] = {};           // C, or the split-k workspace [splits][m][n] (f32)
    const float* bias[MAX_PRODUCTS] = {};
    uint32_t* status = nullptr;
};
struct Maps {
    CUtensorMap a[MAX_PRODUCTS], b[MAX_PRODUCTS], c[MAX_PRODUCTS];
    CUtensorMap beside;  // Epilogue::Gelu: where gelu of the result goes; Epilogue::GeluGrad: the argument of gelu
};
// Products of different shapes and one storage form in one launch.
struct JobArgs : Args {
    uint32_t job_count = 0;
    Job jobs[MAX_JOBS] = {};
};
struct JobMaps {
    CUtensorMap a[MAX_JOBS], b[MAX_JOBS], c[MAX_JOBS];
    CUtensorMap beside;
};

// Unit `u` of a launch: its tile, then the split, the batch index, and the product or job.
struct Unit {
    uint32_t m0, n0, split, product, kblocks, kb0, z_inner, z_outer;
    uint32_t m, n, ldc, splits;
    void* c;
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
    w.bias = w.splits > 1 ? nullptr : args.bias[w.product];
    w.kb0 = w.split * args.per_split;
    w.kblocks = args.chain > 1 ? args.kblocks * args.chain : (w.kb0 >= args.kblocks ? 0u : min(args.per_split, args.kblocks - w.kb0));
    return w;
}
__device__ __forceinline__ Unit unit_of(const JobArgs& args, uint32_t u) {
    uint32_t j = 0;
    while (j + 1 < args.job_count && args.jobs[j + 1].first_unit <= u) ++j;
    const Job& job = args.jobs[j];
    Unit w;
    w.m = job.m; w.n = job.n; w.ldc = job.n; w.splits = job.splits;
    w.split = job.walk.take(u - job.first_unit, &w.m0, &w.n0);
    w.product = j;
    w.z_inner = w.z_outer = 0;
    w.c = job.c;
    w.bias = nullptr;
    w.kb0 = w.split * job.per_split;
    w.kblocks = w.kb0 >= job.kblocks ? 0u : min(job.per_split, job.kblocks - w.kb0);
    return w;
}

template <int CG> __device__ __forceinline__ void mma(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    if constexpr (CG == 1)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                     ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
    else
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                     ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}

template <int CG, int BN, bool A_MN, bool B_MN, Epilogue EPILOGUE, class A, class M>
__global__ void __launch_bounds__(Tile<CG, BN>::THREADS, 1) bf16_kernel(const __grid_constant__ A args, const __grid_constant__ M maps) {
    using T = Tile<CG, BN>;
    constexpr int STAGES = T::STAGES;
    extern __shared__ __align__(1024) char smem[];  // tiles on 1,024 bytes: the swizzle pattern is a function of address bits
    char* const slabs = smem + STAGES * T::STAGE_BYTES;
    float* const bias_tile = reinterpret_cast<float*>(slabs + T::DRAIN_WARPS * 2 * SLAB_BYTES);  // two of BN columns
    uint64_t* const bars = reinterpret_cast<uint64_t*>(bias_tile + 2 * BN);
    uint64_t* const full = bars;               // a stage has landed in every CTA of the group (the first CTA's counts)
    uint64_t* const empty = full + STAGES;     // the MMAs that read it are done
    uint64_t* const acc_full = empty + STAGES;
    uint64_t* const acc_empty = acc_full + 2;  // the first CTA's counts
    uint64_t* const beside_full = acc_empty + 2;  // per drain warp: its slab of the argument of gelu has landed
    uint32_t* const tmem_slot = reinterpret_cast<uint32_t*>(beside_full + T::DRAIN_WARPS);
    volatile uint32_t* const abort_flag = tmem_slot + 1;

    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = cta_rank<CG>();
    const uint32_t first_unit = blockIdx.x / CG, step = gridDim.x / CG, units = args.units;

    if (tid == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(smem_u32(&full[s]), 1);  // the first CTA's TMA warp, with the bytes all CTAs of the group expect
            mbar_init(smem_u32(&empty[s]), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&acc_full[b]), 1);
            mbar_init(smem_u32(&acc_empty[b]), CG * T::DRAIN_WARPS);
        }
        for (int d = 0; d < T::DRAIN_WARPS; ++d) mbar_init(smem_u32(&beside_full[d]), 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0 && lane == 0 && first_unit < units) {
        const uint32_t product = unit_of(args, first_unit).product;
        prefetch_map(&maps.a[product]);
        prefetch_map(&maps.b[product]);
        prefetch_map(&maps.c[product]);
    }
    if (warp == 1) tmem_alloc<CG>(smem_u32(tmem_slot), T::TMEM_COLUMNS);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if constexpr (CG == 2) cluster_barrier();  // the other CTA's barriers exist before anything arrives on them
    else __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    wait_for_producers();

    if (warp == 0) {
        // ---- the TMA warp: the k blocks of every unit of this CTA, in order -----------------------------
        bool alive = true;
        uint32_t stage = 0, parity = 1;  // the parity a free stage shows
        uint32_t issued = 0;
        for (uint32_t u = first_unit; u < units && alive; u += step) {
            const Unit w = unit_of(args, u);
            const uint32_t m0 = w.m0 + rank * 128u, n0 = w.n0 + rank * T::BN_CTA;
            uint32_t product = w.product, k_at = w.kb0;
            for (uint32_t kb = 0; kb < w.kblocks && alive; ++kb, ++issued) {
                alive = warp_wait<CG>(smem_u32(&empty[stage]), parity, abort_flag, args.status);
                if (!alive) break;
                if (lane == 0) {
                    const uint32_t bar = first_cta<CG>(smem_u32(&full[stage]));
                    const uint32_t to_a = smem_u32(smem + stage * T::STAGE_BYTES), to_b = to_a + T::A_BYTES;
                    const uint32_t k0 = k_at * BK;
                    // Both CTAs' bytes count on the first one's barrier (the second's may land before they are
                    // expected: the phase cannot end without the arrival).
                    if (rank == 0) mbar_expect_tx(smem_u32(&full[stage]), CG * T::STAGE_BYTES);
                    if (A_MN) {  // stored [k, m]: two panels of 64 m
#pragma unroll
                        for (uint32_t p = 0; p < 2; ++p) load_tile<CG>(to_a + p * PANEL_BYTES, &maps.a[product], bar, m0 + p * 64u, k0, w.z_inner, w.z_outer);
                    } else {     // stored [m, k]: 128 rows of 64 k
                        load_tile<CG>(to_a, &maps.a[product], bar, k0, m0, w.z_inner, w.z_outer);
                    }
                    if (B_MN) {  // stored [k, n]
#pragma unroll
                        for (uint32_t p = 0; p < T::BN_CTA / 64; ++p) load_tile<CG>(to_b + p * PANEL_BYTES, &maps.b[product], bar, n0 + p * 64u, k0, w.z_inner, w.z_outer);
                    } else {     // stored [n, k]
                        load_tile<CG>(to_b, &maps.b[product], bar, k0, n0, w.z_inner, w.z_outer);
                    }
                }
                if (++stage == STAGES) { stage = 0; parity ^= 1u; }
                if (++k_at == args.kblocks && args.chain > 1) { k_at = 0; ++product; }
                __syncwarp();
            }
        }
        let_next_start();  // what is left of this kernel are its last products and their way out
        // A role gave up: the loads still in flight, of both CTAs, land (a bounded wait each on the first
        // one's barriers) before either CTA, and with it their shared-memory destination, goes away.
        if (*abort_flag && lane == 0 && rank == 0) {
            for (uint32_t back = 0; back < static_cast<uint32_t>(STAGES) && back < issued; ++back) {
                const uint32_t i = issued - 1 - back;
                for (uint32_t spin = 0; spin < WAIT_LIMIT; ++spin)
                    if (try_wait<CG>(smem_u32(&full[i % STAGES]), (i / STAGES) & 1u)) break;
            }
        }
    } else if (warp == 1) {
        // ---- the MMA warp (the pair's first CTA) -------------------------------------------------------
        if (rank == 0) {
            // Shared-memory matrix descriptors as in tcgen05.cuh. K-major: 8-row groups 1024 bytes apart
            // (stride offset), the leading offset unused. MN-major: panels of 64 elements 8192 bytes apart
            // (leading offset), groups of 8 k rows 1024 bytes apart (stride offset).
            const uint32_t idesc = instruction_descriptor(128 * CG, BN, A_MN, B_MN);
            constexpr uint32_t a_lbo = A_MN ? PANEL_BYTES : 16u, b_lbo = B_MN ? PANEL_BYTES : 16u;
            bool alive = true;
            uint32_t stage = 0, parity = 0, turn = 0;
            for (uint32_t u = first_unit; u < units && alive; u += step, ++turn) {
                const uint32_t kblocks = unit_of(args, u).kblocks, acc = turn & 1u;
                alive = warp_wait<CG>(smem_u32(&acc_empty[acc]), ((turn >> 1) & 1u) ^ 1u, abort_flag, args.status);
                if (!alive) break;
                const uint32_t to = tmem_base + acc * BN;
                for (uint32_t kb = 0; kb < kblocks && alive; ++kb) {
                    alive = warp_wait<CG>(smem_u32(&full[stage]), parity, abort_flag, args.status);
                    if (!alive) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (lane == 0) {
                        const uint32_t a_at = smem_u32(smem + stage * T::STAGE_BYTES), b_at = a_at + T::A_BYTES;
#pragma unroll
                        for (uint32_t ks = 0; ks < BK / 16; ++ks)
                            // k = 16: 32 bytes along a K-major row, or 16 rows (2048 bytes) of an MN-major panel.
                            mma<CG>(to, tile_descriptor(a_at + (A_MN ? ks * 2048u : ks * 32u), a_lbo), tile_descriptor(b_at + (B_MN ? ks * 2048u : ks * 32u), b_lbo),
                                    idesc, (kb | ks) != 0u);
                        commit<CG>(smem_u32(&empty[stage]));
                    }
                    if (++stage == STAGES) { stage = 0; parity ^= 1u; }
                    __syncwarp();
                }
                if (alive && lane == 0) commit<CG>(smem_u32(&acc_full[acc]));  // arrives at once when no MMA is pending
                __syncwarp();
            }
        }
    } else if (warp >= FIRST_DRAIN_WARP) {
        // ---- the drain warps ---------------------------------------------------------------------------------
        const uint32_t quarter = warp & 3u, part = (warp - FIRST_DRAIN_WARP) >> 2;
        char* const my_slabs = slabs + (warp - FIRST_DRAIN_WARP) * 2 * SLAB_BYTES;
        const uint32_t beside_bar = smem_u32(&beside_full[warp - FIRST_DRAIN_WARP]);
        const uint32_t first_col = part * T::COLUMNS;
        bool alive = true;
        uint32_t turn = 0, stores = 0, besides = 0;
        for (uint32_t u = first_unit; u < units && alive; u += step, ++turn) {
            const Unit w = unit_of(args, u);
            const uint32_t acc = turn & 1u;
            const bool half_out = args.out_half != 0 && w.splits == 1;
            const uint32_t first_row = w.m0 + rank * 128u + quarter * 32u;
            const bool rows_inside = first_row < w.m;  // else nothing of this warp's is stored
            if (EPILOGUE == Epilogue::GeluGrad && lane == 0 && rows_inside && w.n0 + first_col < w.n) {
                mbar_expect_tx(beside_bar, SLAB_BYTES);
                load_tile<1>(smem_u32(my_slabs + SLAB_BYTES), &maps.beside, beside_bar, w.n0 + first_col, first_row, 0, 0);
            }
            // The bias of the warp's columns, fetched before the wait for the tile (a load issued in the drain
            // would queue behind all the SM has in flight) and put where every lane reads all of it. The
            // buffer is free: its last tile is two turns back, and this tile was begun only when all warps
            // were done with that one.
            float bias[T::COLUMNS / 32];
#pragma unroll
            for (int i = 0; i < T::COLUMNS / 32; ++i) {
                const uint32_t c = w.n0 + first_col + i * 32 + lane;
                bias[i] = w.bias && c < w.n ? load_global(w.bias + c) : 0.0f;
            }
            alive = warp_wait<CG>(smem_u32(&acc_full[acc]), (turn >> 1) & 1u, abort_flag, args.status);
            if (!alive) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            float* const my_bias = bias_tile + acc * BN + first_col;
#pragma unroll
            for (int i = 0; i < T::COLUMNS / 32; ++i) my_bias[i * 32 + lane] = bias[i];
            __syncwarp();
            const uint32_t taddr = tmem_base + ((quarter * 32u) << 16) + acc * BN + first_col;
            const bool has_k = w.kblocks > 0;
            // 32 columns of the lane's row from column `c` of the warp's, with the bias.
            auto columns = [&](uint32_t c, float (&v)[32]) {
                uint32_t r[32];
                if (has_k) {
                    tmem_load32(taddr + c, r);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                }
#pragma unroll
                for (int j = 0; j < 32; j += 4) {
                    const float4 add = *reinterpret_cast<const float4*>(my_bias + c + j);
                    v[j] = (has_k ? __uint_as_float(r[j]) : 0.0f) + add.x;
                    v[j + 1] = (has_k ? __uint_as_float(r[j + 1]) : 0.0f) + add.y;
                    v[j + 2] = (has_k ? __uint_as_float(r[j + 2]) : 0.0f) + add.z;
                    v[j + 3] = (has_k ? __uint_as_float(r[j + 3]) : 0.0f) + add.w;
                }
            };
            auto put8 = [&](char* slab, uint32_t chunk, const float (&v)[8]) {
                float8 f;
                f.lo = make_float4(v[0], v[1], v[2], v[3]);
                f.hi = make_float4(v[4], v[5], v[6], v[7]);
                store8(reinterpret_cast<bf16*>(slab + swizzled_chunk(lane, chunk)), f);
            };
            const uint32_t slab_columns = half_out ? 64u : 32u;
            const uint64_t out_at = w.splits > 1 ? static_cast<uint64_t>(w.split) * w.m * w.n
                                                 : static_cast<uint64_t>(w.z_outer) * args.c_outer + static_cast<uint64_t>(w.z_inner) * args.c_inner;
#pragma unroll 1
            for (uint32_t c0 = 0; c0 < static_cast<uint32_t>(T::COLUMNS); c0 += slab_columns) {
                const uint32_t gn0 = w.n0 + first_col + c0;
                // The same for the whole warp. Rows below C are not drained either: with no store of their own
                // behind them, the wait below would let them into the slab that the last store may still read.
                if (gn0 >= w.n || !rows_inside) break;
                char* const slab = my_slabs + (EPILOGUE == Epilogue::None ? (stores++ & 1u) * SLAB_BYTES : 0u);
                if (args.c_tma) {
                    // The store that last read the slab (two turns ago, or the last) has finished reading it.
                    if (lane == 0) {
                        if (EPILOGUE == Epilogue::None) tma_store_wait_read<1>();
                        else tma_store_wait_read<0>();
                    }
                    __syncwarp();
                }
                if constexpr (EPILOGUE == Epilogue::GeluGrad) {
                    alive = warp_wait<1>(beside_bar, besides & 1u, abort_flag, args.status);
                    if (!alive) break;
                    ++besides;
                }
                if (half_out) {
#pragma unroll
                    for (uint32_t half = 0; half < 2; ++half) {
                        float v[32];
                        columns(c0 + half * 32u, v);
#pragma unroll
                        for (uint32_t j = 0; j < 32; j += 8) {
                            const uint32_t chunk = half * 4u + (j >> 3);
                            float e[8];
#pragma unroll
                            for (int i = 0; i < 8; ++i) e[i] = v[j + i];
                            if constexpr (EPILOGUE == Epilogue::Gelu) {
                                // gelu of the value as stored, as a launch that read it back would see it.
                                put8(slab, chunk, e);
#pragma unroll
                                for (int i = 0; i < 8; ++i) e[i] = gelu_value_for<bf16>(__bfloat162float(__float2bfloat16_rn(e[i])));
                                put8(slab + SLAB_BYTES, chunk, e);
                            } else if constexpr (EPILOGUE == Epilogue::GeluGrad) {
                                // (a plain shared-memory load: load8 reads global memory only)
                                const uint4 x = *reinterpret_cast<const uint4*>(my_slabs + SLAB_BYTES + swizzled_chunk(lane, chunk));
                                const uint32_t pairs[4] = {x.x, x.y, x.z, x.w};
                                float xs[8];
#pragma unroll
                                for (int i = 0; i < 4; ++i) {
                                    xs[2 * i] = __uint_as_float(pairs[i] << 16);
                                    xs[2 * i + 1] = __uint_as_float(pairs[i] & 0xffff0000u);
                                }
#pragma unroll
                                for (int i = 0; i < 8; ++i) e[i] = gelu_grad_value_for<bf16>(xs[i], __bfloat162float(__float2bfloat16_rn(e[i])));
                                put8(slab, chunk, e);
                            } else {
                                put8(slab, chunk, e);
                            }
                        }
                    }
                } else {
                    float v[32];
                    columns(c0, v);
#pragma unroll
                    for (uint32_t j = 0; j < 32; j += 4)
                        *reinterpret_cast<float4*>(slab + swizzled_chunk(lane, j >> 2)) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
                }
                if (args.c_tma) {
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) {
                        store_tile(&maps.c[w.product], smem_u32(slab), gn0, first_row, w.splits > 1 ? 0u : w.z_inner, w.splits > 1 ? w.split : w.z_outer);
                        if (EPILOGUE == Epilogue::Gelu) store_tile(&maps.beside, smem_u32(slab + SLAB_BYTES), gn0, first_row, 0, 0);
                        // The warp has read its slab of the argument: the next one may land there.
                        if (EPILOGUE == Epilogue::GeluGrad && c0 + 64 < static_cast<uint32_t>(T::COLUMNS) && gn0 + 64 < w.n) {
                            mbar_expect_tx(beside_bar, SLAB_BYTES);
                            load_tile<1>(smem_u32(my_slabs + SLAB_BYTES), &maps.beside, beside_bar, gn0 + 64, first_row, 0, 0);
                        }
                    }
                    continue;
                }
                // C cannot be a TMA target: the slab's rows one after the other, a lane a column.
                __syncwarp();
                for (uint32_t row = 0; row < 32 && first_row + row < w.m; ++row) {
                    const uint64_t at = out_at + static_cast<uint64_t>(first_row + row) * w.ldc;
                    for (uint32_t c = lane; c < slab_columns; c += 32) {
                        if (gn0 + c >= w.n) continue;
                        if (half_out)
                            static_cast<bf16*>(w.c)[at + gn0 + c] = *reinterpret_cast<const bf16*>(slab + swizzled_chunk(row, c >> 3) + (c & 7u) * 2);
                        else
                            static_cast<float*>(w.c)[at + gn0 + c] = *reinterpret_cast<const float*>(slab + swizzled_chunk(row, c >> 2) + (c & 3u) * 4);
                    }
                }
                __syncwarp();
            }
            // The warp's share of the accumulator and of the bias has been read.
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) arrive_first<CG>(smem_u32(&acc_empty[acc]));
        }
        // The slabs must outlive the stores that read them (and the load, if a role gave up, that fills one).
        if (lane == 0) tma_store_wait_read<0>();
        if (EPILOGUE == Epilogue::GeluGrad && !alive && lane == 0)
            for (uint32_t spin = 0; spin < WAIT_LIMIT && !mbar_try_wait(beside_bar, besides & 1u); ++spin) {}
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncwarp();
    if constexpr (CG == 2) cluster_barrier();  // the pair's remote arrivals have landed before either CTA goes away
    else __syncthreads();
    if (warp == 1) tmem_dealloc<CG>(tmem_base, T::TMEM_COLUMNS);
}

// The sum of the split-k partial tiles, ascending split order, into C (either type) with the bias.
__global__ void splitk_reduce_bf16_kernel(const float* ws, void* c, uint32_t out_half, uint64_t m, uint32_t n,
                                          uint32_t ldc, uint32_t splits, const float* bias) {
    after_producers();
    const uint64_t count = m * n, stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < count; i += stride) {
        float acc = ws[i];
        for (uint32_t s = 1; s < splits; ++s) acc += ws[static_cast<uint64_t>(s) * count + i];
        const uint32_t col = static_cast<uint32_t>(i % n);
        if (bias) acc += bias[col];
        const uint64_t at = i / n * ldc + col;
        if (out_half) static_cast<__nv_bfloat16*>(c)[at] = __float2bfloat16_rn(acc);
        else static_cast<float*>(c)[at] = acc;
    }
}

template <int CG, int BN, bool A_MN, bool B_MN, Epilogue EPILOGUE, class A, class M> void launch(cudaStream_t s, const A& args, const M& maps) {
    using T = Tile<CG, BN>;
    auto kernel = bf16_kernel<CG, BN, A_MN, B_MN, EPILOGUE, A, M>;
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
    check(cudaLaunchKernelEx(&config, kernel, args, maps), "matmul_bf16");
}
template <int CG, int BN, Epilogue EPILOGUE, class A, class M> void launch_form(cudaStream_t s, bool a_mn, bool b_mn, const A& args, const M& maps) {
    if (a_mn && b_mn) launch<CG, BN, true, true, EPILOGUE>(s, args, maps);
    else if (a_mn) launch<CG, BN, true, false, EPILOGUE>(s, args, maps);
    else if (b_mn) launch<CG, BN, false, true, EPILOGUE>(s, args, maps);
    else launch<CG, BN, false, false, EPILOGUE>(s, args, maps);
}
template <Epilogue EPILOGUE, class A, class M> void launch_tile(cudaStream_t s, uint32_t bn, bool a_mn, bool b_mn, const A& args, const M& maps) {
    if (bn == 256) launch_form<2, 256, EPILOGUE>(s, a_mn, b_mn, args, maps);
    else if (bn == 128) launch_form<1, 128, EPILOGUE>(s, a_mn, b_mn, args, maps);
    else launch_form<1, 64, EPILOGUE>(s, a_mn, b_mn, args, maps);
}

// `rows` rows of `cols` contiguous elements (bf16, or f32 for a result), `pitch` apart, inner x outer such
// matrices, as a tensor map of boxes of 128 bytes by `box_rows` rows: coordinates (column, row, inner, outer).
bool addressable(const void* base, uint64_t pitch, uint64_t inner_stride, uint64_t outer_stride, uint64_t unit) {
    return reinterpret_cast<uintptr_t>(base) % 16 == 0 && pitch % unit == 0 && inner_stride % unit == 0 && outer_stride % unit == 0;
}
CUtensorMap encode_tiles(const void* base, bool f32, uint64_t cols, uint64_t rows, uint64_t pitch, uint64_t inner, uint64_t inner_stride, uint64_t outer,
                         uint64_t outer_stride, uint32_t box_rows, const char* what) {
    const uint64_t bytes = f32 ? 4 : 2;
    if (!addressable(base, pitch, inner_stride, outer_stride, 16 / bytes))
        throw std::invalid_argument(std::string("matmul_bf16: operand ") + what + " is not a TMA source (base on 16 bytes, pitch and batch strides multiples of 16 bytes)");
    // A dimension of one element may carry any stride.
    const uint64_t whole = pitch * rows;
    const cuuint64_t size[4] = {cols, rows, inner, outer};
    const cuuint64_t stride[3] = {pitch * bytes, (inner > 1 ? inner_stride : whole) * bytes, (outer > 1 ? outer_stride : whole) * bytes};
    const cuuint32_t box[4] = {static_cast<cuuint32_t>(128 / bytes), box_rows, 1, 1}, element[4] = {1, 1, 1, 1};
    CUtensorMap map;
    const CUresult r = encode_tiled()(&map, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), size, stride,
                                      box, element, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) throw std::invalid_argument(std::string("matmul_bf16: cuTensorMapEncodeTiled refused operand ") + what + " (" + std::to_string(static_cast<int>(r)) + ")");
    return map;
}
// A: stored [m, k] (K-major: loads of 128 rows) or [k, m] (MN-major: loads of 64 k rows); B: stored
// [n, k] (K-major: loads of a CTA's columns) or [k, n] (MN-major).
CUtensorMap encode_a(const HalfMatrix& a, uint64_t m, uint64_t k, uint32_t inner, uint32_t outer) {
    return a.transposed ? encode_tiles(a.base, false, m, k, a.pitch, inner, a.stride_inner, outer, a.stride_outer, 64, "A")
                        : encode_tiles(a.base, false, k, m, a.pitch, inner, a.stride_inner, outer, a.stride_outer, 128, "A");
}
CUtensorMap encode_b(const HalfMatrix& b, uint64_t n, uint64_t k, uint32_t inner, uint32_t outer, uint32_t rows) {
    return b.transposed ? encode_tiles(b.base, false, k, n, b.pitch, inner, b.stride_inner, outer, b.stride_outer, rows, "B")
                        : encode_tiles(b.base, false, n, k, b.pitch, inner, b.stride_inner, outer, b.stride_outer, 64, "B");
}

}  // namespace

// Tile and k split by a cost model in microseconds, fitted to the times of single products with each tile
// forced: a launch's fixed part, and for each tile of a CTA (or pair) its k blocks or its drain, whichever
// is longer (the two overlap). Pairs of CTAs on 256 x 256 tiles where those keep the pairs busy, else
// 128-row tiles 128 or 64 wide; a product with too few tiles for the device splits its k range (weight
// gradients: few tiles, k = the batch's rows). Measured, earlier 128 x 256 tiles of one CTA -> now:
// 16,384 x 768 x 3,072 73 -> 62 us (1,240 TFLOP/s), 16,384 x 3,072 x 768 75 -> 58, 4,096 x 128 x 512
// 8.5 -> 6.3, 4,096 x 512 x 128 8.3 -> 6.6.
MatmulBf16Plan matmul_bf16_plan(uint64_t m, uint64_t n, uint64_t k, uint64_t products, uint64_t chain, uint64_t batch) {
    struct Candidate {
        uint32_t bm, bn;
        double fixed, block, drain, at_once;
    };
    static const Candidate candidates[] = {{256, 256, 5.0, 0.40, 2.7, 74.0}, {128, 128, 4.2, 0.35, 1.3, 148.0}, {128, 64, 3.9, 0.33, 0.7, 148.0}};
    constexpr double kReduceFixed = 2.0, kReduceBytesPerUs = 2.5e6;
    const uint64_t kblocks = (k + BK - 1) / BK;
    MatmulBf16Plan best = {};
    double best_cost = 0.0;
    for (const Candidate& c : candidates) {
        const uint64_t tiles = (m + c.bm - 1) / c.bm * ((n + c.bn - 1) / c.bn) * products * batch;
        const uint64_t most = batch > 1 || chain > 1 ? 1 : std::max<uint64_t>(1, std::min<uint64_t>(32, kblocks / 4));
        for (uint64_t splits = 1; splits <= most; ++splits) {
            const uint64_t per = (kblocks + splits - 1) / splits;
            if (kblocks && (kblocks + per - 1) / per != splits) continue;
            double cost = c.fixed + std::ceil(static_cast<double>(tiles * splits) / c.at_once) * std::max(static_cast<double>(per * chain) * c.block, c.drain);
            if (splits > 1) cost += kReduceFixed + static_cast<double>(products * m * n * (splits + 1)) * 4.0 / kReduceBytesPerUs;
            if (best.bn != 0 && cost >= best_cost) continue;
            best_cost = cost;
            best.bn = c.bn;
            best.splits = static_cast<uint32_t>(splits);
            best.kblocks_per_split = static_cast<uint32_t>(per == 0 ? 1 : per);
        }
    }
    best.workspace_floats = best.splits > 1 ? best.splits * m * n : 0;
    return best;
}

void matmul_bf16_group(cudaStream_t s, const HalfProduct* products, uint32_t count, uint64_t m, uint64_t n, uint64_t k, uint32_t outer, uint32_t inner,
                       uint32_t chain, Epilogue epilogue, const HalfResult& beside, uint32_t* status, bool leave_partials) {
    if (m == 0 || n == 0 || outer == 0 || inner == 0 || count == 0) return;
    if (count > MAX_PRODUCTS) throw std::invalid_argument("matmul_bf16: more products than one launch carries");
    const uint64_t problems = static_cast<uint64_t>(outer) * inner;
    const uint32_t results = chain > 1 ? 1 : count;
    const MatmulBf16Plan p = matmul_bf16_plan(m, n, k, results, chain, problems);
    const bool partial = p.splits > 1;
    Args args;
    Maps maps = {};
    args.status = status;
    args.m = static_cast<uint32_t>(m);
    args.n = static_cast<uint32_t>(n);
    const HalfResult& first = products[0].c;
    args.ldc = partial ? args.n : (first.pitch ? first.pitch : args.n);
    args.splits = Divisor(p.splits);
    args.kblocks = static_cast<uint32_t>((k + BK - 1) / BK);
    args.per_split = p.kblocks_per_split;
    args.chain = chain;
    args.batch = Divisor(static_cast<uint32_t>(problems));
    args.batch_inner = Divisor(inner);
    args.c_outer = first.stride_outer;
    args.c_inner = first.stride_inner;
    args.out_half = first.half ? 1u : 0u;
    const uint32_t group = p.bn == 256 ? 2 : 1;
    args.walk = TileWalk(m, n, 128 * group, p.bn);
    const bool float_out = partial || !first.half;
    for (uint32_t g = 0; g < count; ++g) {
        const HalfProduct& q = products[g];
        maps.a[g] = encode_a(q.a, m, k, inner, outer);
        maps.b[g] = encode_b(q.b, n, k, inner, outer, p.bn / group);
        if (g >= results) continue;
        if (partial && q.workspace == nullptr) throw std::invalid_argument("matmul_bf16: a split k needs its workspace");
        args.c[g] = partial ? static_cast<void*>(q.workspace) : q.c.base;
        args.bias[g] = partial ? nullptr : q.bias;
        args.c_tma = args.c_tma && addressable(args.c[g], args.ldc, partial ? 0 : q.c.stride_inner, partial ? m * n : q.c.stride_outer, float_out ? 4 : 8);
    }
    // The result matrices as the operands are described, the split-k workspace as `splits` dense ones.
    for (uint32_t g = 0; g < results && args.c_tma; ++g)
        maps.c[g] = partial ? encode_tiles(args.c[g], true, n, m, n, 1, 0, p.splits, m * n, 32, "C")
                            : encode_tiles(args.c[g], float_out, n, m, args.ldc, inner, products[g].c.stride_inner, outer, products[g].c.stride_outer, 32, "C");
    if (epilogue != Epilogue::None) {
        if (!args.c_tma || partial || !first.half || results > 1 || problems > 1) throw std::invalid_argument("matmul_bf16: an epilogue on a result that has none");
        maps.beside = encode_tiles(beside.base, false, n, m, beside.pitch ? beside.pitch : n, 1, 0, 1, 0, 32, "beside C");
    }
    args.units = static_cast<uint32_t>(args.walk.count() * problems * p.splits * results);
    const bool a_mn = products[0].a.transposed, b_mn = !products[0].b.transposed;
    if (epilogue == Epilogue::Gelu) launch_tile<Epilogue::Gelu>(s, p.bn, a_mn, b_mn, args, maps);
    else if (epilogue == Epilogue::GeluGrad) launch_tile<Epilogue::GeluGrad>(s, p.bn, a_mn, b_mn, args, maps);
    else launch_tile<Epilogue::None>(s, p.bn, a_mn, b_mn, args, maps);
    if (partial && !leave_partials) {
        const uint64_t wanted = (m * n + 255) / 256;
        for (uint32_t g = 0; g < results; ++g) {
            const HalfResult& c = products[g].c;
            splitk_reduce_bf16_kernel<<<static_cast<uint32_t>(std::min<uint64_t>(wanted, 148 * 8)), 256, 0, s>>>(
                products[g].workspace, c.base, c.half ? 1u : 0u, m, static_cast<uint32_t>(n), c.pitch ? c.pitch : static_cast<uint32_t>(n), p.splits,
                products[g].bias);
            check_launch("splitk_reduce_bf16");
        }
    }
}

void matmul_bf16(cudaStream_t s, const HalfMatrix& a, const HalfMatrix& b, const HalfResult& c, uint64_t m, uint64_t n, uint64_t k,
                 uint32_t outer, uint32_t inner, float* workspace, const float* bias, uint32_t* status, bool leave_partials) {
    const HalfProduct one = {a, b, c, bias, workspace};
    matmul_bf16_group(s, &one, 1, m, n, k, outer, inner, 1, Epilogue::None, {}, status, leave_partials);
}

// A job's k is split so that a unit (a 128 x 128 tile of one split) gets about 16 k blocks: the jobs of a
// launch fill the device together, so a job does not have to on its own.
MatmulBf16Plan matmul_bf16_job_plan(uint64_t m, uint64_t n, uint64_t k) {
    const uint64_t kblocks = std::max<uint64_t>((k + BK - 1) / BK, 1);
    uint64_t splits = std::min<uint64_t>(std::max<uint64_t>(kblocks / 16, 1), 32);
    MatmulBf16Plan p = {};
    p.bn = 128;
    p.kblocks_per_split = static_cast<uint32_t>((kblocks + splits - 1) / splits);
    p.splits = static_cast<uint32_t>((kblocks + p.kblocks_per_split - 1) / p.kblocks_per_split);
    p.workspace_floats = p.splits * m * n;
    return p;
}

void matmul_bf16_jobs(cudaStream_t s, const HalfJob* jobs, uint32_t count, uint32_t* status) {
    if (count == 0) return;
    if (count > MAX_JOBS) throw std::invalid_argument("matmul_bf16_jobs: more jobs than one launch carries");
    JobArgs args;
    JobMaps maps = {};
    args.status = status;
    for (uint32_t j = 0; j < count; ++j) {
        const HalfJob& job = jobs[j];
        const MatmulBf16Plan p = matmul_bf16_job_plan(job.m, job.n, job.k);
        Job& to = args.jobs[args.job_count++];
        to.c = job.partial;
        to.m = static_cast<uint32_t>(job.m);
        to.n = static_cast<uint32_t>(job.n);
        to.splits = p.splits;
        to.kblocks = static_cast<uint32_t>((job.k + BK - 1) / BK);
        to.per_split = p.kblocks_per_split;
        to.first_unit = args.units;
        to.walk = TileWalk(job.m, job.n, 128, 128);
        args.units += to.walk.count() * p.splits;
        maps.a[j] = encode_a(job.a, job.m, job.k, 1, 1);
        maps.b[j] = encode_b(job.b, job.n, job.k, 1, 1, 128);
        maps.c[j] = encode_tiles(to.c, true, job.n, job.m, job.n, 1, 0, p.splits, job.m * job.n, 32, "C");
    }
    launch_form<1, 128, Epilogue::None>(s, jobs[0].a.transposed, !jobs[0].b.transposed, args, maps);
}

}  // namespace k
}  // namespace msx
