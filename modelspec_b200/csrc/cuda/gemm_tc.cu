// f32 matmul: the choice of kernel for a product, and the 64-row tensor-core tiles, which take what the
// other two kernels do not: operands TMA cannot address (bases or row pitches off 16 bytes) once a
// product is too large for the FMA tiles of gemm_small.cu, and batched products. gemm_tf32.cu has the
// TMA-fed tiles, gemm.cu the exact kernel of bit-level parity runs.
//
// The 64-row tiles: tcgen05.mma with the accumulator in tensor memory, f32 operands as a split-TF32
// product (tolerance class). Each f32 operand x is split into hi (its top 11 significant bits) and
// lo = x - hi, both exact tf32 values (the tensor core keeps 11 significant bits of lo, so x is
// represented to about 2^-21 |x|).
//
// On the 64-row tile the four partial products are not four MMAs: the hi and lo halves of A are
// stacked along M (64 rows each of one 128-row operand) and those of B along N (BN columns each of
// one 2 BN-wide operand). One MMA per 8-deep k slice then yields all four products, in four
// quadrants of tensor memory that the epilogue adds.
//
// One CTA computes a 64 x BN tile (BN = 32, 64 or 128) over a range of 32-deep k blocks:
//   warps 0-7  load the A and B blocks from global memory, split them and store hi and lo in the
//              128-byte-swizzled shared-memory layouts tcgen05 reads (K-major or MN-major by how
//              the operand is stored, so NN, TN and NT need no transposed copy), then drain the
//              accumulator: tcgen05.ld, the quadrant sums, row-wise stores to C or to the
//              split-K workspace;
//   warp 8     allocates tensor memory, issues 4 MMAs per k block from one thread, and releases
//              each shared-memory stage with tcgen05.commit.
//
// Shared memory stays under half an SM's (2 to 4 stages of 24 to 48 KB) and registers under
// half its file, so two CTAs share an SM and one drains while the other loads. Stage hand-off is
// by mbarriers; every wait is bounded and, when it runs out, raises bit 1 of the status word,
// makes every role leave its loop, frees the tensor memory and returns. A k range split across
// CTAs (grid.z, k blocks dealt out round-robin) writes partial tiles that `splitk_reduce_kernel`
// or the step's finalize launch adds in ascending split order (deterministic).
#include <atomic>
#include <cmath>
#include <cstdlib>

#include "common.cuh"
#include "kernels.cuh"
#include "tcgen05.cuh"

namespace msx {
namespace k {

namespace {

constexpr int BK = 32;
constexpr int LOADER_THREADS = 256, THREADS = LOADER_THREADS + 32;
constexpr uint32_t WAIT_LIMIT = 1u << 24;  // try_wait polls before a wait gives up
#ifndef MSX_TC_JOB_KBLOCKS
#define MSX_TC_JOB_KBLOCKS 32  // k blocks a unit of matmul_tc_jobs gets (BERT-tiny's 13 weight gradients on the 128 x 128 tile: 33 us with 8, 43 with 16, 34 with 32, which leaves the fewest partial tiles)
#endif

// The 64-row tile described above, two CTAs per SM.
template <int BM, int BN> struct Config {
    static_assert(BM == 64, "the stacked-A tile has 64 rows");
    static constexpr int STAGES = BN == 128 ? 2 : (BN == 64 ? 3 : 4);  // shared-memory stages
    static constexpr int SETS = BN == 32 ? 4 : (BN == 128 ? 2 : 3);    // register sets of loads in flight
    static constexpr int CTAS_PER_SM = 2;
    static constexpr uint32_t A_BYTES = 2 * BM * BK * 4;  // hi rows 0-63, lo rows 64-127
    static constexpr uint32_t B_BYTES = 2 * BN * BK * 4;  // hi columns 0..BN-1, lo columns BN..2BN-1
    static constexpr uint32_t STAGE_BYTES = A_BYTES + B_BYTES;
    static constexpr uint32_t TOTAL = STAGES * STAGE_BYTES + 1024 /* alignment slack */ + 256 /* barriers */;
    static constexpr uint32_t TMEM_COLUMNS = 2 * BN;
};

constexpr int MAX_GROUP = 4;  // products of one shape that one launch can carry
constexpr int MAX_JOBS = 24;  // products of different shapes that one launch can carry

struct TcArgs {
    // Per product of the group (grid.z = product * splits + split when not batched):
    const float* a[MAX_GROUP];
    const float* b[MAX_GROUP];
    float* c[MAX_GROUP];           // C, or the split-K workspace [splits][m][n]
    const float* bias[MAX_GROUP];  // added to every row of C by the CTA that writes C; null for none
    uint32_t splits;
    uint32_t m, n, k;
    uint32_t lda, ldb, ldc;        // row pitch, in elements, of each matrix as stored
    uint32_t a_vec, b_vec, c_vec;  // 16-byte accesses are aligned for this operand
    uint32_t c_padded;             // the columns of C between n and ldc are padding that may be overwritten
    Epilogue epilogue;             // of one product
    float* beside;
    uint32_t beside_vec;
    // Batched products: grid.z = batch index z, split as (z / inner, z % inner); each matrix of
    // problem z starts at outer * stride_outer + inner * stride_inner elements. inner = 0: not batched.
    uint32_t batch_inner;
    uint64_t a_outer, a_inner, b_outer, b_inner, c_outer, c_inner;
    uint32_t* status;
    // Products of different shapes in one launch (one storage form, one tile width): a 1-D grid
    // whose block b belongs to the job whose block range holds it; `job_count` = 0 otherwise.
    uint32_t job_count;
    struct Job {
        const float* a;
        const float* b;
        float* c;  // C, or the job's split-K workspace
        uint32_t m, n, k, lda, ldb, ldc, splits, first_block;  // first_block: the job's first block
    } jobs[MAX_JOBS];
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Waits for `parity` of `bar`; false when the wait ran out or another role gave up.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile uint32_t* abort_flag, uint32_t* status) {
    for (uint32_t spin = 0; spin < WAIT_LIMIT; ++spin) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((spin & 255u) == 255u && *abort_flag) return false;
    }
    *abort_flag = 1;
    atomicOr(status, 2u);
    return false;
}

__device__ __forceinline__ void mma_tf32(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
        ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(0u), "r"(0u), "r"(0u), "r"(0u)
        : "memory");
}

__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// 32 lanes x 32 consecutive columns of tensor memory: r[j] = column `taddr.column + j` of this
// thread's lane.
__device__ __forceinline__ void tmem_load32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}

// Byte offset of the 16-byte chunk holding elements (row, 4 c16 .. 4 c16 + 3) of a K-major tile:
// 128-byte rows, 8-row groups of 1024 bytes, chunk index xor-ed with the row within its group.
__device__ __forceinline__ uint32_t k_major_offset(uint32_t row, uint32_t c16) {
    return (row >> 3) * 1024u + (row & 7u) * 128u + ((c16 ^ (row & 7u)) << 4);
}
// The same for an MN-major tile: for each k a 128-byte row of 32 consecutive MN elements, the
// 32 k rows of a block forming one 4096-byte panel per 32 MN elements; within a row the 32-byte
// chunk index is xor-ed with the k row modulo 4 (groups of 4 rows, 512 bytes). `c` counts 16-byte
// chunks along MN.
__device__ __forceinline__ uint32_t mn_major_offset(uint32_t krow, uint32_t c) {
    uint32_t in_panel = c & 7u;
    return (c >> 3) * (BK * 128u) + krow * 128u + (((in_panel >> 1) ^ (krow & 3u)) << 5) + ((in_panel & 1u) << 4);
}

__device__ __forceinline__ float4 load4(const float* __restrict__ p, uint64_t index, uint32_t valid, bool vec) {
    // `valid` = how many of the 4 elements from `index` are inside the matrix (0..4).
    // Volatile asm keeps every load where it is written: the prefetch depth is the point, and
    // the compiler otherwise sinks the loads to their first use.
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    const float* at = p + index;
    if (valid == 4 && vec) {
        asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(at));
        return v;
    }
    if (valid > 0) asm volatile("ld.global.f32 %0, [%1];" : "=f"(v.x) : "l"(at));
    if (valid > 1) asm volatile("ld.global.f32 %0, [%1];" : "=f"(v.y) : "l"(at + 1));
    if (valid > 2) asm volatile("ld.global.f32 %0, [%1];" : "=f"(v.z) : "l"(at + 2));
    if (valid > 3) asm volatile("ld.global.f32 %0, [%1];" : "=f"(v.w) : "l"(at + 3));
    return v;
}

// hi = x with the 13 mantissa bits below tf32 cleared (an exact tf32, whatever rounding the tensor
// core would apply to a wider value), lo = x - hi exactly (at most 13 significant bits, below
// 2^-10 |x|). One logic op and one subtraction per element: the split must not cost more than
// the MMAs it feeds.
__device__ __forceinline__ float top_tf32(float x) { return __uint_as_float(__float_as_uint(x) & 0xffffe000u); }

__device__ __forceinline__ void store_split(char* tile, uint32_t hi_offset, uint32_t lo_offset, float4 v) {
    float4 h, l;
    h.x = top_tf32(v.x); h.y = top_tf32(v.y); h.z = top_tf32(v.z); h.w = top_tf32(v.w);
    l.x = v.x - h.x; l.y = v.y - h.y; l.z = v.z - h.z; l.w = v.w - h.w;
    *reinterpret_cast<float4*>(tile + hi_offset) = h;
    *reinterpret_cast<float4*>(tile + lo_offset) = l;
}

__device__ __forceinline__ uint32_t in_range(uint32_t start, uint32_t limit) {
    return start >= limit ? 0u : (limit - start >= 4u ? 4u : limit - start);
}

__device__ __forceinline__ void loaders_barrier(uint32_t threads) {
    asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
}

// ACT: with an epilogue.
template <int BM, int BN, bool A_T, bool B_T, bool ACT>
__global__ void __launch_bounds__(THREADS, Config<BM, BN>::CTAS_PER_SM) matmul_tc_kernel(TcArgs args) {
    using Cfg = Config<BM, BN>;
    constexpr int STAGES = Cfg::STAGES, SETS = Cfg::SETS;
    extern __shared__ char smem_raw[];
    // Tiles need 1024-byte alignment for the swizzle pattern to line up with address bits.
    char* tiles = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(tiles + STAGES * Cfg::STAGE_BYTES);
    // bars[0 .. STAGES) full, bars[STAGES .. 2 STAGES) empty, bars[2 STAGES] accumulator ready;
    // then the TMEM address and the abort flag.
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 1);
    volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(bars + 2 * STAGES + 2);

    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // The problem this CTA works on: the launch's own, or one job of a launch that carries several.
    uint32_t pm = args.m, pn = args.n, pk = args.k, plda = args.lda, pldb = args.ldb, pldc = args.ldc, psplits = args.splits;
    uint32_t tile_x = blockIdx.x, tile_y = blockIdx.y, tile_z = blockIdx.z;
    const float* job_a = nullptr;
    const float* job_b = nullptr;
    float* job_c = nullptr;
    if (args.job_count) {
        uint32_t j = 0;
        while (j + 1 < args.job_count && args.jobs[j + 1].first_block <= blockIdx.x) ++j;
        const TcArgs::Job& job = args.jobs[j];
        pm = job.m; pn = job.n; pk = job.k; plda = job.lda; pldb = job.ldb; pldc = job.ldc; psplits = job.splits;
        job_a = job.a; job_b = job.b; job_c = job.c;
        const uint32_t local = blockIdx.x - job.first_block, across = (pn + BN - 1) / BN, down = (pm + BM - 1) / BM;
        tile_x = local % across;
        tile_y = (local / across) % down;
        tile_z = local / (across * down);
    }
    const uint32_t m0 = tile_y * BM, n0 = tile_x * BN;
    const uint32_t kblocks_total = (pk + BK - 1) / BK;
    const bool batched = args.batch_inner != 0;
    const uint32_t z_outer = batched ? tile_z / args.batch_inner : 0, z_inner = batched ? tile_z % args.batch_inner : 0;
    const uint32_t product = (batched || args.job_count) ? 0 : tile_z / psplits, split = batched ? 0 : tile_z % psplits;
    // A split k is dealt out block by block: split s takes k blocks s, s + splits, ... The CTAs of
    // the splits of one tile run side by side, so at any time they read neighbouring 128-byte
    // pieces of the same operand rows (one DRAM page) instead of pieces a whole k range apart.
    const uint32_t stride = batched ? 1u : psplits;
    const uint32_t kblocks = kblocks_total > split ? (kblocks_total - split + stride - 1) / stride : 0;

    // ---- loaders, first part: where this thread's chunks sit, and the first loads. They are issued
    // before the barriers and the tensor memory are set up, so that the set-up hides under them.
    const float* __restrict__ a = job_a ? job_a : args.a[product] + z_outer * args.a_outer + z_inner * args.a_inner;
    const float* __restrict__ b = job_b ? job_b : args.b[product] + z_outer * args.b_outer + z_inner * args.b_inner;
    constexpr int A_CHUNKS = BM * BK / 4 / LOADER_THREADS, B_CHUNKS = BN * BK / 4 / LOADER_THREADS;
    // Where this thread's chunks sit in a block does not depend on the block: the shared-memory
    // offsets, the address of each chunk in the first k block and whether all four of its elements
    // lie inside the matrix rows are computed once. A k block that lies wholly inside k then costs
    // one pointer addition and one 16-byte load per chunk: address arithmetic and bounds checks
    // per block would be as many instructions again as the split itself. The lo half of an operand
    // lies half the operand's bytes after the hi half (64 rows, BN rows, or as many 32-element
    // panels).
    uint32_t aoff[A_CHUNKS], boff[B_CHUNKS];
    const float* a_at[A_CHUNKS];
    const float* b_at[B_CHUNKS];
    bool a_whole[A_CHUNKS], b_whole[B_CHUNKS];
    constexpr uint32_t a_per_k_row = BM / 4, b_per_k_row = BN / 4;  // 16-byte chunks of one k row of an MN-major tile
    auto a_place = [&](int i, uint32_t* row, uint32_t* col) {
        const uint32_t q = tid + i * LOADER_THREADS;
        if (A_T) { *row = q / a_per_k_row; *col = (q % a_per_k_row) * 4; }  // (k, m)
        else     { *row = q >> 3; *col = (q & 7u) * 4; }                    // (m, k)
    };
    auto b_place = [&](int i, uint32_t* row, uint32_t* col) {
        const uint32_t q = tid + i * LOADER_THREADS;
        if (B_T) { *row = q >> 3; *col = (q & 7u) * 4; }                    // (n, k)
        else     { *row = q / b_per_k_row; *col = (q % b_per_k_row) * 4; }  // (k, n)
    };
    const uint32_t first_k = split * BK;
#pragma unroll
    for (int i = 0; i < A_CHUNKS; ++i) {
        uint32_t row, col;
        a_place(i, &row, &col);
        aoff[i] = A_T ? mn_major_offset(row, col / 4) : k_major_offset(row, col / 4);
        a_at[i] = A_T ? a + static_cast<uint64_t>(first_k + row) * plda + m0 + col
                      : a + static_cast<uint64_t>(m0 + row) * plda + first_k + col;
        a_whole[i] = args.a_vec && (A_T ? m0 + col + 4 <= pm : m0 + row < pm);
    }
#pragma unroll
    for (int i = 0; i < B_CHUNKS; ++i) {
        uint32_t row, col;
        b_place(i, &row, &col);
        boff[i] = B_T ? k_major_offset(row, col / 4) : mn_major_offset(row, col / 4);
        b_at[i] = B_T ? b + static_cast<uint64_t>(n0 + row) * pldb + first_k + col
                      : b + static_cast<uint64_t>(first_k + row) * pldb + n0 + col;
        b_whole[i] = args.b_vec && (B_T ? n0 + row < pn : n0 + col + 4 <= pn);
    }
    // Elements from one k block of this CTA to its next.
    const uint64_t a_step = static_cast<uint64_t>(BK) * stride * (A_T ? plda : 1u);
    const uint64_t b_step = static_cast<uint64_t>(BK) * stride * (B_T ? 1u : pldb);
    auto fetch = [&](uint32_t kb, float4 (&av)[A_CHUNKS], float4 (&bv)[B_CHUNKS]) {
        const uint32_t k0 = (kb * stride + split) * BK;
        const bool inside = k0 + BK <= pk;
#pragma unroll
        for (int i = 0; i < A_CHUNKS; ++i) {
            if (inside && a_whole[i]) {
                av[i] = load4(a_at[i] + kb * a_step, 0, 4, true);
                continue;
            }
            uint32_t row, col;
            a_place(i, &row, &col);
            if (A_T) {  // stored [k, m]: 4 consecutive m of one k row
                uint32_t gk = k0 + row, gm = m0 + col;
                uint32_t valid = gk < pk ? in_range(gm, pm) : 0u;
                av[i] = load4(a, static_cast<uint64_t>(gk) * plda + gm, valid, args.a_vec);
            } else {    // stored [m, k]: 4 consecutive k of one row
                uint32_t gm = m0 + row, gk = k0 + col;
                uint32_t valid = gm < pm ? in_range(gk, pk) : 0u;
                av[i] = load4(a, static_cast<uint64_t>(gm) * plda + gk, valid, args.a_vec);
            }
        }
#pragma unroll
        for (int i = 0; i < B_CHUNKS; ++i) {
            if (inside && b_whole[i]) {
                bv[i] = load4(b_at[i] + kb * b_step, 0, 4, true);
                continue;
            }
            uint32_t row, col;
            b_place(i, &row, &col);
            if (B_T) {  // stored [n, k]
                uint32_t gn = n0 + row, gk = k0 + col;
                uint32_t valid = gn < pn ? in_range(gk, pk) : 0u;
                bv[i] = load4(b, static_cast<uint64_t>(gn) * pldb + gk, valid, args.b_vec);
            } else {    // stored [k, n]
                uint32_t gk = k0 + row, gn = n0 + col;
                uint32_t valid = gk < pk ? in_range(gn, pn) : 0u;
                bv[i] = load4(b, static_cast<uint64_t>(gk) * pldb + gn, valid, args.b_vec);
            }
        }
    };
    // SETS register sets: the loads of the next SETS - 1 blocks are in flight while a block is
    // split and stored.
    float4 av[SETS][A_CHUNKS], bv[SETS][B_CHUNKS];
    // The four bias values this thread adds in the epilogue, fetched with the first loads: a load
    // issued in the epilogue would be a round trip to memory with nothing to hide behind.
    const float* __restrict__ bias_row = (job_c || args.job_count) ? nullptr : args.bias[product];
    float bias_mine[4] = {0.f, 0.f, 0.f, 0.f};
    wait_for_producers();
    if (warp < 8) {
        if (bias_row) {
            const uint32_t gn = n0 + (lane % (BN / 4)) * 4;
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (gn + q < pn) bias_mine[q] = load_global(bias_row + gn + q);
        }
#pragma unroll
        for (int s = 0; s < SETS - 1; ++s)
            if (static_cast<uint32_t>(s) < kblocks) fetch(s, av[s], bv[s]);
    }

    if (tid == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(smem_u32(&bars[s]), LOADER_THREADS);
            mbar_init(smem_u32(&bars[STAGES + s]), 1);
        }
        mbar_init(smem_u32(&bars[2 * STAGES]), 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 8) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(Cfg::TMEM_COLUMNS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;

    if (warp < 8) {
        // ---- loaders: global -> (hi, lo) -> swizzled shared memory ---------------------------
        bool alive = true;
        auto deposit = [&](uint32_t kb, const float4 (&a_regs)[A_CHUNKS], const float4 (&b_regs)[B_CHUNKS]) -> bool {
            const uint32_t stage = kb % STAGES, round = kb / STAGES;
            char* a_tile = tiles + stage * Cfg::STAGE_BYTES;
            char* b_tile = a_tile + Cfg::A_BYTES;
            // The stage is free once the MMAs that read its previous contents have completed.
            if (!mbar_wait(smem_u32(&bars[STAGES + stage]), (round & 1u) ^ 1u, abort_flag, args.status)) return false;
#pragma unroll
            for (int i = 0; i < A_CHUNKS; ++i) store_split(a_tile, aoff[i], aoff[i] + Cfg::A_BYTES / 2, a_regs[i]);
#pragma unroll
            for (int i = 0; i < B_CHUNKS; ++i) store_split(b_tile, boff[i], boff[i] + Cfg::B_BYTES / 2, b_regs[i]);
            // Make the generic-proxy stores visible to the tensor core's async-proxy reads.
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            mbar_arrive(smem_u32(&bars[stage]));
            return true;
        };
        for (uint32_t kb0 = 0; kb0 < kblocks && alive; kb0 += SETS) {
#pragma unroll
            for (int s = 0; s < SETS; ++s) {
                const uint32_t kb = kb0 + s;
                if (kb >= kblocks || !alive) break;
                if (kb + SETS - 1 < kblocks) fetch(kb + SETS - 1, av[(s + SETS - 1) % SETS], bv[(s + SETS - 1) % SETS]);
                alive = deposit(kb, av[s], bv[s]);
            }
        }
        let_next_start();
        // ---- epilogue: tensor memory -> shared memory -> global --------------------------------
        // Lanes 0-63 of tensor memory hold the A_hi rows, 64-127 the A_lo rows of the same 64 tile
        // rows; columns [0, BN) the products with B_hi, [BN, 2 BN) those with B_lo. A warp reads
        // its lane quarter, adds the two column halves and writes the sums, row-major, into one of
        // two shared-memory tiles (hi rows, lo rows; the stages are free by now). After a barrier
        // all eight warps add the two tiles and write C a whole tile row at a time, 16 bytes per
        // lane where the pitch of C allows.
        if (alive && kblocks > 0) alive = mbar_wait(smem_u32(&bars[2 * STAGES]), 0, abort_flag, args.status);
        alive = __all_sync(0xffffffffu, alive);  // tcgen05.ld is warp-wide: decide as a warp
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t quarter = warp & 3u, half = warp >> 2;
        constexpr int PARTS = BN == 128 ? 2 : 1;
        constexpr uint32_t PITCH = BN + 4;  // 16-byte phases of consecutive rows fall on distinct banks
        const bool drains = BN != 32 || half == 0;  // a 32-column tile is one block per lane quarter
        float* tile_hi = reinterpret_cast<float*>(tiles);
        float* tile_lo = tile_hi + 64 * PITCH;  // the sums of the A_lo rows
        if (drains) {
            // Lane quarters 0-1 hold the A_hi rows, 2-3 the A_lo rows.
            float* to_row = (quarter < 2 ? tile_hi : tile_lo) + ((quarter & 1u) * 32u + lane) * PITCH;
#pragma unroll
            for (int part = 0; part < PARTS; ++part) {
                const uint32_t col = BN == 128 ? half * 64u + part * 32u : (BN == 64 ? half * 32u : 0u);
                uint32_t r1[32], r2[32];
                if (alive && kblocks > 0) {
                    const uint32_t taddr = tmem_base + ((quarter * 32u) << 16) + col;
                    tmem_load32(taddr, r1);
                    tmem_load32(taddr + BN, r2);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                } else {
#pragma unroll
                    for (int j = 0; j < 32; ++j) { r1[j] = 0u; r2[j] = 0u; }  // an empty k range contributes zeros
                }
#pragma unroll
                for (int j = 0; j < 32; j += 4) {
                    float4 v;
                    v.x = __uint_as_float(r1[j]) + __uint_as_float(r2[j]);
                    v.y = __uint_as_float(r1[j + 1]) + __uint_as_float(r2[j + 1]);
                    v.z = __uint_as_float(r1[j + 2]) + __uint_as_float(r2[j + 2]);
                    v.w = __uint_as_float(r1[j + 3]) + __uint_as_float(r2[j + 3]);
                    *reinterpret_cast<float4*>(to_row + col + j) = v;
                }
            }
        }
        loaders_barrier(LOADER_THREADS);
        float* __restrict__ out = batched ? args.c[0] + z_outer * args.c_outer + z_inner * args.c_inner
                                          : (job_c ? job_c : args.c[product]) + static_cast<uint64_t>(split) * pm * pldc;
        constexpr uint32_t LANES_PER_ROW = BN / 4, ROWS_PER_PASS = 32 / LANES_PER_ROW;
        const uint32_t c4 = (lane % LANES_PER_ROW) * 4, gn = n0 + c4;
#pragma unroll 4
        for (uint32_t r = warp * ROWS_PER_PASS + lane / LANES_PER_ROW; r < BM; r += 8 * ROWS_PER_PASS) {
            const uint32_t gm = m0 + r;
            if (gm >= pm || gn >= pn) continue;
            const float4 h = *reinterpret_cast<const float4*>(tile_hi + r * PITCH + c4);
            const float4 l = *reinterpret_cast<const float4*>(tile_lo + r * PITCH + c4);
            // `x + 0` turns a -0 sum of zero products into the +0 a skipped term gives.
            float v[4] = {(h.x + l.x) + 0.0f, (h.y + l.y) + 0.0f, (h.z + l.z) + 0.0f, (h.w + l.w) + 0.0f};
            if (bias_row) {
#pragma unroll
                for (int q = 0; q < 4; ++q) v[q] = v[q] + bias_mine[q];
            }
            if (ACT) {
                // The second matrix has C's rows.
                float* const at = args.beside + static_cast<uint64_t>(gm) * pldc + gn;
                const bool whole = args.beside_vec && gn + 4 <= pn;
                float other[4] = {0.f, 0.f, 0.f, 0.f};
                if (args.epilogue == Epilogue::GeluGrad || args.epilogue == Epilogue::ReluGrad) {
                    if (whole) {
                        const float4 f = load_global(reinterpret_cast<const float4*>(at));
                        other[0] = f.x; other[1] = f.y; other[2] = f.z; other[3] = f.w;
                    } else {
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            if (gn + q < pn) other[q] = load_global(at + q);
                    }
#pragma unroll
                    for (int q = 0; q < 4; ++q) v[q] = args.epilogue == Epilogue::GeluGrad ? gelu_grad_value(other[q], v[q]) : relu_grad_value(other[q], v[q]);
                } else {
#pragma unroll
                    for (int q = 0; q < 4; ++q) other[q] = args.epilogue == Epilogue::Gelu ? gelu_value(v[q]) : relu_value(v[q]);
                    if (whole) {
                        *reinterpret_cast<float4*>(at) = make_float4(other[0], other[1], other[2], other[3]);
                    } else {
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            if (gn + q < pn) at[q] = other[q];
                    }
                }
            }
            float* dst = out + static_cast<uint64_t>(gm) * pldc + gn;
            // Inside the pitch a whole float4 may be written: what lies past n is padding.
            if (args.c_vec && (gn + 4 <= pn || (args.c_padded && gn + 4 <= pldc))) {
                *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (gn + q < pn) dst[q] = v[q];
            }
        }
    } else {
        // ---- the MMA warp: one thread issues, the tensor core runs asynchronously ---------------
        // Instruction descriptor: f32 accumulator, tf32 A and B, their majors, N >> 3, M >> 4, for
        // the stacked operands: M = 128 (hi and lo rows), N = 2 BN (hi and lo columns).
        const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((A_T ? 1u : 0u) << 15) | ((B_T ? 0u : 1u) << 16) |
                               (static_cast<uint32_t>((2 * BN) >> 3) << 17) | (static_cast<uint32_t>(128 >> 4) << 24);
        // The shared-memory matrix descriptor of tcgen05 (version 1): start address (bits 0-13),
        // leading (16-29) and stride (32-45) byte offsets, all in 16-byte units, bit 46 set (the
        // sm_100 version), and in bits 61-63 the swizzle of the tile: 2 = 128-byte swizzle of
        // 16-byte chunks (K-major tiles), 1 = 128-byte swizzle of 32-byte chunks, the one layout
        // the tensor core reads MN-major 32-bit operands from. The descriptors of a k block differ
        // only in the start address: everything else is built once.
        constexpr uint32_t a_lbo = A_T ? BK * 128u : 16u, b_lbo = B_T ? 16u : BK * 128u;
        constexpr uint32_t a_sbo = A_T ? 512u : 1024u, b_sbo = B_T ? 1024u : 512u;
        constexpr uint32_t a_type = A_T ? 1u : 2u, b_type = B_T ? 2u : 1u;
        constexpr uint32_t a_high = ((a_sbo >> 4) & 0x3FFFu) | (1u << 14) | (a_type << 29);
        constexpr uint32_t b_high = ((b_sbo >> 4) & 0x3FFFu) | (1u << 14) | (b_type << 29);
        constexpr uint32_t a_low = ((a_lbo >> 4) & 0x3FFFu) << 16, b_low = ((b_lbo >> 4) & 0x3FFFu) << 16;
        const uint32_t tiles16 = (smem_u32(tiles) & 0x3FFFFu) >> 4;
        auto desc = [](uint32_t high, uint32_t low) { return (static_cast<uint64_t>(high) << 32) | low; };
        bool alive = true;
        uint32_t stage = 0, parity = 0;
        for (uint32_t kb = 0; kb < kblocks && alive; ++kb) {
            alive = mbar_wait(smem_u32(&bars[stage]), parity, abort_flag, args.status);
            if (!alive) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (lane == 0) {
                const uint32_t a16 = a_low + tiles16 + stage * (Cfg::STAGE_BYTES >> 4);
                const uint32_t b16 = b_low + tiles16 + stage * (Cfg::STAGE_BYTES >> 4) + (Cfg::A_BYTES >> 4);
#pragma unroll
                for (uint32_t ks = 0; ks < BK / 8; ++ks) {
                    // One MMA covers k = 8: 32 bytes along a K-major row (8-row groups 1024 bytes
                    // apart), or 8 rows of an MN-major panel (4-row groups 512 bytes apart, panels
                    // of 32 MN elements 4096 bytes apart).
                    const uint32_t a_step = (A_T ? ks * 1024u : ks * 32u) >> 4;
                    const uint32_t b_step = (B_T ? ks * 32u : ks * 1024u) >> 4;
                    mma_tf32(tmem_base, desc(a_high, a16 + a_step), desc(b_high, b16 + b_step), idesc, (kb | ks) != 0u);
                }
                mma_commit(smem_u32(&bars[STAGES + stage]));                   // frees the stage when they finish
                if (kb + 1 == kblocks) mma_commit(smem_u32(&bars[2 * STAGES]));  // and, at the end, the accumulator
            }
            if (++stage == STAGES) { stage = 0; parity ^= 1u; }
            __syncwarp();
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 8) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(Cfg::TMEM_COLUMNS) : "memory");
    }
}

__global__ void splitk_reduce_kernel(const float* ws, float* c, uint64_t count, uint32_t splits,
                                     const float* bias, uint32_t n) {
    after_producers();
    uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < count; i += stride) {
        float acc = ws[i];
        for (uint32_t s = 1; s < splits; ++s) acc += ws[static_cast<uint64_t>(s) * count + i];
        c[i] = bias ? acc + bias[i % n] : acc;
    }
}

template <int BM, int BN, bool ACT, bool A_T, bool B_T> void launch(cudaStream_t s, const TcArgs& args, dim3 grid) {
    auto kernel = matmul_tc_kernel<BM, BN, A_T, B_T, ACT>;
    static std::atomic<int> configured_device{-1};
    set_shared_memory(kernel, static_cast<int>(Config<BM, BN>::TOTAL), configured_device);
    kernel<<<grid, THREADS, Config<BM, BN>::TOTAL, s>>>(args);
    check_launch("matmul_tc");
}

template <int BM, int BN, bool ACT> void launch_forms(cudaStream_t s, const TcArgs& args, dim3 grid, bool a_t, bool b_t) {
    if (a_t && b_t) launch<BM, BN, ACT, true, true>(s, args, grid);
    else if (a_t) launch<BM, BN, ACT, true, false>(s, args, grid);
    else if (b_t) launch<BM, BN, ACT, false, true>(s, args, grid);
    else launch<BM, BN, ACT, false, false>(s, args, grid);
}

template <bool ACT> void launch_tile(cudaStream_t s, const TcArgs& args, dim3 grid, uint32_t bn, bool a_t, bool b_t) {
    if (bn == 32) launch_forms<64, 32, ACT>(s, args, grid, a_t, b_t);
    else if (bn == 64) launch_forms<64, 64, ACT>(s, args, grid, a_t, b_t);
    else launch_forms<64, 128, ACT>(s, args, grid, a_t, b_t);
}

bool aligned16(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

}  // namespace

// Which kernel, tile and k split by a cost model in microseconds, fitted to measured times of single
// products (64 x 10 x 128 to 16,384 x 3,072 x 768, all storage forms): a launch's fixed part (set-up,
// first loads, last drain), a part per k block, one per tile, and the bytes all SMs pull through the L2.
// The 64-row tiles' figures are fitted to 470 products on rows off 16 bytes (24 to 50,000 a side), each timed with
// every tile and up to 36 splits: the choice is 1.8 % above the fastest on average (4.9 % with the figures
// before, 1.47 times it at most: 92 x 17,609 x 2,207 took 178 us on narrow tiles, 122 on wide ones).
//   * small tiles on the FMA units while the product fits a few of them per SM;
//   * operands TMA can address: 128-row tiles 32, 64 or 128 wide (the narrow ones when the wide ones would
//     leave SMs idle), or pairs of CTAs on 256 x 256 tiles once there are enough of those;
//   * the rest, and empty products, the 64-row tiles of this file.
// A split k adds the reduce launch and its partial tiles.
MatmulTcPlan matmul_tc_plan(uint64_t m, uint64_t n, uint64_t k, uint64_t problems, uint64_t group, bool tma_ok, uint64_t chain, bool batched) {
    enum Kernel { Fma, Tma, Rows64 };
    struct Candidate {
        Kernel kernel;
        uint32_t bm, bn;
        double fixed, block, tile;  // per launch, per k block of a tile, per tile
        double at_once;             // tiles the device works on at a time
    };
    static const Candidate candidates[] = {
        {Fma, 32, 32, 3.5, 1.2, 0.0, 0.0},
        {Tma, 128, 32, 4.2, 0.51, 0.25, 148.0},
        {Tma, 128, 64, 4.55, 0.52, 0.4, 148.0},
        {Tma, 128, 128, 5.3, 0.6, 1.1, 148.0},
        {Tma, 256, 256, 7.2, 1.02, 1.3, 74.0},
        // Two CTAs share an SM; a k block takes at least the last figure of an SM's time.
        {Rows64, 64, 32, 3.5, 0.25, 0.60, 296.0},
        {Rows64, 64, 64, 3.5, 0.47, 0.38, 296.0},
        {Rows64, 64, 128, 3.5, 0.80, 0.45, 296.0},
    };
    constexpr uint64_t kDeepest = 96;
    const uint64_t kblocks = (k + BK - 1) / BK;
    MatmulTcPlan best = {};
    double best_cost = 0.0;
    for (const Candidate& c : candidates) {
        if (c.kernel == Fma ? batched || kblocks == 0 || chain > 1 : (c.kernel == Tma) != (kblocks > 0 && tma_ok)) continue;
        const bool rows64 = c.kernel == Rows64;
        if (rows64 && c.bn > 32 && c.bn / 2 >= n) continue;  // a narrower tile holds the same columns
        const double bytes_per_us = rows64 ? 8.3e6 : 7.0e6, reduce_fixed = rows64 ? 1.7 : 2.0, reduce_bytes_per_us = rows64 ? 7.3e6 : 2.5e6;
        const uint64_t m_tiles = (m + c.bm - 1) / c.bm, n_tiles = (n + c.bn - 1) / c.bn, tiles = m_tiles * n_tiles * problems * group;
        auto consider = [&](double cost, uint64_t splits, uint64_t per, uint32_t cluster) {
            // (A split product's second launch is a microsecond more beside the one launch of the FMA tiles.)
            if (best.bn != 0 && cost + (rows64 && best.fma && splits > 1 ? 1.0 : 0.0) >= best_cost) return;
            best_cost = cost;
            best = MatmulTcPlan{c.bm, c.bn, static_cast<uint32_t>(splits), static_cast<uint32_t>(per == 0 ? 1 : per), c.kernel == Fma, cluster, 0};
        };
        if (c.kernel == Fma) {
            // As many CTAs to a tile as leave every group one slab; what all tiles together ask of the SMs
            // (0.22 us a slab of a tile) bounds it from the other side.
            const uint64_t slabs = (k + 15) / 16;
            uint32_t cluster = 1;
            while (cluster < 8 && slabs > 8 * cluster && tiles * cluster * 2 <= 296) cluster *= 2;
            const double chain = c.fixed + (cluster > 1 ? 0.8 : 0.0) + static_cast<double>((slabs + 8 * cluster - 1) / (8 * cluster) - 1) * c.block;
            const double streamed = 2.6 + static_cast<double>(tiles * slabs) / 148.0 * 0.22;
            consider(chain > streamed ? chain : streamed, 1, kblocks, cluster);
            continue;
        }
        const uint64_t most = batched || chain > 1 ? 1 : (kblocks / 2 > 0 ? kblocks / 2 : 1);
        for (uint64_t splits = 1; splits <= most && splits <= 64; ++splits) {
            const uint64_t per = (kblocks + splits - 1) / splits;
            const uint64_t used = kblocks == 0 ? 1 : (kblocks + per - 1) / per;
            if (used != splits) continue;  // the same partition as a smaller count
            const double waves = std::ceil(static_cast<double>(tiles * splits) / c.at_once);
            double cost;
            if (c.kernel == Tma) {
                cost = c.fixed + waves * (static_cast<double>(per * chain) * c.block + c.tile);
            } else {
                const double paired = waves * (c.fixed + static_cast<double>(per) * c.block);
                const double streamed = std::ceil(static_cast<double>(tiles * splits) / 148.0) * static_cast<double>(per) * c.tile;
                cost = paired > streamed ? paired : streamed;
                // These tiles sum their k in tensor memory, which truncates: no deeper than 96 k blocks (7e-6 of a
                // product's norm; 139 in one sum 1.1e-5) where k can be split.
                if (per > kDeepest && most > 1) cost *= 4.0;
            }
            // Every tile reads its rows of A and columns of B over k.
            const double bytes = 4.0 * static_cast<double>(problems * group) *
                                 (static_cast<double>(m * k * n_tiles) + static_cast<double>(n * k * m_tiles) + static_cast<double>(m * n * splits));
            const double traffic = bytes / bytes_per_us;
            if (traffic > cost) cost = traffic;
            if (splits > 1) cost += reduce_fixed + static_cast<double>(m * n * (splits + 1)) * 4.0 / reduce_bytes_per_us;
            consider(cost, splits, per, 1);
        }
    }
    best.workspace_floats = best.splits > 1 ? best.splits * m * n : 0;
    return best;
}

void matmul_tc_group(cudaStream_t s, const MatmulOperands* products, uint32_t count, bool a_t, bool b_t, uint64_t m, uint64_t n,
                     uint64_t k, uint32_t* status, bool leave_partials, MatmulPitches pitches, Epilogue epilogue, float* beside) {
    if (m == 0 || n == 0 || count == 0) return;
    if (count > MAX_GROUP) throw std::invalid_argument("matmul_tc_group: more products than one launch carries");
    // The TMA-fed tiles want bases on 16 bytes and rows a multiple of 16 bytes apart.
    bool tma_ok = (pitches.a ? pitches.a : (a_t ? m : k)) % 4 == 0 && (pitches.b ? pitches.b : (b_t ? k : n)) % 4 == 0;
    for (uint32_t g = 0; g < count; ++g) tma_ok = tma_ok && aligned16(products[g].a) && aligned16(products[g].b);
    MatmulTcPlan p = matmul_tc_plan(m, n, k, 1, count, tma_ok);
    if (pitches.c && p.splits > 1) throw std::invalid_argument("matmul_tc_group: a pitched result with a split k");
    if (epilogue != Epilogue::None && (count != 1 || pitches.c || !beside || !matmul_takes_epilogue(p)))
        throw std::invalid_argument("matmul_tc_group: an epilogue for one dense product on the small tiles");
    if (p.fma) {
        matmul_small(s, p, products, count, a_t, b_t, m, n, k, pitches, epilogue, beside);
    } else if (p.bm >= 128) {
        matmul_tf32(s, p, products, count, a_t, b_t, m, n, k, 1, pitches, status);
    } else {
        TcArgs args = {};
        args.m = static_cast<uint32_t>(m);
        args.n = static_cast<uint32_t>(n);
        args.k = static_cast<uint32_t>(k);
        args.lda = pitches.a ? pitches.a : static_cast<uint32_t>(a_t ? m : k);
        args.ldb = pitches.b ? pitches.b : static_cast<uint32_t>(b_t ? k : n);
        // Partial tiles of a split k are dense; the pitch of C applies to the CTAs that write C itself.
        args.ldc = (pitches.c && p.splits == 1) ? pitches.c : static_cast<uint32_t>(n);
        args.splits = p.splits;
        // A float4 read starts at a multiple of 4 elements within a row, so rows must keep that phase.
        args.a_vec = args.lda % 4 == 0;
        args.b_vec = args.ldb % 4 == 0;
        args.c_vec = args.ldc % 4 == 0;
        args.c_padded = pitches.c != 0 && p.splits == 1;
        for (uint32_t g = 0; g < count; ++g) {
            args.c_vec = args.c_vec && aligned16(p.splits > 1 ? products[g].workspace : products[g].c);
            args.a[g] = products[g].a;
            args.b[g] = products[g].b;
            args.c[g] = p.splits > 1 ? products[g].workspace : products[g].c;
            args.bias[g] = p.splits > 1 ? nullptr : products[g].bias;
            args.a_vec = args.a_vec && aligned16(products[g].a);
            args.b_vec = args.b_vec && aligned16(products[g].b);
        }
        args.status = status;
        args.epilogue = epilogue;
        args.beside = beside;
        args.beside_vec = args.ldc % 4 == 0 && aligned16(beside);
        const dim3 grid(static_cast<uint32_t>((n + p.bn - 1) / p.bn), static_cast<uint32_t>((m + p.bm - 1) / p.bm), p.splits * count);
        if (epilogue != Epilogue::None) launch_tile<true>(s, args, grid, p.bn, a_t, b_t);
        else launch_tile<false>(s, args, grid, p.bn, a_t, b_t);
    }
    if (p.splits > 1 && !leave_partials) {
        uint64_t total = m * n;
        uint64_t blocks = (total + 255) / 256;
        for (uint32_t g = 0; g < count; ++g) {
            splitk_reduce_kernel<<<static_cast<uint32_t>(blocks > 148 * 8 ? 148 * 8 : blocks), 256, 0, s>>>(
                products[g].workspace, products[g].c, total, p.splits, products[g].bias, static_cast<uint32_t>(n));
            check_launch("splitk_reduce");
        }
    }
}

void matmul_tc(cudaStream_t s, const float* a, bool a_t, const float* b, bool b_t, float* c, uint64_t m, uint64_t n,
               uint64_t k, float* workspace, uint32_t* status, const float* bias, bool leave_partials) {
    MatmulOperands one = {a, b, c, bias, workspace};
    matmul_tc_group(s, &one, 1, a_t, b_t, m, n, k, status, leave_partials);
}

// One job of matmul_tc_jobs: k split so that a unit (a 128 x 128 tile of one split, or a CTA of
// the 64 x 64 tiles where TMA cannot address the job) gets about MSX_TC_JOB_KBLOCKS k blocks (the
// jobs of a launch fill the device together, so a job does not have to on its own).
MatmulTcPlan matmul_tc_job_plan(uint64_t m, uint64_t n, uint64_t k) {
    const uint64_t kblocks = (k + BK - 1) / BK;
    uint64_t splits = kblocks / MSX_TC_JOB_KBLOCKS;
    if (splits < 1) splits = 1;
    if (splits > 32) splits = 32;
    MatmulTcPlan p = {};
    p.bm = 64;
    p.bn = 64;
    p.kblocks_per_split = static_cast<uint32_t>((kblocks + splits - 1) / splits);
    p.splits = static_cast<uint32_t>(kblocks == 0 ? 1 : (kblocks + p.kblocks_per_split - 1) / p.kblocks_per_split);
    p.workspace_floats = p.splits > 1 ? p.splits * m * n : 0;
    return p;
}

// Up to this many microseconds of FMA work. The tensor-core launch takes 8 us and 25 ns a row of the batch, the FMA
// tiles 5 us and more than their work: below the limit they win (the jobs of two layers 64 wide over 256 rows 12.5 -> 8.0 us, over
// 512 rows 16.9 -> 10.4). From 6 to 12 us of work they would win with more than about 350 rows (1,600: 49 -> 25 us) and lose
// with fewer (320: 16 -> 20 us; 80: 10 -> 19).
constexpr double kSmallJobsUs = 6.0;
void matmul_tc_jobs(cudaStream_t s, const MatmulJob* jobs, uint32_t count, bool a_t, bool b_t, uint32_t* status) {
    if (count == 0) return;
    if (count > MAX_JOBS) throw std::invalid_argument("matmul_tc_jobs: more jobs than one launch carries");
    for (uint32_t j = 0; j < count; ++j)
        if (jobs[j].m == 0 || jobs[j].n == 0) throw std::invalid_argument("matmul_tc_jobs: an empty product");
    // The FMA tiles while all jobs together are a few of them per SM (0.22 us a 16-deep slab of one), where
    // the tensor-core launch is mostly its fixed 7 us.
    double slabs = 0.0;
    for (uint32_t j = 0; j < count; ++j)
        slabs += static_cast<double>(((jobs[j].m + 31) / 32) * ((jobs[j].n + 31) / 32) * ((jobs[j].k + 15) / 16));
    if (slabs / 148.0 * 0.22 < kSmallJobsUs) {
        matmul_small_jobs(s, jobs, count, a_t, b_t);
        return;
    }
    if (matmul_tf32_jobs(s, jobs, count, a_t, b_t, status)) return;
    TcArgs args = {};
    args.splits = 1;
    args.a_vec = args.b_vec = args.c_vec = 1;
    args.status = status;
    uint32_t blocks = 0;
    for (uint32_t j = 0; j < count; ++j) {
        const MatmulJob& job = jobs[j];
        if (job.m == 0 || job.n == 0) throw std::invalid_argument("matmul_tc_jobs: an empty product");
        const MatmulTcPlan p = matmul_tc_job_plan(job.m, job.n, job.k);
        TcArgs::Job& to = args.jobs[args.job_count++];
        to.a = job.a;
        to.b = job.b;
        to.c = p.splits > 1 ? job.workspace : job.c;
        to.m = static_cast<uint32_t>(job.m);
        to.n = static_cast<uint32_t>(job.n);
        to.k = static_cast<uint32_t>(job.k);
        to.lda = static_cast<uint32_t>(a_t ? job.m : job.k);
        to.ldb = static_cast<uint32_t>(b_t ? job.k : job.n);
        to.ldc = to.n;
        to.splits = p.splits;
        to.first_block = blocks;
        blocks += static_cast<uint32_t>(((job.m + 63) / 64) * ((job.n + 63) / 64)) * p.splits;
        args.a_vec = args.a_vec && aligned16(job.a) && to.lda % 4 == 0;
        args.b_vec = args.b_vec && aligned16(job.b) && to.ldb % 4 == 0;
        args.c_vec = args.c_vec && aligned16(to.c) && to.ldc % 4 == 0;
    }
    launch_tile<false>(s, args, dim3(blocks), 64, a_t, b_t);
}

namespace {
// One batched product on the 64-row tiles: operands that TMA cannot address.
void launch_batched(cudaStream_t s, const BatchedOperand& a, const BatchedOperand& b, const BatchedOperand& c, uint64_t m, uint64_t n, uint64_t k,
                    uint32_t outer, uint32_t inner, uint32_t* status) {
    TcArgs args = {};
    args.a[0] = a.base;
    args.b[0] = b.base;
    args.c[0] = const_cast<float*>(c.base);
    args.splits = 1;
    args.m = static_cast<uint32_t>(m);
    args.n = static_cast<uint32_t>(n);
    args.k = static_cast<uint32_t>(k);
    args.lda = a.pitch;
    args.ldb = b.pitch;
    args.ldc = c.pitch;
    auto vec = [](const BatchedOperand& o) {
        return aligned16(o.base) && o.pitch % 4 == 0 && o.stride_outer % 4 == 0 && o.stride_inner % 4 == 0;
    };
    args.a_vec = vec(a);
    args.b_vec = vec(b);
    args.c_vec = vec(c);
    args.batch_inner = inner;
    args.a_outer = a.stride_outer; args.a_inner = a.stride_inner;
    args.b_outer = b.stride_outer; args.b_inner = b.stride_inner;
    args.c_outer = c.stride_outer; args.c_inner = c.stride_inner;
    args.status = status;
    const MatmulTcPlan p = matmul_tc_plan(m, n, k, static_cast<uint64_t>(outer) * inner, 1, false, 1, true);
    dim3 grid(static_cast<uint32_t>((n + p.bn - 1) / p.bn), static_cast<uint32_t>((m + p.bm - 1) / p.bm), outer * inner);
    launch_tile<false>(s, args, grid, p.bn, a.transposed, b.transposed);
}
}  // namespace

void matmul_tc_batched(cudaStream_t s, const BatchedProduct* products, uint32_t count, uint64_t m, uint64_t n, uint64_t k, uint32_t outer, uint32_t inner,
                       uint32_t* status) {
    if (m == 0 || n == 0 || outer == 0 || inner == 0 || matmul_tf32_batched(s, products, count, m, n, k, outer, inner, status)) return;
    for (uint32_t g = 0; g < count; ++g) launch_batched(s, products[g].a, products[g].b, products[g].c, m, n, k, outer, inner, status);
}

}  // namespace k
}  // namespace msx
