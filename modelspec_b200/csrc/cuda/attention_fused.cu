// Fused attention for mixed-precision plans: forward in one kernel, the three gradients in one.
//
// The score matrix never reaches memory. What the op computes is the reference's
// (crates/modelspec-runtime/src/cpu/interpreter.rs:1035-1119, helper :1308-1510): per sequence b,
// head a and query i, s_ij = (q_i . k_j) / sqrt(d), a softmax over the unmasked keys,
// O_i = sum_j p_ij v_j; dS = p (dP - D_i) with dP = g_i . v_j and D_i = sum_j p_ij dP_ij,
// dQ_i = scale sum_j dS_ij k_j, dK_j = scale sum_i dS_ij q_i, dV_j = sum_i p_ij g_i; a masked key has
// probability 0 and zero gradient rows. Here q, k, v, g and every result are bf16 [rows, H] read and
// written in place (row pitch H, head a at columns a d ..), all products are tcgen05.mma kind::f16
// with f32 accumulation in tensor memory on TMA-loaded tiles, and softmax statistics are f32.
//
// Every operand tile is 128 rows of 64 head columns: 128 bytes a row, 128-byte swizzle, one TMA
// load. The same bytes serve as a K-major operand (k = head columns: Q K^T, G V^T) and as an
// MN-major one (k = rows: P^T G, dS^T Q, P V, dS K), so nothing is transposed or copied.
// Probabilities and score gradients are written by the row threads as bf16, into tensor memory where
// they are the A operand of the next product as they lie, else into two such tiles of 64 keys each.
//
//   forward   one CTA per (128 queries, head, sequence); key tiles of 128 in turn: S = Q K^T into
//             tensor memory, online softmax by 128 threads (one query row each: running max and
//             sum, the row of O in registers, rescaled when the max moves), P V into tensor memory,
//             added to the registers. Writes O and per (row, head) the max and the sum.
//   backward  one CTA per (128 queries or 128 keys, head, sequence), or one per (head, sequence), at
//             most 512 keys and 512 queries: S, P from the forward's statistics, dP, dS, and the
//             products of P and dS. D_i comes from sum_c O g.
//
// Heads of up to 64 columns (a multiple of 8). Every mbarrier wait is bounded; when one runs out
// the role raises bit 1 of the status word, the other roles leave their loops, the producer waits
// (bounded) for its copies in flight, tensor memory is freed and the CTA returns.
#include "tcgen05.cuh"

namespace msx {
namespace k {

namespace {

using namespace tc;

constexpr uint32_t TILE = 128;                 // rows of a tile (queries or keys)
constexpr uint32_t TILE_BYTES = TILE * 128;    // 64 bf16 columns a row

struct FusedArgs {
    const float* mask;   // [batch, keys]
    void* out;           // forward: O; backward: unused
    float* stats;        // [(row * heads + head) * 2 + {0, 1}] = max, sum of exp
    const void* o;       // backward: the forward's O
    const void* g;       // backward: the adjoint of O (also read through its tensor map)
    void* dq;
    void* dk;
    void* dv;
    uint32_t* status;
    uint32_t batch, q_len, k_len, heads, d, h;
    float scale, scale_log2;  // 1 / sqrt(d), and times log2(e)
    CoordOrder order;    // of every [rows, H] operand's tensor map
};

// Which of the 32 keys from `first` on count (inside the sequence and not masked out): bit c for
// key first + c, the same word in every lane of the warp.
__device__ __forceinline__ uint32_t keys_that_count(const float* __restrict__ mask, uint32_t seq, uint32_t first, uint32_t k_len, uint32_t lane) {
    const uint32_t key = first + lane;
    const bool counts = key < k_len && mask[static_cast<uint64_t>(seq) * k_len + key] != 0.0f;
    return __ballot_sync(0xffffffffu, counts);
}

// The row work is bound by instructions (16,384 scores a tile), so an element gets as few as there are:
// the maximum over the products as they are, then exp(scale (x - max)) as one fused multiply-add and one
// base-2 exponential, and a mask only where one of the 32 keys is masked: -inf, whose exponential is 0.
// (A product, a difference, a product with log2(e) and a test of the mask each, before the maximum and
// again behind it, came to 27 instructions an element: forward 165 us, backward 264 at
// 32 x 12 x 512 x 64, and so 121 and 182. The forward as it is below takes 80.)
__device__ __forceinline__ void hide_masked(uint32_t (&r)[32], uint32_t counts) {
    if (counts == 0xffffffffu) return;
#pragma unroll
    for (int c = 0; c < 32; ++c)
        if (!((counts >> c) & 1u)) r[c] = 0xff800000u;
}

// One [128 rows, 64 columns] tile of a [rows, H] operand: rows row0.. of sequence `seq`, head `head`.
__device__ __forceinline__ void load_tile(uint32_t dst, const CUtensorMap* map, uint32_t bar, const CoordOrder& order, uint32_t row0,
                                          uint32_t head, uint32_t seq) {
    uint32_t upper[3];
    upper[order.row] = row0;
    upper[order.inner] = head;
    upper[order.outer] = seq;
    tma_load(dst, map, bar, 0, upper);
}

// 16 f32 values as bf16 to global memory (columns c0 .. c0 + 15 of a head's row, those below d).
__device__ __forceinline__ void store_part_bf16(void* base, uint64_t element, const float (&v)[16], uint32_t c0, uint32_t d) {
    bf16* to = static_cast<bf16*>(base) + element + c0;
#pragma unroll
    for (uint32_t c = 0; c < 16; c += 8) {
        if (c0 + c + 8 > d) break;
        float8 f;
        f.lo = make_float4(v[c], v[c + 1], v[c + 2], v[c + 3]);
        f.hi = make_float4(v[c + 4], v[c + 5], v[c + 6], v[c + 7]);
        store8(to + c, f);
    }
}

// ---- forward --------------------------------------------------------------------------------------
// A thread a query row (four row warps, a loading one and one that issues MMAs), two CTAs to an SM: what bounds the
// kernel is the exponentials (16,384 a tile at 16 a cycle and SM: half of the softmax's instruction slots), and a CTA whose
// rows wait for a product leaves them to the other one's. With four threads a row and one CTA an SM, every tile waited
// for its maxima to meet, for its scores and for its P V in turn: 5,500 cycles a tile, 3,600 now
// (32 x 12 x 512 x 64: 121 -> 80 us).
// Shared memory: Q, two stages of K and of V: 80 KB, then barriers. Tensor memory: S [0, 128), P as bf16 pairs
// [128, 192), where the tensor core reads it as the A operand of P V, and P V [192, 256).
// The rows add P_j V_j to their result one key tile late, behind the maximum of tile j + 1.
constexpr int FWD_ROW_WARPS = 4, FWD_THREADS = 32 * (FWD_ROW_WARPS + 2);
constexpr uint32_t FWD_TILES = 5 * TILE_BYTES;
constexpr uint32_t FWD_SMEM = FWD_TILES + 1024 /* alignment slack */ + 256 /* barriers */;
constexpr uint32_t FWD_TMEM = 256;

// D (+)= A (tensor memory: a lane a row, a column two bf16 elements) B (shared memory).
__device__ __forceinline__ void mma_bf16_from_tmem(uint32_t d, uint32_t a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(d), "r"(a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}

__global__ void __launch_bounds__(FWD_THREADS, 2)
attention_forward_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                         const __grid_constant__ CUtensorMap map_v, const FusedArgs args) {
    extern __shared__ char smem_raw[];
    char* tiles = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    char* q_tile = tiles;
    auto k_tile = [&](uint32_t stage) { return tiles + (1 + stage) * TILE_BYTES; };
    auto v_tile = [&](uint32_t stage) { return tiles + (3 + stage) * TILE_BYTES; };
    uint64_t* bars = reinterpret_cast<uint64_t*>(tiles + FWD_TILES);
    // S_FULL: the scores of a tile. P_READY: the rows have read them and written P. PV_FULL: P V of a tile.
    enum { Q_FULL, K_FULL0, K_FULL1, K_EMPTY0, K_EMPTY1, V_FULL0, V_FULL1, V_EMPTY0, V_EMPTY1, S_FULL, P_READY, PV_FULL, BARS };
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + BARS);
    volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(tmem_slot + 1);

    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t q0 = blockIdx.x * TILE, head = blockIdx.y, seq = blockIdx.z;
    const uint32_t key_tiles = (args.k_len + TILE - 1) / TILE;
    auto bar = [&](int which) { return smem_u32(&bars[which]); };

    if (tid == 0) {
        for (int b = 0; b < BARS; ++b) mbar_init(bar(b), b == P_READY ? static_cast<uint32_t>(FWD_ROW_WARPS) : 1u);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == FWD_ROW_WARPS + 1) tmem_alloc<1>(smem_u32(tmem_slot), FWD_TMEM);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_s = *tmem_slot, tmem_p = tmem_s + 128, tmem_pv = tmem_s + 192;
    wait_for_producers();

    if (warp == FWD_ROW_WARPS) {
        if (lane == 0) {
            bool alive = true;
            uint32_t issued_k = 0, issued_v = 0;
            mbar_expect_tx(bar(Q_FULL), TILE_BYTES);
            load_tile(smem_u32(q_tile), &map_q, bar(Q_FULL), args.order, q0, head, seq);
            for (uint32_t j = 0; j < key_tiles && alive; ++j) {
                const uint32_t stage = j & 1u, use = j >> 1;
                alive = mbar_wait(bar(K_EMPTY0 + stage), (use & 1u) ^ 1u, abort_flag, args.status);
                if (!alive) break;
                mbar_expect_tx(bar(K_FULL0 + stage), TILE_BYTES);
                load_tile(smem_u32(k_tile(stage)), &map_k, bar(K_FULL0 + stage), args.order, j * TILE, head, seq);
                ++issued_k;
                alive = mbar_wait(bar(V_EMPTY0 + stage), (use & 1u) ^ 1u, abort_flag, args.status);
                if (!alive) break;
                mbar_expect_tx(bar(V_FULL0 + stage), TILE_BYTES);
                load_tile(smem_u32(v_tile(stage)), &map_v, bar(V_FULL0 + stage), args.order, j * TILE, head, seq);
                ++issued_v;
            }
            let_next_start();
            if (!alive || *abort_flag) {
                // The copies already issued still write into this CTA's shared memory: wait (bounded).
                for (uint32_t spin = 0; spin < WAIT_LIMIT && !mbar_try_wait(bar(Q_FULL), 0); ++spin) {}
                for (uint32_t back = 1; back <= 2; ++back) {
                    if (back <= issued_k) for (uint32_t i = issued_k - back, spin = 0; spin < WAIT_LIMIT && !mbar_try_wait(bar(K_FULL0 + (i & 1u)), (i >> 1) & 1u); ++spin) {}
                    if (back <= issued_v) for (uint32_t i = issued_v - back, spin = 0; spin < WAIT_LIMIT && !mbar_try_wait(bar(V_FULL0 + (i & 1u)), (i >> 1) & 1u); ++spin) {}
                }
            }
        }
    } else if (warp == FWD_ROW_WARPS + 1) {
        const uint32_t idesc_s = instruction_descriptor(TILE, TILE, false, false);
        const uint32_t idesc_pv = instruction_descriptor(TILE, 64, false, true);
        // S_j = Q K_j^T: k runs over the 64 head columns, 16 (32 bytes of a row) per MMA.
        auto scores = [&](uint32_t j) -> bool {
            const uint32_t stage = j & 1u;
            if (!mbar_wait(bar(K_FULL0 + stage), (j >> 1) & 1u, abort_flag, args.status)) return false;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (lane == 0) {
#pragma unroll
                for (uint32_t ks = 0; ks < 4; ++ks)
                    mma_bf16(tmem_s, tile_descriptor(smem_u32(q_tile) + ks * 32, 16), tile_descriptor(smem_u32(k_tile(stage)) + ks * 32, 16), idesc_s, ks != 0);
                mma_commit(bar(K_EMPTY0 + stage));
                mma_commit(bar(S_FULL));
            }
            __syncwarp();
            return true;
        };
        bool alive = mbar_wait(bar(Q_FULL), 0, abort_flag, args.status);
        if (alive) alive = scores(0);
        for (uint32_t j = 0; j < key_tiles && alive; ++j) {
            const uint32_t stage = j & 1u;
            alive = mbar_wait(bar(P_READY), j & 1u, abort_flag, args.status);
            // The rows have read S_j: the next scores go ahead of this tile's P V.
            if (alive && j + 1 < key_tiles) alive = scores(j + 1);
            if (alive) alive = mbar_wait(bar(V_FULL0 + stage), (j >> 1) & 1u, abort_flag, args.status);
            if (!alive) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (lane == 0) {
                // k runs over the 128 keys, 16 per MMA: 8 columns of P, 16 rows (2048 bytes) of the V tile.
#pragma unroll
                for (uint32_t ks = 0; ks < 8; ++ks)
                    mma_bf16_from_tmem(tmem_pv, tmem_p + ks * 8, tile_descriptor(smem_u32(v_tile(stage)) + ks * 2048, TILE_BYTES), idesc_pv, ks != 0);
                mma_commit(bar(V_EMPTY0 + stage));
                mma_commit(bar(PV_FULL));
            }
            __syncwarp();
        }
    } else {
        // Row q0 + t is lane t of tensor memory.
        const uint32_t t = warp * 32 + lane, lane_base = (warp * 32u) << 16, row = q0 + t;
        float best = -INFINITY, total = 0.0f;  // best: of the products q . k, before the scale
        float o[64];
#pragma unroll
        for (int c = 0; c < 64; ++c) o[c] = 0.0f;
        bool alive = true;
        // o_j = o_j-1 * shrink_j + P_j V_j, with the factor by which the maximum moved at tile j.
        float pending_shrink = 0.0f;
        auto add_product = [&](uint32_t j) -> bool {
            const bool ok = __all_sync(0xffffffffu, mbar_wait(bar(PV_FULL), j & 1u, abort_flag, args.status));
            if (!ok) return false;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            uint32_t pv[2][32];
            tmem_load32(tmem_pv + lane_base, pv[0]);
            tmem_load32(tmem_pv + lane_base + 32, pv[1]);
            tmem_loaded();
#pragma unroll
            for (int c = 0; c < 64; ++c) o[c] = fmaf(o[c], pending_shrink, __uint_as_float(pv[c / 32][c % 32]));
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            return true;
        };
        for (uint32_t j = 0; j < key_tiles; ++j) {
            uint32_t counts[4];
#pragma unroll
            for (uint32_t c = 0; c < 4; ++c) counts[c] = keys_that_count(args.mask, seq, j * TILE + c * 32, args.k_len, lane);
            alive = __all_sync(0xffffffffu, mbar_wait(bar(S_FULL), j & 1u, abort_flag, args.status));
            if (!alive) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            // The scores are read twice, for the maximum and for the exponentials: a row of them would take every
            // register that the row of O leaves.
            float most[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll 1
            for (uint32_t c = 0; c < 4; c += 2) {
                uint32_t r[2][32];
                tmem_load32(tmem_s + lane_base + c * 32, r[0]);
                tmem_load32(tmem_s + lane_base + c * 32 + 32, r[1]);
                tmem_loaded();
                hide_masked(r[0], c == 0 ? counts[0] : counts[2]);
                hide_masked(r[1], c == 0 ? counts[1] : counts[3]);
#pragma unroll
                for (int i = 0; i < 32; ++i) most[i & 3] = fmaxf(most[i & 3], fmaxf(__uint_as_float(r[0][i]), __uint_as_float(r[1][i])));
            }
            const float new_best = fmaxf(best, fmaxf(fmaxf(most[0], most[1]), fmaxf(most[2], most[3])));
            // exp(-inf - -inf) never forms: a row that has seen no key yet keeps zeros.
            const float shrink = best == -INFINITY ? 0.0f : exp2_fast((best - new_best) * args.scale_log2);
            const float shift = new_best == -INFINITY ? 0.0f : new_best * args.scale_log2;
            best = new_best;
            // The product of the tile before; with it, P's columns are free.
            if (j > 0) {
                alive = add_product(j - 1);
                if (!alive) break;
            }
            float sums[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 1
            for (uint32_t c = 0; c < 4; c += 2) {
                uint32_t r[2][32];
                tmem_load32(tmem_s + lane_base + c * 32, r[0]);
                tmem_load32(tmem_s + lane_base + c * 32 + 32, r[1]);
                tmem_loaded();
                hide_masked(r[0], c == 0 ? counts[0] : counts[2]);
                hide_masked(r[1], c == 0 ? counts[1] : counts[3]);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t packed[16];
#pragma unroll
                    for (int i = 0; i < 32; i += 2) {
                        const float a = exp2_fast(fmaf(__uint_as_float(r[h][i]), args.scale_log2, -shift));
                        const float b = exp2_fast(fmaf(__uint_as_float(r[h][i + 1]), args.scale_log2, -shift));
                        sums[i & 2] += a;
                        sums[(i & 2) + 1] += b;
                        const __nv_bfloat162 pair = __floats2bfloat162_rn(a, b);
                        packed[i / 2] = *reinterpret_cast<const uint32_t*>(&pair);
                    }
                    tmem_store(tmem_p + lane_base + (c + h) * 16, packed);
                }
            }
            tmem_stored();
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(P_READY));
            total = fmaf(total, shrink, (sums[0] + sums[1]) + (sums[2] + sums[3]));
            pending_shrink = shrink;
        }
        if (alive && key_tiles > 0) alive = add_product(key_tiles - 1);
        if (alive && row < args.q_len) {
            const float inverse = total > 0.0f ? 1.0f / total : 0.0f;
            const uint64_t global_row = static_cast<uint64_t>(seq) * args.q_len + row;
            bf16* const to = static_cast<bf16*>(args.out) + global_row * args.h + head * args.d;
#pragma unroll
            for (uint32_t c = 0; c < 64; c += 8) {
                if (c + 8 > args.d) break;
                store8(to + c, {make_float4(o[c] * inverse, o[c + 1] * inverse, o[c + 2] * inverse, o[c + 3] * inverse),
                                make_float4(o[c + 4] * inverse, o[c + 5] * inverse, o[c + 6] * inverse, o[c + 7] * inverse)});
            }
            if (args.stats != nullptr) {
                float* st = args.stats + (global_row * args.heads + head) * 2;
                st[0] = best * args.scale;
                st[1] = total;
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == FWD_ROW_WARPS + 1) tmem_dealloc<1>(tmem_s, FWD_TMEM);
}

// ---- backward -------------------------------------------------------------------------------------
// One launch of two kinds of CTAs, two to an SM: one per (128 queries, head, sequence) walks the keys in tiles of 64 and
// forms dQ, one per (128 keys, head, sequence) walks the queries and forms dK and dV. Both multiply their own rows X and Y
// (Q and G; K and V) by a tile's A and B (K and V; Q and G): S = X A^T and dP = Y B^T, rows of S being queries or keys. P
// and dS go back into tensor memory as bf16 pairs, the A operand of dQ += dS K, or of dV += P G and dK += dS Q.
//
// What bounds it: the latency of a step's chain (MMA, rows, MMA, rows, MMA), which a second CTA on the SM fills, and the tensor
// core's time for its narrow products. A CTA per (head, sequence) for all three gradients (below) forms no scores twice (five
// products instead of seven) but leaves most of the device idle where there are few heads: 16 heads of 512 x 48 55 -> 24 us,
// 32 of 256 x 32 17 -> 13.5, 55 of 200 x 40 19 -> 17.5.
//
// Shared memory: X, Y, three stages of (A, B): 80 KB, then barriers and the statistics of up to 512 queries.
// Tensor memory: S [0, 64), dP [64, 128), then, of queries, dS [128, 160) and dQ [160, 224); of keys, P in the columns of S
// that its own warps have read, dS in those of dP, dV [128, 192), dK [192, 256).
constexpr int BWD_ROW_WARPS = 8, BWD_THREADS = 32 * (BWD_ROW_WARPS + 2);
constexpr uint32_t BWD_STEP = 64, BWD_STEP_BYTES = BWD_STEP * 128, BWD_STAGES = 3;
constexpr uint32_t BWD_TILES = 2 * TILE_BYTES + BWD_STAGES * 2 * BWD_STEP_BYTES;
constexpr uint32_t BWD_ROWS = 512;
constexpr uint32_t BWD_SMEM = BWD_TILES + 1024 /* alignment slack */ + 256 /* barriers */ + 2 * BWD_ROWS * 4;
constexpr uint32_t BWD_TMEM = 256;

// Q, K, V, G in boxes of 128 rows and of 64.
struct BackwardMaps {
    CUtensorMap rows[4], steps[4];
};
enum { MAP_Q, MAP_K, MAP_V, MAP_G };

// 32 f32 values of a lane as bf16 pairs, in 16 columns of tensor memory.
__device__ __forceinline__ void store_packed(uint32_t at, const float (&v)[32]) {
    uint32_t packed[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const __nv_bfloat162 pair = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
        packed[i] = *reinterpret_cast<const uint32_t*>(&pair);
    }
    tmem_store(at, packed);
}

template <bool KEYS>
__device__ __forceinline__ void backward_rows(const BackwardMaps& maps, const FusedArgs& args, uint32_t row_tile, uint32_t head, uint32_t seq) {
    extern __shared__ char smem_raw[];
    char* tiles = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    char *const x_tile = tiles, *const y_tile = tiles + TILE_BYTES;
    auto a_tile = [&](uint32_t stage) { return tiles + 2 * TILE_BYTES + stage * 2 * BWD_STEP_BYTES; };
    auto b_tile = [&](uint32_t stage) { return a_tile(stage) + BWD_STEP_BYTES; };
    uint64_t* bars = reinterpret_cast<uint64_t*>(tiles + BWD_TILES);
    // S_FULL, DP_FULL: a tile's products. P_DONE (keys only), DS_DONE: the rows have written P (and read S) / dS (and read
    // dP). STEP_DONE: a tile's last product is complete. STATS_MET: every query's statistics are in shared memory.
    enum { XY_FULL, FULL0, FULL1, FULL2, EMPTY0, EMPTY1, EMPTY2, S_FULL, DP_FULL, P_DONE, DS_DONE, STEP_DONE, STATS_MET, BARS };
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + BARS);
    volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(tmem_slot + 1);
    // P = exp(score - max) / sum = 2^(x scale_log2 - shift), shift = max log2(e) + log2(sum).
    float* row_shift = reinterpret_cast<float*>(tiles + BWD_TILES + 256);  // [BWD_ROWS]
    float* row_dot = row_shift + BWD_ROWS;                                 // D_i = O_i . G_i

    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t own_len = KEYS ? args.k_len : args.q_len, other_len = KEYS ? args.q_len : args.k_len;
    const uint32_t steps = (other_len + BWD_STEP - 1) / BWD_STEP, row0 = row_tile * TILE;
    auto bar = [&](int which) { return smem_u32(&bars[which]); };

    if (tid == 0) {
        for (int b = 0; b < BARS; ++b)
            mbar_init(bar(b), (b == P_DONE || b == DS_DONE || b == STATS_MET) ? static_cast<uint32_t>(BWD_ROW_WARPS) : 1u);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == BWD_ROW_WARPS + 1) tmem_alloc<1>(smem_u32(tmem_slot), BWD_TMEM);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot, tmem_s = tmem, tmem_dp = tmem + 64;
    wait_for_producers();
    const uint32_t tmem_ds = KEYS ? tmem_dp : tmem + 128, tmem_dq = tmem + 160, tmem_dv = tmem + 128, tmem_dk = tmem + 192;

    if (warp == BWD_ROW_WARPS) {
        if (lane == 0) {
            bool alive = true;
            uint32_t issued = 0;
            mbar_expect_tx(bar(XY_FULL), 2 * TILE_BYTES);
            load_tile(smem_u32(x_tile), &maps.rows[KEYS ? MAP_K : MAP_Q], bar(XY_FULL), args.order, row0, head, seq);
            load_tile(smem_u32(y_tile), &maps.rows[KEYS ? MAP_V : MAP_G], bar(XY_FULL), args.order, row0, head, seq);
            for (; issued < steps; ++issued) {
                const uint32_t stage = issued % BWD_STAGES, use = issued / BWD_STAGES;
                alive = mbar_wait(bar(EMPTY0 + stage), (use & 1u) ^ 1u, abort_flag, args.status);
                if (!alive) break;
                mbar_expect_tx(bar(FULL0 + stage), 2 * BWD_STEP_BYTES);
                load_tile(smem_u32(a_tile(stage)), &maps.steps[KEYS ? MAP_Q : MAP_K], bar(FULL0 + stage), args.order, issued * BWD_STEP, head, seq);
                load_tile(smem_u32(b_tile(stage)), &maps.steps[KEYS ? MAP_G : MAP_V], bar(FULL0 + stage), args.order, issued * BWD_STEP, head, seq);
            }
            let_next_start();
            if (!alive || *abort_flag) {
                // The copies already issued still write into this CTA's shared memory: wait (bounded).
                for (uint32_t spin = 0; spin < WAIT_LIMIT && !mbar_try_wait(bar(XY_FULL), 0); ++spin) {}
                for (uint32_t back = 1; back <= BWD_STAGES && back <= issued; ++back)
                    for (uint32_t i = issued - back, spin = 0; spin < WAIT_LIMIT && !mbar_try_wait(bar(FULL0 + i % BWD_STAGES), (i / BWD_STAGES) & 1u); ++spin) {}
            }
        }
    } else if (warp == BWD_ROW_WARPS + 1) {
        const uint32_t idesc_scores = instruction_descriptor(TILE, BWD_STEP, false, false);  // X A^T, Y B^T
        const uint32_t idesc_sums = instruction_descriptor(TILE, 64, false, true);           // P G, dS Q, dS K
        // `from`: the A operand of 64 rows' worth of k, 8 columns for each 16 of them; of keys its second half lies 32
        // columns on. The tile is MN-major: 16 rows (2048 bytes) a step.
        auto sums = [&](uint32_t d, uint32_t from, uint32_t tile, bool first) {
#pragma unroll
            for (uint32_t ks = 0; ks < 4; ++ks)
                mma_bf16_from_tmem(d, from + (KEYS ? (ks >> 1) * 32 + (ks & 1u) * 8 : ks * 8), tile_descriptor(tile + ks * 2048, BWD_STEP_BYTES), idesc_sums,
                                   !first || ks != 0);
        };
        bool alive = mbar_wait(bar(XY_FULL), 0, abort_flag, args.status);
        // S and dP of step t, once its tile is there.
        auto scores = [&](uint32_t t) -> bool {
            const uint32_t stage = t % BWD_STAGES;
            if (!mbar_wait(bar(FULL0 + stage), (t / BWD_STAGES) & 1u, abort_flag, args.status)) return false;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (lane == 0) {
                const uint32_t x = smem_u32(x_tile), y = smem_u32(y_tile), a = smem_u32(a_tile(stage)), b = smem_u32(b_tile(stage));
#pragma unroll
                for (uint32_t ks = 0; ks < 4; ++ks) mma_bf16(tmem_s, tile_descriptor(x + ks * 32, 16), tile_descriptor(a + ks * 32, 16), idesc_scores, ks != 0);
                mma_commit(bar(S_FULL));
#pragma unroll
                for (uint32_t ks = 0; ks < 4; ++ks) mma_bf16(tmem_dp, tile_descriptor(y + ks * 32, 16), tile_descriptor(b + ks * 32, 16), idesc_scores, ks != 0);
                mma_commit(bar(DP_FULL));
            }
            __syncwarp();
            return true;
        };
        if (alive) alive = scores(0);
        for (uint32_t t = 0; t < steps && alive; ++t) {
            const uint32_t stage = t % BWD_STAGES;
            if (KEYS) {
                alive = mbar_wait(bar(P_DONE), t & 1u, abort_flag, args.status);
                if (!alive) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (lane == 0) sums(tmem_dv, tmem_s, smem_u32(b_tile(stage)), t == 0);
                __syncwarp();
            }
            alive = mbar_wait(bar(DS_DONE), t & 1u, abort_flag, args.status);
            if (!alive) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            // Of queries the next step's scores go ahead of this one's dQ (dS has columns of its own); of keys they wait for
            // the products that read P and dS out of their columns.
            if (!KEYS && t + 1 < steps) alive = scores(t + 1);
            if (!alive) break;
            if (lane == 0) {
                sums(KEYS ? tmem_dk : tmem_dq, tmem_ds, smem_u32(a_tile(stage)), t == 0);
                mma_commit(bar(EMPTY0 + stage));
                mma_commit(bar(STEP_DONE));
            }
            __syncwarp();
            if (KEYS && t + 1 < steps) {
                alive = mbar_wait(bar(STEP_DONE), t & 1u, abort_flag, args.status);
                if (alive) alive = scores(t + 1);
            }
        }
    } else {
        // Row row0 + r is lane r of tensor memory; two threads share it, 32 columns of a step each.
        const uint32_t quarter = warp & 3u, half = warp >> 2, r = quarter * 32 + lane, lane_base = (quarter * 32u) << 16, row = row0 + r;
        bool alive = true;
        // The statistics: of this block's queries (a row's thread of the first half), or of all the sequence's.
        float own_shift = INFINITY, own_dot = 0.0f;
        auto statistics = [&](uint32_t query, float* shift, float* dot) {
            *shift = INFINITY;  // a row past the end, or of masked keys alone: its probabilities are zeros
            *dot = 0.0f;
            if (query >= args.q_len) return;
            const uint64_t global_row = static_cast<uint64_t>(seq) * args.q_len + query;
            const float* const st = args.stats + (global_row * args.heads + head) * 2;
            const float best = load_global(st), total = load_global(st + 1);
            if (total > 0.0f) *shift = fmaf(best, 1.4426950408889634f, log2f(total));
            const bf16* o = static_cast<const bf16*>(args.o) + global_row * args.h + head * args.d;
            const bf16* g = static_cast<const bf16*>(args.g) + global_row * args.h + head * args.d;
            float sum = 0.0f;
            for (uint32_t c = 0; c + 8 <= args.d; c += 8) {
                const float8 a = load8(o + c), b = load8(g + c);
                sum = fmaf(a.lo.x, b.lo.x, sum); sum = fmaf(a.lo.y, b.lo.y, sum); sum = fmaf(a.lo.z, b.lo.z, sum); sum = fmaf(a.lo.w, b.lo.w, sum);
                sum = fmaf(a.hi.x, b.hi.x, sum); sum = fmaf(a.hi.y, b.hi.y, sum); sum = fmaf(a.hi.z, b.hi.z, sum); sum = fmaf(a.hi.w, b.hi.w, sum);
            }
            *dot = sum;
        };
        bool counted = true;
        if (KEYS) {
            for (uint32_t query = tid; query < steps * BWD_STEP; query += 32 * BWD_ROW_WARPS) statistics(query, &row_shift[query], &row_dot[query]);
            counted = row < args.k_len && load_global(args.mask + static_cast<uint64_t>(seq) * args.k_len + row) != 0.0f;
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(STATS_MET));
            alive = __all_sync(0xffffffffu, mbar_wait(bar(STATS_MET), 0, abort_flag, args.status));
        } else {
            statistics(row, &own_shift, &own_dot);
        }
        for (uint32_t t = 0; t < steps && alive; ++t) {
            const uint32_t first = t * BWD_STEP + half * 32;
            uint32_t counts = 0xffffffffu;
            if (!KEYS) counts = keys_that_count(args.mask, seq, first, args.k_len, lane);
            alive = __all_sync(0xffffffffu, mbar_wait(bar(S_FULL), t & 1u, abort_flag, args.status));
            if (!alive) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            uint32_t raw[32];
            float p[32];
            tmem_load32(tmem_s + lane_base + half * 32, raw);
            tmem_loaded();
            if (!KEYS) hide_masked(raw, counts);
#pragma unroll
            for (int c = 0; c < 32; c += 4) {
                float4 shift = make_float4(own_shift, own_shift, own_shift, own_shift);
                if (KEYS) shift = *reinterpret_cast<const float4*>(row_shift + first + c);
                const float by[4] = {shift.x, shift.y, shift.z, shift.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    p[c + i] = exp2_fast(fmaf(__uint_as_float(raw[c + i]), args.scale_log2, -by[i]));
                    if (KEYS && !counted) p[c + i] = 0.0f;
                }
            }
            if (KEYS) {
                store_packed(tmem_s + lane_base + half * 32, p);
                tmem_stored();
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(bar(P_DONE));
            }
            alive = mbar_wait(bar(DP_FULL), t & 1u, abort_flag, args.status);
            // (dS's columns of queries are free once the dQ of the step before has been formed)
            if (!KEYS && alive && t > 0) alive = mbar_wait(bar(STEP_DONE), (t - 1) & 1u, abort_flag, args.status);
            alive = __all_sync(0xffffffffu, alive);
            if (!alive) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            tmem_load32(tmem_dp + lane_base + half * 32, raw);
            tmem_loaded();
#pragma unroll
            for (int c = 0; c < 32; c += 4) {
                float4 dot = make_float4(own_dot, own_dot, own_dot, own_dot);
                if (KEYS) dot = *reinterpret_cast<const float4*>(row_dot + first + c);
                // dS, its scale left to dK and dQ
                p[c] = p[c] * (__uint_as_float(raw[c]) - dot.x);
                p[c + 1] = p[c + 1] * (__uint_as_float(raw[c + 1]) - dot.y);
                p[c + 2] = p[c + 2] * (__uint_as_float(raw[c + 2]) - dot.z);
                p[c + 3] = p[c + 3] * (__uint_as_float(raw[c + 3]) - dot.w);
            }
            store_packed(tmem_ds + lane_base + half * (KEYS ? 32 : 16), p);
            tmem_stored();
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(DS_DONE));
        }
        // The sums, 32 columns a thread.
        if (alive && steps > 0) alive = __all_sync(0xffffffffu, mbar_wait(bar(STEP_DONE), (steps - 1) & 1u, abort_flag, args.status));
        if (alive) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint64_t at = (static_cast<uint64_t>(seq) * own_len + row) * args.h + head * args.d;
#pragma unroll
            for (int which = 0; which < (KEYS ? 2 : 1); ++which) {
                uint32_t raw[32];
                tmem_load32((KEYS ? (which == 0 ? tmem_dv : tmem_dk) : tmem_dq) + lane_base + half * 32, raw);
                tmem_loaded();
                void* const to = KEYS ? (which == 0 ? args.dv : args.dk) : args.dq;
                const float by = KEYS && which == 0 ? 1.0f : args.scale;
                if (to == nullptr || row >= own_len) continue;
#pragma unroll
                for (uint32_t part = 0; part < 2; ++part) {
                    float v[16];
#pragma unroll
                    for (int c = 0; c < 16; ++c) v[c] = __uint_as_float(raw[part * 16 + c]) * by;
                    store_part_bf16(to, at, v, half * 32 + part * 16, args.d);
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == BWD_ROW_WARPS + 1) tmem_dealloc<1>(tmem, BWD_TMEM);
}

__global__ void __launch_bounds__(BWD_THREADS, 2) attention_backward_kernel(const __grid_constant__ BackwardMaps maps, const __grid_constant__ FusedArgs args) {
    // (the blocks that take longer go first)
    const uint32_t key_tiles = args.dk || args.dv ? (args.k_len + TILE - 1) / TILE : 0;
    if (blockIdx.x < key_tiles) backward_rows<true>(maps, args, blockIdx.x, blockIdx.y, blockIdx.z);
    else backward_rows<false>(maps, args, blockIdx.x - key_tiles, blockIdx.y, blockIdx.z);
}

// 32 f32 values of row `row`, columns chunk * 32 .., as bf16 into a pair of [128 rows, 64 columns]
// tiles (columns 0-63 in the first, 64-127 in the second) in the layout the tensor core reads.
__device__ __forceinline__ void store_chunk_bf16(char* tile_pair, uint32_t row, uint32_t chunk, const float (&v)[32]) {
    char* to = tile_pair + (chunk >> 1) * TILE_BYTES;
    const uint32_t first16 = (chunk & 1u) * 4;  // 16-byte chunk index of column chunk * 32 within its tile row
#pragma unroll
    for (int c = 0; c < 32; c += 8) {
        float8 f;
        f.lo = make_float4(v[c], v[c + 1], v[c + 2], v[c + 3]);
        f.hi = make_float4(v[c + 4], v[c + 5], v[c + 6], v[c + 7]);
        store8(reinterpret_cast<bf16*>(to + swizzled_chunk(row, first16 + (c >> 3))), f);
    }
}

// ---- backward, one CTA per (head, sequence) --------------------------------------------------------
// All three gradients of a head in one CTA: no scores are formed twice, but all of tensor memory is taken and one CTA an SM
// works through the pairs of tiles in turn. The faster way where heads fill the device several times over
// (`whole_heads_pay`). Four threads a row: 32 score columns, 16 result columns each.
constexpr int WHOLE_ROW_WARPS = 16, WHOLE_THREADS = 64 + 32 * WHOLE_ROW_WARPS;
// Shared memory: K_j, V_j, two stages of (Q_i, G_i), P (two tiles), dS (two tiles): 160 KB; then
// barriers and the row statistics of every query (the shift of its exponents, D).
// Tensor memory (512 columns): S / dP [0, 128), dV [128, 192), dK [192, 256), dQ_i [256 + 64 i, ..).
constexpr uint32_t WHOLE_TILES = 10 * TILE_BYTES;
constexpr uint32_t WHOLE_SMEM = WHOLE_TILES + 1024 /* alignment slack */ + 256 /* barriers */ + 2 * BWD_ROWS * 4;
constexpr uint32_t WHOLE_TMEM = 512;

__global__ void __launch_bounds__(WHOLE_THREADS, 1)
attention_backward_whole_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                          const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_g, const FusedArgs args) {
    extern __shared__ char smem_raw[];
    char* tiles = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    char* k_tile = tiles;
    char* v_tile = tiles + TILE_BYTES;
    auto q_tile = [&](uint32_t stage) { return tiles + (2 + 2 * stage) * TILE_BYTES; };
    auto g_tile = [&](uint32_t stage) { return tiles + (3 + 2 * stage) * TILE_BYTES; };
    char* p_tile = tiles + 6 * TILE_BYTES;
    char* ds_tile = tiles + 8 * TILE_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(tiles + WHOLE_TILES);
    // KV_FULL/KV_EMPTY: the key tile's K and V. QG_FULL/QG_EMPTY [2]: a stage of Q_i and G_i. S_FULL,
    // DP_FULL: the S / dP region holds a product. P_DONE, DS_DONE: the row threads have written P
    // (and are done with S) / dS. P_FREE, DS_FREE: the MMAs that read the P / dS tiles are complete.
    // ACC_FULL: dV_j and dK_j are complete; ACC_EMPTY: they have been drained. DQ_FULL: everything is.
    // STATS_MET: every row's statistics are in shared memory.
    enum { KV_FULL, KV_EMPTY, QG_FULL0, QG_FULL1, QG_EMPTY0, QG_EMPTY1, S_FULL, DP_FULL, P_DONE, DS_DONE, P_FREE, DS_FREE, ACC_FULL, ACC_EMPTY,
           DQ_FULL, STATS_MET, BARS };
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + BARS);
    volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(tmem_slot + 1);
    // P = exp(score - max) / sum = 2^(x scale_log2 - shift), shift = max log2(e) + log2(sum).
    float* row_shift = reinterpret_cast<float*>(tiles + WHOLE_TILES + 256);  // [BWD_ROWS]
    float* row_dot = row_shift + BWD_ROWS;                                 // D_i

    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t head = blockIdx.x, seq = blockIdx.y;
    const uint32_t key_tiles = (args.k_len + TILE - 1) / TILE, query_tiles = (args.q_len + TILE - 1) / TILE;
    auto bar = [&](int which) { return smem_u32(&bars[which]); };

    if (tid == 0) {
        for (int b = 0; b < BARS; ++b)
            mbar_init(bar(b), (b == P_DONE || b == DS_DONE || b == ACC_EMPTY || b == STATS_MET) ? static_cast<uint32_t>(WHOLE_ROW_WARPS) : 1u);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(WHOLE_TMEM) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tmem_sp = tmem_base, tmem_dv = tmem_base + 128, tmem_dk = tmem_base + 192, tmem_dq = tmem_base + 256;
    wait_for_producers();

    if (warp == 0) {
        if (lane == 0) {
            bool alive = true;
            uint32_t pair = 0;  // (j, i) pairs issued so far: stage = pair & 1
            uint32_t armed = 0, armed_phase = 0;  // bit 0 KV, bits 1-2 the QG stages
            for (uint32_t j = 0; j < key_tiles && alive; ++j) {
                alive = mbar_wait(bar(KV_EMPTY), (j & 1u) ^ 1u, abort_flag, args.status);
                if (!alive) break;
                mbar_expect_tx(bar(KV_FULL), 2 * TILE_BYTES);
                load_tile(smem_u32(k_tile), &map_k, bar(KV_FULL), args.order, j * TILE, head, seq);
                load_tile(smem_u32(v_tile), &map_v, bar(KV_FULL), args.order, j * TILE, head, seq);
                armed |= 1u;
                armed_phase = (armed_phase & ~1u) | (j & 1u);
                for (uint32_t i = 0; i < query_tiles; ++i, ++pair) {
                    const uint32_t stage = pair & 1u, use = pair >> 1;
                    alive = mbar_wait(bar(QG_EMPTY0 + stage), (use & 1u) ^ 1u, abort_flag, args.status);
                    if (!alive) break;
                    mbar_expect_tx(bar(QG_FULL0 + stage), 2 * TILE_BYTES);
                    load_tile(smem_u32(q_tile(stage)), &map_q, bar(QG_FULL0 + stage), args.order, i * TILE, head, seq);
                    load_tile(smem_u32(g_tile(stage)), &map_g, bar(QG_FULL0 + stage), args.order, i * TILE, head, seq);
                    armed |= 2u << stage;
                    armed_phase = (armed_phase & ~(2u << stage)) | ((use & 1u) << (1 + stage));
                }
            }
            let_next_start();
            if (!alive) {
                if (armed & 1u) for (uint32_t spin = 0; spin < WAIT_LIMIT && !mbar_try_wait(bar(KV_FULL), armed_phase & 1u); ++spin) {}
                for (uint32_t stage = 0; stage < 2; ++stage)
                    if (armed & (2u << stage))
                        for (uint32_t spin = 0; spin < WAIT_LIMIT && !mbar_try_wait(bar(QG_FULL0 + stage), (armed_phase >> (1 + stage)) & 1u); ++spin) {}
            }
        }
    } else if (warp == 1) {
        const uint32_t idesc_scores = instruction_descriptor(TILE, TILE, false, false);   // Q K^T, G V^T
        const uint32_t idesc_keys = instruction_descriptor(TILE, 64, true, true);         // P^T G, dS^T Q
        const uint32_t idesc_queries = instruction_descriptor(TILE, 64, false, true);     // dS K
        bool alive = true;
        uint32_t pair = 0;
        // S = Q_i K_j^T of a pair, once its Q and G are there.
        auto scores = [&](uint32_t of) -> bool {
            const uint32_t stage = of & 1u;
            if (!mbar_wait(bar(QG_FULL0 + stage), (of >> 1) & 1u, abort_flag, args.status)) return false;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (lane == 0) {
#pragma unroll
                for (uint32_t ks = 0; ks < 4; ++ks)
                    mma_bf16(tmem_sp, tile_descriptor(smem_u32(q_tile(stage)) + ks * 32, 16), tile_descriptor(smem_u32(k_tile) + ks * 32, 16), idesc_scores, ks != 0);
                mma_commit(bar(S_FULL));
            }
            __syncwarp();
            return true;
        };
        for (uint32_t j = 0; j < key_tiles && alive; ++j) {
            alive = mbar_wait(bar(KV_FULL), j & 1u, abort_flag, args.status);
            // dV_j and dK_j start from zero: the previous key tile's must have been drained.
            if (alive) alive = mbar_wait(bar(ACC_EMPTY), (j & 1u) ^ 1u, abort_flag, args.status);
            for (uint32_t i = 0; i < query_tiles && alive; ++i, ++pair) {
                const uint32_t stage = pair & 1u, ph = pair & 1u;
                const uint32_t q_at = smem_u32(q_tile(stage)), g_at = smem_u32(g_tile(stage));
                if (i == 0) alive = scores(pair);
                if (!alive) break;
                // The row threads have read S and written P: dP may take the region, P^T G may read P.
                alive = mbar_wait(bar(P_DONE), ph, abort_flag, args.status);
                if (!alive) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (lane == 0) {
#pragma unroll
                    for (uint32_t ks = 0; ks < 4; ++ks)
                        mma_bf16(tmem_sp, tile_descriptor(g_at + ks * 32, 16), tile_descriptor(smem_u32(v_tile) + ks * 32, 16), idesc_scores, ks != 0);
                    mma_commit(bar(DP_FULL));
                    // dV_j += P^T G_i: m = keys (two panels of 64, 16 KB apart), k = the 128 queries, 16 rows per MMA.
#pragma unroll
                    for (uint32_t ks = 0; ks < 8; ++ks)
                        mma_bf16(tmem_dv, tile_descriptor(smem_u32(p_tile) + ks * 2048, TILE_BYTES), tile_descriptor(g_at + ks * 2048, TILE_BYTES),
                                 idesc_keys, (i | ks) != 0);
                    mma_commit(bar(P_FREE));
                }
                __syncwarp();
                alive = mbar_wait(bar(DS_DONE), ph, abort_flag, args.status);
                if (!alive) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                // The row threads have read dP as well: the next queries' S goes ahead of this pair's dK and
                // dQ, which then run under its softmax.
                if (i + 1 < query_tiles) alive = scores(pair + 1);
                if (!alive) break;
                if (lane == 0) {
                    // dK_j += dS^T Q_i, and dQ_i += dS K_j: k = the 128 keys, 16 per MMA (32 bytes of
                    // a dS row, 16 rows of the K tile).
#pragma unroll
                    for (uint32_t ks = 0; ks < 8; ++ks)
                        mma_bf16(tmem_dk, tile_descriptor(smem_u32(ds_tile) + ks * 2048, TILE_BYTES), tile_descriptor(q_at + ks * 2048, TILE_BYTES),
                                 idesc_keys, (i | ks) != 0);
#pragma unroll
                    for (uint32_t ks = 0; ks < 8; ++ks)
                        mma_bf16(tmem_dq + 64 * i, tile_descriptor(smem_u32(ds_tile) + (ks >> 2) * TILE_BYTES + (ks & 3u) * 32, 16),
                                 tile_descriptor(smem_u32(k_tile) + ks * 2048, TILE_BYTES), idesc_queries, (j | ks) != 0);
                    mma_commit(bar(DS_FREE));
                    mma_commit(bar(QG_EMPTY0 + stage));
                    if (i + 1 == query_tiles) {
                        mma_commit(bar(ACC_FULL));
                        mma_commit(bar(KV_EMPTY));
                        if (j + 1 == key_tiles) mma_commit(bar(DQ_FULL));
                    }
                }
                __syncwarp();
            }
        }
    } else {
        // Four threads a row of a tile (lane t of tensor memory): score columns chunk * 32 .., and
        // columns chunk * 16 .. of the gradients when they are drained.
        const uint32_t quarter = warp & 3u, chunk = (warp - 2) >> 2, t = quarter * 32 + lane;
        const uint32_t lane_base = (quarter * 32u) << 16;
        bool alive = true;
        // Row statistics of every query of this (sequence, head), one row a thread: the forward's
        // max and sum, and D = sum_c O g over the head's columns.
        {
            const uint32_t row = chunk * TILE + t;
            float shift = INFINITY, dot = 0.0f;  // +inf: a row past the end, or of masked keys alone: its probabilities are zeros
            if (row < args.q_len) {
                const uint64_t global_row = static_cast<uint64_t>(seq) * args.q_len + row;
                const float* st = args.stats + (global_row * args.heads + head) * 2;
                if (st[1] > 0.0f) shift = fmaf(st[0], 1.4426950408889634f, log2f(st[1]));
                const bf16* o = static_cast<const bf16*>(args.o) + global_row * args.h + head * args.d;
                const bf16* g = static_cast<const bf16*>(args.g) + global_row * args.h + head * args.d;
                for (uint32_t c = 0; c + 8 <= args.d; c += 8) {
                    const float8 a = load8(o + c), b = load8(g + c);
                    dot = fmaf(a.lo.x, b.lo.x, dot); dot = fmaf(a.lo.y, b.lo.y, dot); dot = fmaf(a.lo.z, b.lo.z, dot); dot = fmaf(a.lo.w, b.lo.w, dot);
                    dot = fmaf(a.hi.x, b.hi.x, dot); dot = fmaf(a.hi.y, b.hi.y, dot); dot = fmaf(a.hi.z, b.hi.z, dot); dot = fmaf(a.hi.w, b.hi.w, dot);
                }
            }
            row_shift[row] = shift;
            row_dot[row] = dot;
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(STATS_MET));
            alive = mbar_wait(bar(STATS_MET), 0, abort_flag, args.status);
            alive = __all_sync(0xffffffffu, alive);
        }
        uint32_t pair = 0;
        for (uint32_t j = 0; j < key_tiles && alive; ++j) {
            const uint32_t counts = keys_that_count(args.mask, seq, j * TILE + chunk * 32, args.k_len, lane);
            for (uint32_t i = 0; i < query_tiles; ++i, ++pair) {
                const uint32_t ph = pair & 1u;
                const uint32_t row = i * TILE + t;
                const float shift = row_shift[row], dot = row_dot[row];
                alive = mbar_wait(bar(S_FULL), ph, abort_flag, args.status);
                // The P tile is free once the P^T G of the previous pair has been read by the tensor core.
                if (alive) alive = mbar_wait(bar(P_FREE), ph ^ 1u, abort_flag, args.status);
                alive = __all_sync(0xffffffffu, alive);
                if (!alive) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                uint32_t r[32];
                tmem_load32(tmem_sp + lane_base + chunk * 32, r);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                hide_masked(r, counts);
                float p[32];
#pragma unroll
                for (int c = 0; c < 32; ++c) p[c] = exp2_fast(fmaf(__uint_as_float(r[c]), args.scale_log2, -shift));
                store_chunk_bf16(p_tile, t, chunk, p);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(bar(P_DONE));
                alive = mbar_wait(bar(DP_FULL), ph, abort_flag, args.status);
                if (alive) alive = mbar_wait(bar(DS_FREE), ph ^ 1u, abort_flag, args.status);
                alive = __all_sync(0xffffffffu, alive);
                if (!alive) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                tmem_load32(tmem_sp + lane_base + chunk * 32, r);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int c = 0; c < 32; ++c) p[c] = p[c] * (__uint_as_float(r[c]) - dot);  // dS, its scale left to dK and dQ
                store_chunk_bf16(ds_tile, t, chunk, p);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(bar(DS_DONE));
            }
            if (!alive) break;
            // dV_j and dK_j are complete: rows are keys now. Drain them, then free the accumulators.
            alive = mbar_wait(bar(ACC_FULL), j & 1u, abort_flag, args.status);
            alive = __all_sync(0xffffffffu, alive);
            if (!alive) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t key = j * TILE + t;
            const uint64_t key_at = (static_cast<uint64_t>(seq) * args.k_len + key) * args.h + head * args.d;
#pragma unroll
            for (int which = 0; which < 2; ++which) {
                uint32_t raw[16];
                tmem_load((which == 0 ? tmem_dv : tmem_dk) + lane_base + chunk * 16, raw);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                float v[16];
#pragma unroll
                for (int c = 0; c < 16; ++c) v[c] = __uint_as_float(raw[c]) * (which == 0 ? 1.0f : args.scale);
                void* to = which == 0 ? args.dv : args.dk;
                if (to != nullptr && key < args.k_len) store_part_bf16(to, key_at, v, chunk * 16, args.d);
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(ACC_EMPTY));
        }
        if (alive) {
            alive = mbar_wait(bar(DQ_FULL), 0, abort_flag, args.status);
            alive = __all_sync(0xffffffffu, alive);
        }
        if (alive && args.dq != nullptr) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (uint32_t i = 0; i < query_tiles; ++i) {
                uint32_t raw[16];
                tmem_load(tmem_dq + 64 * i + lane_base + chunk * 16, raw);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                float v[16];
#pragma unroll
                for (int c = 0; c < 16; ++c) v[c] = __uint_as_float(raw[c]) * args.scale;
                const uint32_t row = i * TILE + t;
                if (row < args.q_len) store_part_bf16(args.dq, (static_cast<uint64_t>(seq) * args.q_len + row) * args.h + head * args.d, v, chunk * 16, args.d);
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(WHOLE_TMEM) : "memory");
}

// The tensor map of a [batch * rows, H] operand read head by head in tiles of 128 rows (or `box`).
CUtensorMap head_map(const void* base, uint32_t rows, const AttentionShape& sh, CoordOrder* order, const char* what, uint32_t box = TILE) {
    const uint32_t h = sh.heads * sh.head_dim;
    const HalfMatrix x = {base, h, static_cast<uint64_t>(rows) * h, sh.head_dim, false};
    return encode(x, sh.head_dim, rows, sh.heads, sh.batch, box, order, what);
}

FusedArgs fused_args(const float* mask, AttentionShape sh, uint32_t* status) {
    FusedArgs a = {};
    a.mask = mask;
    a.status = status;
    a.batch = sh.batch;
    a.q_len = sh.q_len;
    a.k_len = sh.k_len;
    a.heads = sh.heads;
    a.d = sh.head_dim;
    a.h = sh.heads * sh.head_dim;
    a.scale = 1.0f / sqrtf(static_cast<float>(sh.head_dim));
    a.scale_log2 = a.scale * 1.4426950408889634f;
    return a;
}

// Which kernel forms the gradients sooner, in us: a CTA a head takes 3 and 3.9 for each pair of tiles of 128, one wave an SM;
// the CTAs of 128 queries or keys 2 and, for each step of 64, 2.8 alone on an SM and 3.3 with another. Measured (a CTA a head,
// CTAs of rows): 384 heads of 512 x 64 181, 266; 16 of 512 x 48 55, 24; 32 of 256 x 32 17, 13.5; 55 of 200 x 40 19, 17.5; 512 of
// 64 x 64 30.7, 28.4; 768 of 16 x 64 40.9, 35.
bool whole_heads_pay(const AttentionShape& sh) {
    constexpr uint64_t SMS = 148;
    auto up = [](uint64_t x, uint64_t to) { return (x + to - 1) / to; };
    const uint64_t heads = static_cast<uint64_t>(sh.batch) * sh.heads, tiles_q = up(sh.q_len, TILE), tiles_k = up(sh.k_len, TILE);
    const double whole = static_cast<double>(up(heads, SMS)) * (3.0 + 3.9 * static_cast<double>(tiles_q * tiles_k));
    const uint64_t blocks = heads * (tiles_q + tiles_k), steps = up(std::max(sh.q_len, sh.k_len), BWD_STEP);
    const double rows = static_cast<double>(up(blocks, 2 * SMS)) * (2.0 + (blocks <= SMS ? 2.8 : 3.3) * static_cast<double>(steps));
    return whole <= rows;
}

template <class K> void opt_in(K kernel, uint32_t bytes) {
    check(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes)), "attention_fused shared memory");
}

}  // namespace

bool attention_fused_supported(AttentionShape sh) {
    return sh.head_dim <= 64 && sh.head_dim % 8 == 0 && sh.k_len <= BWD_ROWS && sh.q_len <= BWD_ROWS && sh.batch > 0 && sh.q_len > 0;
}

uint64_t attention_fused_stats_floats(AttentionShape sh) { return static_cast<uint64_t>(sh.batch) * sh.q_len * sh.heads * 2; }

void attention_fused_forward(cudaStream_t s, const void* q, const void* k, const void* v, const float* mask, void* out, float* stats,
                             AttentionShape sh, uint32_t* status) {
    if (!attention_fused_supported(sh)) throw std::invalid_argument("attention_fused_forward: heads of up to 64 columns, up to 512 keys and queries");
    FusedArgs args = fused_args(mask, sh, status);
    args.out = out;
    args.stats = stats;
    CoordOrder order = {}, same = {};
    const CUtensorMap map_q = head_map(q, sh.q_len, sh, &order, "q");
    const CUtensorMap map_k = head_map(k, sh.k_len, sh, &same, "k");
    const CUtensorMap map_v = head_map(v, sh.k_len, sh, &same, "v");
    args.order = order;
    opt_in(attention_forward_kernel, FWD_SMEM);
    const dim3 grid((sh.q_len + TILE - 1) / TILE, sh.heads, sh.batch);
    attention_forward_kernel<<<grid, FWD_THREADS, FWD_SMEM, s>>>(map_q, map_k, map_v, args);
    check_launch("attention_fused_forward");
}

void attention_fused_backward(cudaStream_t s, const void* q, const void* k, const void* v, const float* mask, const void* g, const void* o,
                              const float* stats, void* dq, void* dk, void* dv, AttentionShape sh, uint32_t* status) {
    if (!attention_fused_supported(sh)) throw std::invalid_argument("attention_fused_backward: heads of up to 64 columns, up to 512 keys and queries");
    FusedArgs args = fused_args(mask, sh, status);
    args.stats = const_cast<float*>(stats);
    args.o = o;
    args.g = g;
    args.dq = dq;
    args.dk = dk;
    args.dv = dv;
    if (!dq && !dk && !dv) return;
    CoordOrder order = {}, same = {};
    BackwardMaps maps;
    const bool whole = whole_heads_pay(sh);
    const struct { const void* base; uint32_t rows; const char* what; } operands[4] = {{q, sh.q_len, "q"}, {k, sh.k_len, "k"}, {v, sh.k_len, "v"}, {g, sh.q_len, "g"}};
    for (int i = 0; i < 4; ++i) {
        maps.rows[i] = head_map(operands[i].base, operands[i].rows, sh, i == MAP_Q ? &order : &same, operands[i].what);
        if (!whole) maps.steps[i] = head_map(operands[i].base, operands[i].rows, sh, &same, operands[i].what, BWD_STEP);
    }
    args.order = order;
    if (whole) {
        opt_in(attention_backward_whole_kernel, WHOLE_SMEM);
        attention_backward_whole_kernel<<<dim3(sh.heads, sh.batch), WHOLE_THREADS, WHOLE_SMEM, s>>>(maps.rows[MAP_Q], maps.rows[MAP_K], maps.rows[MAP_V], maps.rows[MAP_G], args);
    } else {
        opt_in(attention_backward_kernel, BWD_SMEM);
        const dim3 grid((dk || dv ? (sh.k_len + TILE - 1) / TILE : 0) + (dq ? (sh.q_len + TILE - 1) / TILE : 0), sh.heads, sh.batch);
        attention_backward_kernel<<<grid, BWD_THREADS, BWD_SMEM, s>>>(maps, args);
    }
    check_launch("attention_fused_backward");
}

}  // namespace k
}  // namespace msx
