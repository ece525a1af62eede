// f32 attention and its gradients with the scores on the chip: heads of up to 64 columns, any strides.
//
// What the op computes is the reference's (crates/modelspec-runtime/src/cpu/interpreter.rs:1035-1119, helper
// :1308-1510; the formulas stand in attention_tc.cu). Every product is tcgen05.mma kind::tf32 on operands split
// into hi = the top 11 significant bits and lo = x - hi: hi hi + hi lo + lo hi in f32 accumulators, the two
// cross products in accumulators of their own (gemm_tf32.cu), so the tolerance class is that of the products.
//
//   forward   one CTA per (128 queries, head, sequence), key tiles of 128: S = Q K^T into tensor memory, online
//             softmax in registers (four threads a row), P back into tensor memory as hi and lo halves, where the
//             tensor core reads it as the A operand of P V. Only O and a row's maximum and sum are written.
//   backward  one launch of CTAs per (128 queries, head, sequence), over key tiles of 64, and per (128 keys, head,
//             sequence), over query tiles of 64. Each forms S and dP = G V^T (or both transposed), P from the
//             forward's statistics, dS = scale P (dP - O . G), and dQ += dS K, or dV += P^T G and dK += dS^T Q, with P and
//             dS as the A operand out of tensor memory.
//
// What bounds it: for long sequences the chain of a tile (MMA, row work, MMA), one CTA an SM; for short ones the
// latency of the launch, of which there are one forward and one backward instead of three and four. As batched
// products with row kernels between, a layer's scores cross memory four times forward and six times backward.
// A launch, us (as batched products): 64 heads of 128 x 64 forward 12.7 (20.6), backward 20.6 (28.7); 15 heads of 77 x 33
// 11.3 (17.6), 19.8 (33.4); 32 heads of 256 x 32 14.5 (24.8), 24.8 (34.9); 384 heads of 512 x 64 322 (395), 985 (615:
// which way a shape goes is decided at the end of this file).
// Operands come through registers, which split them on the way to shared memory (so no alignment is asked for):
// K-major tiles in the 128-byte swizzle of 16-byte chunks; V, and K where it is contracted over the keys, MN-major
// in the swizzle of 32-byte chunks. Q and G are A operands in tensor memory.
//
// Waits are bounded: when one runs out, bit 1 of the status word is raised and every thread leaves the tile loop
// at the next barrier, together.
#include <algorithm>
#include <atomic>

#include "common.cuh"
#include "kernels.cuh"
#include "tcgen05.cuh"

namespace msx {
namespace k {

namespace {

using tc::tmem_load;
using tc::tmem_loaded;
using tc::tmem_store;
using tc::tmem_stored;

constexpr int THREADS = 512;
constexpr uint64_t SMS = 148;
constexpr uint32_t QUERIES = 128, FORWARD_KEYS = 128, BACKWARD_TILE = 64;

// The halves the tensor core multiplies. It reads the upper 19 bits of a word, so what it drops of both halves has
// their sign, and with it the lo lo products that are left out: products come out low by some 2^-21 (8 to 10 10^-7 of
// the norm of O). Both are therefore rounded: 0.7 2^-11 of a value added to it is between a third and two thirds of
// its last kept bit (and, unlike an addition to the word, leaves a NaN one): 2 to 5 10^-7 of the norm of O and of the
// gradients, as batched products 6 to 27 10^-7. (The addition rounds towards zero: the largest finite values stay finite.)
constexpr float kHalfBit = 0.7f / 2048.0f;
__device__ __forceinline__ float high_of(float x) { return __uint_as_float(__float_as_uint(__fmaf_rz(x, kHalfBit, x)) & 0xffffe000u); }
__device__ __forceinline__ float low_of(float x, float h) {
    const float l = x - h;
    return fmaf(l, kHalfBit, l);
}
__device__ __forceinline__ float4 high_of(float4 v) { return make_float4(high_of(v.x), high_of(v.y), high_of(v.z), high_of(v.w)); }
__device__ __forceinline__ float4 low_of(float4 v, float4 h) { return make_float4(low_of(v.x, h.x), low_of(v.y, h.y), low_of(v.z, h.z), low_of(v.w, h.w)); }

// D (tensor memory) (+)= A (tensor memory, K-major: a lane a row, a column an element) B (shared memory).
__device__ __forceinline__ void mma_from_tmem(uint32_t d, uint32_t a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(d), "r"(a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}

__device__ __forceinline__ void before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// x as the hi and lo halves that the tensor core multiplies, into two places of tensor memory.
template <int COUNT> __device__ __forceinline__ void store_split(uint32_t hi_at, uint32_t lo_at, const float (&x)[COUNT]) {
#pragma unroll
    for (int first = 0; first < COUNT; first += 8) {
        uint32_t hi[8], lo[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float h = high_of(x[first + i]);
            hi[i] = __float_as_uint(h);
            lo[i] = __float_as_uint(low_of(x[first + i], h));
        }
        tmem_store(hi_at + first, hi);
        tmem_store(lo_at + first, lo);
    }
}

// Matrix descriptors (tcgen05.cuh, gemm_tf32.cu): a K-major operand of 128-byte rows in the swizzle of 16-byte
// chunks, and an MN-major one in the swizzle of 32-byte chunks whose panels of 32 elements are `panel` bytes apart.
__device__ __forceinline__ uint64_t k_major(uint32_t at) {
    constexpr uint32_t high = ((1024u >> 4) & 0x3FFFu) | (1u << 14) | (2u << 29);
    return (static_cast<uint64_t>(high) << 32) | (1u << 16) | ((at & 0x3FFFFu) >> 4);
}
__device__ __forceinline__ uint64_t mn_major(uint32_t at, uint32_t panel) {
    constexpr uint32_t high = ((512u >> 4) & 0x3FFFu) | (1u << 14) | (1u << 29);
    return (static_cast<uint64_t>(high) << 32) | (((panel >> 4) & 0x3FFFu) << 16) | ((at & 0x3FFFFu) >> 4);
}
// Instruction descriptor: f32 accumulator, tf32 operands, 128 rows, n columns.
__device__ __forceinline__ uint32_t instruction(uint32_t n, bool b_mn) {
    return (1u << 4) | (2u << 7) | (2u << 10) | ((b_mn ? 1u : 0u) << 16) | ((n >> 3) << 17) | ((128u >> 4) << 24);
}

// Four elements from column c on of a row of d, zeros past its end.
template <bool VEC> __device__ __forceinline__ float4 fetch4(const float* __restrict__ row, uint32_t c, uint32_t d) {
    if constexpr (VEC) return c < d ? load_global(reinterpret_cast<const float4*>(row + c)) : make_float4(0.f, 0.f, 0.f, 0.f);
    return make_float4(c < d ? load_global(row + c) : 0.f, c + 1 < d ? load_global(row + c + 1) : 0.f, c + 2 < d ? load_global(row + c + 2) : 0.f,
                       c + 3 < d ? load_global(row + c + 3) : 0.f);
}

// `rows` rows of a head, as fetched by the block: piece i of a thread is row i 512/(DP/4) + tid / (DP/4), four
// columns from tid % (DP/4) on.
template <int DP, uint32_t ROWS, bool VEC> struct Piece {
    static constexpr int COUNT = ROWS * (DP / 4) / THREADS;
    static constexpr uint32_t PANELS = DP / 32;
    float4 v[COUNT];
    __device__ __forceinline__ static uint32_t row(int i) { return (i * THREADS + threadIdx.x) / (DP / 4); }
    __device__ __forceinline__ static uint32_t column() { return threadIdx.x % (DP / 4) * 4; }
    __device__ __forceinline__ void fetch(const float* __restrict__ base, uint32_t ld, uint32_t rows, uint32_t d) {
#pragma unroll
        for (int i = 0; i < COUNT; ++i)
            v[i] = row(i) < rows ? fetch4<VEC>(base + static_cast<uint64_t>(row(i)) * ld, column(), d) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    // As a K-major operand of `kt` rows: per panel of 32 columns the hi rows, then the lo rows.
    __device__ __forceinline__ void store_k_major(char* tile, uint32_t kt) const {
        const uint32_t c = column();
#pragma unroll
        for (int i = 0; i < COUNT; ++i) {
            if (row(i) >= kt) continue;
            char* const at = tile + (c / 32) * 2 * kt * 128 + tc::swizzled_chunk(row(i), c % 32 / 4);
            const float4 h = high_of(v[i]);
            *reinterpret_cast<float4*>(at) = h;
            *reinterpret_cast<float4*>(at + kt * 128) = low_of(v[i], h);
        }
    }
    // As an MN-major one, contracted over its rows: the hi panels, then the lo panels, of `kt` 128-byte rows.
    __device__ __forceinline__ void store_mn_major(char* tile, uint32_t kt) const {
        const uint32_t c = column();
#pragma unroll
        for (int i = 0; i < COUNT; ++i) {
            if (row(i) >= kt) continue;
            char* const at = tile + (c / 32) * kt * 128 + row(i) * 128 + (((c % 32 / 8) ^ (row(i) & 3u)) << 5) + c % 8 * 4;
            const float4 h = high_of(v[i]);
            *reinterpret_cast<float4*>(at) = h;
            *reinterpret_cast<float4*>(at + PANELS * kt * 128) = low_of(v[i], h);
        }
    }
};

struct Shape {
    uint32_t l, s, h, heads, d;              // queries, keys, row pitch, heads, head width
    uint32_t tiles, key_tiles, key_blocks;  // tiles of 128 queries and keys of a head; blocks of the backward that take keys
    float scale;
    uint32_t p_vec;  // the probabilities' rows lie on 16 bytes
};
struct Place {
    uint32_t b, a, first;
};
__device__ __forceinline__ Place place_of(const Shape& sh, uint32_t block, uint32_t tiles) {
    const uint32_t head = block / tiles;
    return {head / sh.heads, head % sh.heads, (block - head * tiles) * QUERIES};
}

// What every CTA keeps beside its tiles.
struct Control {
    float part[4][QUERIES], part2[4][QUERIES];
    uint64_t bars[3];
    uint32_t tmem_slot, abort_flag;
};
__device__ __forceinline__ uint32_t begin(Control* c) {
    if (threadIdx.x == 0) {
        tc::mbar_init(tc::smem_u32(&c->bars[0]), 1);
        tc::mbar_init(tc::smem_u32(&c->bars[1]), 1);
        tc::mbar_init(tc::smem_u32(&c->bars[2]), 1);
        c->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (threadIdx.x < 32) tc::tmem_alloc<1>(tc::smem_u32(&c->tmem_slot), 512);
    before_sync();
    __syncthreads();
    after_sync();
    wait_for_producers();
    return c->tmem_slot;
}
__device__ __forceinline__ void finish(uint32_t tmem) {
    before_sync();
    __syncthreads();
    if (threadIdx.x < 32) tc::tmem_dealloc<1>(tmem, 512);
}

// This thread's DP / 4 columns of its query row, zeros outside.
template <int DP, bool VEC> __device__ __forceinline__ void fetch_row(const float* __restrict__ base, uint32_t ld, uint32_t row, uint32_t rows, uint32_t first,
                                                                      uint32_t d, float (&x)[DP / 4]) {
#pragma unroll
    for (int i = 0; i < DP / 4; i += 4) {
        const float4 f = row < rows ? fetch4<VEC>(base + static_cast<uint64_t>(row) * ld, first + i, d) : make_float4(0.f, 0.f, 0.f, 0.f);
        x[i] = f.x; x[i + 1] = f.y; x[i + 2] = f.z; x[i + 3] = f.w;
    }
}
template <int DP, bool VEC> __device__ __forceinline__ void put_row(float* __restrict__ base, uint32_t ld, uint32_t row, uint32_t rows, uint32_t first, uint32_t d,
                                                                    const float (&x)[DP / 4]) {
    if (row >= rows) return;
    float* const to = base + static_cast<uint64_t>(row) * ld + first;
#pragma unroll
    for (int i = 0; i < DP / 4; i += 4) {
        if constexpr (VEC) {
            if (first + i < d) *reinterpret_cast<float4*>(to + i) = make_float4(x[i], x[i + 1], x[i + 2], x[i + 3]);
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (first + i + j < d) to[i + j] = x[i + j];
        }
    }
}

// What one thread issues. Unrolled, with every descriptor a constant away from the first: a loop that makes them
// takes longer for an MMA than the tensor core does.
// D = (rows hi at `a`, lo 64 columns on) x tile^T: K-major tiles of `kt` rows, `steps` k slices of 8.
__device__ __forceinline__ void issue_scores(uint32_t d, uint32_t a, uint32_t tile, uint32_t kt, uint32_t steps) {
    const uint64_t first = k_major(tile), panel = (2 * kt * 128) >> 4;
    const uint32_t wide = instruction(2 * kt, false), narrow = instruction(kt, false);
#pragma unroll
    for (uint32_t ks = 0; ks < 8; ++ks) {
        if (ks >= steps) break;
        const uint64_t b = first + (ks >> 2) * panel + (ks & 3u) * 2;
        mma_from_tmem(d, a + ks * 8, b, wide, ks != 0);  // the tile's hi and lo rows
        mma_from_tmem(d + kt, a + 64 + ks * 8, b, narrow, 1);
    }
}
// D = (hi at `a`, lo `lo` columns on) x the MN-major tile of `kt` rows, contracted over `count` (up to 8 STEPS) of them.
template <int DP, uint32_t STEPS> __device__ __forceinline__ void issue_product(uint32_t d, uint32_t a, uint32_t lo, uint32_t tile, uint32_t kt, uint32_t count) {
    const uint64_t first = mn_major(tile, kt * 128);
    const uint32_t steps = (count + 7) / 8;
#pragma unroll
    for (uint32_t ks = 0; ks < STEPS; ++ks) {
        if (ks >= steps) break;
        mma_from_tmem(d, a + ks * 8, first + ks * 64, instruction(2 * DP, true), ks != 0);
        mma_from_tmem(d + DP, a + lo + ks * 8, first + ks * 64, instruction(DP, true), 1);
    }
}

// ---- forward -------------------------------------------------------------------------------------------
// Tensor memory: scores (hi products, cross products; then P hi, P lo) in columns 0..255, P V in 256..383,
// Q hi and lo in 384..511.
template <int DP> constexpr int forward_bytes() { return 2 * (DP / 32) * 2 * FORWARD_KEYS * 128 + static_cast<int>(sizeof(Control)); }

template <int DP, bool VEC>
__global__ void __launch_bounds__(THREADS, 1) attention_f32_forward_kernel(const float* q, const float* k, const float* v,
                                                                           const float* mask, float* out, float2* stats,
                                                                           float* p_out, const Shape sh, uint32_t* status) {
    constexpr uint32_t PANELS = DP / 32, SCORES = 0, P_HI = 0, P_LO = 128, PV = 256, Q_HI = 384, Q_LO = 448, OWN = DP / 4;
    extern __shared__ __align__(1024) char smem[];
    char* const k_tile = smem;
    char* const v_tile = smem + PANELS * 2 * FORWARD_KEYS * 128;
    Control* const ctl = reinterpret_cast<Control*>(v_tile + PANELS * 2 * FORWARD_KEYS * 128);
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, quarter = warp & 3u, part = warp >> 2;
    const uint32_t row = quarter * 32 + lane;  // of the tile; four threads share it, `part` of its columns each
    const Place at = place_of(sh, blockIdx.x, sh.tiles);
    const uint32_t kt = min(FORWARD_KEYS, (sh.s + 15) / 16 * 16);
    const float* const kb = k + static_cast<uint64_t>(at.b) * sh.s * sh.h + at.a * sh.d;
    const float* const vb = v + static_cast<uint64_t>(at.b) * sh.s * sh.h + at.a * sh.d;
    const uint64_t q_at = static_cast<uint64_t>(at.b) * sh.l * sh.h + at.a * sh.d;
    const float* const mb = mask + static_cast<uint64_t>(at.b) * sh.s;

    Piece<DP, FORWARD_KEYS, VEC> kp, vp;
    float mine = 0.0f;  // the mask of key part * 32 + lane
    auto fetch = [&](uint32_t j0) {
        const uint32_t rows = min(kt, sh.s - j0);
        kp.fetch(kb + static_cast<uint64_t>(j0) * sh.h, sh.h, rows, sh.d);
        vp.fetch(vb + static_cast<uint64_t>(j0) * sh.h, sh.h, rows, sh.d);
        mine = part * 32 + lane < rows ? load_global(mb + j0 + part * 32 + lane) : 0.0f;
    };
    const uint32_t tmem = begin(ctl), lanes = tmem + ((quarter * 32u) << 16);
    fetch(0);
    float x[OWN];
    fetch_row<DP, VEC>(q + q_at, sh.h, at.first + row, sh.l, part * OWN, sh.d, x);
    store_split(lanes + Q_HI + part * OWN, lanes + Q_LO + part * OWN, x);
    tmem_stored();
    before_sync();

    float o[OWN] = {}, best = -INFINITY, total = 0.0f;
    uint32_t parity = 0;
    for (uint32_t j0 = 0;; parity ^= 1u) {
        kp.store_k_major(k_tile, kt);
        vp.store_mn_major(v_tile, kt);
        const uint32_t counts = __ballot_sync(0xffffffffu, mine != 0.0f), here = min(kt, sh.s - j0);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (tid == 0) {
            after_sync();
            issue_scores(tmem + SCORES, tmem + Q_HI, tc::smem_u32(k_tile), kt, (sh.d + 7) / 8);
            tc::mma_commit(tc::smem_u32(&ctl->bars[0]));
        }
        __syncwarp();
        const uint32_t next = j0 + kt;
        if (next < sh.s) fetch(next);
        bool alive = tc::warp_wait<1>(tc::smem_u32(&ctl->bars[0]), parity, &ctl->abort_flag, status);
        after_sync();
        float p[32];
        float top = -INFINITY;
        const bool busy = part * 32 < kt;  // (the same for a warp)
        if (busy) {
            // (sixteen columns at a time, here and below: a thread's 128 registers hold a tile of K and V on its way too)
#pragma unroll
            for (int first = 0; first < 32; first += 16) {
                uint32_t hi[16], cross[16];
                tmem_load(lanes + SCORES + part * 32 + first, hi);
                tmem_load(lanes + SCORES + kt + part * 32 + first, cross);
                tmem_loaded();
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    p[first + i] = (__uint_as_float(hi[i]) + __uint_as_float(cross[i])) * sh.scale;
                    if ((counts >> (first + i)) & 1u) top = fmaxf(top, p[first + i]);
                }
            }
        }
        ctl->part[part][row] = top;
        before_sync();
        alive = __syncthreads_and(alive);
        after_sync();
        top = fmaxf(fmaxf(ctl->part[0][row], ctl->part[1][row]), fmaxf(ctl->part[2][row], ctl->part[3][row]));
        top = fmaxf(best, top);
        // (tiles of masked keys only leave the maximum at -inf)
        const float base = top == -INFINITY ? 0.0f : top, again = best == -INFINITY ? 0.0f : expf(best - base);
        best = top;
        total *= again;
        if (busy) {
#pragma unroll
            for (int first = 0; first < 32; first += 16) {
                float e[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    p[first + i] = e[i] = (counts >> (first + i)) & 1u ? expf(p[first + i] - base) : 0.0f;
                    total += e[i];
                }
                store_split(lanes + P_HI + part * 32 + first, lanes + P_LO + part * 32 + first, e);
            }
            tmem_stored();
        }
        if (p_out) ctl->part2[part][row] = total;
        before_sync();
        __syncthreads();
        if (tid == 0) {
            after_sync();
            issue_product<DP, FORWARD_KEYS / 8>(tmem + PV, tmem + P_HI, P_LO - P_HI, tc::smem_u32(v_tile), kt, here);
            tc::mma_commit(tc::smem_u32(&ctl->bars[1]));
        }
        __syncwarp();
        // The probabilities themselves, for gradients formed as batched products (one tile holds all keys).
        if (p_out && busy && at.first + row < sh.l) {
            const float inverse = 1.0f / ((ctl->part2[0][row] + ctl->part2[1][row]) + (ctl->part2[2][row] + ctl->part2[3][row]));
            float* const to = p_out + ((static_cast<uint64_t>(at.b) * sh.heads + at.a) * sh.l + at.first + row) * sh.s + part * 32;
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
                const uint32_t c = part * 32 + i;
                const float4 f = make_float4(p[i] * inverse, p[i + 1] * inverse, p[i + 2] * inverse, p[i + 3] * inverse);
                if (sh.p_vec) {
                    if (c < sh.s) *reinterpret_cast<float4*>(to + i) = f;
                } else {
                    if (c < sh.s) to[i] = f.x;
                    if (c + 1 < sh.s) to[i + 1] = f.y;
                    if (c + 2 < sh.s) to[i + 2] = f.z;
                    if (c + 3 < sh.s) to[i + 3] = f.w;
                }
            }
        }
        alive = tc::warp_wait<1>(tc::smem_u32(&ctl->bars[1]), parity, &ctl->abort_flag, status) && alive;
        after_sync();
        uint32_t hi[OWN], cross[OWN];
        tmem_load(lanes + PV + part * OWN, hi);
        tmem_load(lanes + PV + DP + part * OWN, cross);
        tmem_loaded();
        before_sync();
#pragma unroll
        for (int i = 0; i < static_cast<int>(OWN); ++i) o[i] = fmaf(o[i], again, __uint_as_float(hi[i]) + __uint_as_float(cross[i]));
        j0 = next;
        if (!__syncthreads_and(alive && j0 < sh.s)) break;
    }
    let_next_start();
    ctl->part2[part][row] = total;
    __syncthreads();
    total = (ctl->part2[0][row] + ctl->part2[1][row]) + (ctl->part2[2][row] + ctl->part2[3][row]);
#pragma unroll
    for (int i = 0; i < static_cast<int>(OWN); ++i) o[i] = o[i] / total;
    put_row<DP, VEC>(out + q_at, sh.h, at.first + row, sh.l, part * OWN, sh.d, o);
    if (stats && part == 0 && at.first + row < sh.l) stats[(static_cast<uint64_t>(at.b) * sh.heads + at.a) * sh.l + at.first + row] = make_float2(best, total);
    finish(tmem);
}

// ---- backward ------------------------------------------------------------------------------------------
// Blocks of 128 queries, which form dQ, and blocks of 128 keys, which form dK and dV, in one launch; each recomputes the
// scores it needs (seven products of the scores' size instead of five, but none of them crosses memory and nothing
// waits for another launch). Tensor memory: this block's rows of two operands as A halves in columns 0..255, the
// tile's scores in 256..383 (later a tile's dQ, or P and then dS), dP in 384..511 (later dS, or a tile's dV and then dK).
constexpr uint32_t ROWS_A_HI = 0, ROWS_A_LO = 64, ROWS_B_HI = 128, ROWS_B_LO = 192, SCORES_AT = 256, DP_AT = 384;
template <int DP> constexpr uint32_t TILE_BYTES = DP / 32 * 2 * BACKWARD_TILE * 128;
template <int DP> constexpr int backward_bytes() {
    return static_cast<int>(4 * TILE_BYTES<DP> + 3 * BACKWARD_TILE * 4 + sizeof(Control));
}

struct BackwardArgs {
    const float *q, *k, *v, *mask, *g, *out;
    const float2* stats;
    float *dq, *dk, *dv;
    uint32_t* status;
};

// Sixteen columns of a product and of its cross products.
__device__ __forceinline__ void load_sum16(uint32_t at, uint32_t cross_at, float (&x)[16]) {
    uint32_t hi[16], cross[16];
    tmem_load(at, hi);
    tmem_load(cross_at, cross);
    tmem_loaded();
#pragma unroll
    for (int i = 0; i < 16; ++i) x[i] = __uint_as_float(hi[i]) + __uint_as_float(cross[i]);
}
template <int OWN> __device__ __forceinline__ void add_product(uint32_t at, uint32_t cross_at, float (&sum)[OWN]) {
    uint32_t hi[OWN], cross[OWN];
    tmem_load(at, hi);
    tmem_load(cross_at, cross);
    tmem_loaded();
    before_sync();
#pragma unroll
    for (int i = 0; i < OWN; ++i) sum[i] += __uint_as_float(hi[i]) + __uint_as_float(cross[i]);
}

template <int DP, bool VEC> __device__ __forceinline__ void backward_queries(char* smem, Control* ctl, const BackwardArgs& x, const Shape& sh) {
    constexpr uint32_t OWN = DP / 4, TILE = TILE_BYTES<DP>;
    char *const k_tile = smem, *const v_tile = smem + TILE, *const kn_tile = smem + 2 * TILE;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, quarter = warp & 3u, part = warp >> 2;
    const uint32_t row = quarter * 32 + lane;
    const Place at = place_of(sh, blockIdx.x - sh.key_blocks, sh.tiles);
    const uint32_t kt = min(BACKWARD_TILE, (sh.s + 15) / 16 * 16);
    const uint64_t k_at = static_cast<uint64_t>(at.b) * sh.s * sh.h + at.a * sh.d, q_at = static_cast<uint64_t>(at.b) * sh.l * sh.h + at.a * sh.d;
    const float* const mb = x.mask + static_cast<uint64_t>(at.b) * sh.s;

    Piece<DP, BACKWARD_TILE, VEC> kp, vp;
    float mine = 0.0f;  // the mask of key part * 16 + lane
    auto fetch = [&](uint32_t j0) {
        const uint32_t keys = min(kt, sh.s - j0);
        kp.fetch(x.k + k_at + static_cast<uint64_t>(j0) * sh.h, sh.h, keys, sh.d);
        vp.fetch(x.v + k_at + static_cast<uint64_t>(j0) * sh.h, sh.h, keys, sh.d);
        mine = lane < 16 && part * 16 + lane < keys ? load_global(mb + j0 + part * 16 + lane) : 0.0f;
    };
    const uint32_t tmem = begin(ctl), lanes = tmem + ((quarter * 32u) << 16);
    fetch(0);
    const float2 stat = at.first + row < sh.l ? load_global(x.stats + (static_cast<uint64_t>(at.b) * sh.heads + at.a) * sh.l + at.first + row) : make_float2(0.f, 1.f);
    float own[OWN], other[OWN];
    fetch_row<DP, VEC>(x.q + q_at, sh.h, at.first + row, sh.l, part * OWN, sh.d, own);
    fetch_row<DP, VEC>(x.g + q_at, sh.h, at.first + row, sh.l, part * OWN, sh.d, other);
    store_split(lanes + ROWS_A_HI + part * OWN, lanes + ROWS_A_LO + part * OWN, own);
    store_split(lanes + ROWS_B_HI + part * OWN, lanes + ROWS_B_LO + part * OWN, other);
    tmem_stored();
    before_sync();
    // The row's O . G = sum_j P dP.
    fetch_row<DP, VEC>(x.out + q_at, sh.h, at.first + row, sh.l, part * OWN, sh.d, own);
    float dot = 0.0f;
#pragma unroll
    for (int i = 0; i < static_cast<int>(OWN); ++i) dot = fmaf(own[i], other[i], dot);
    ctl->part[part][row] = dot;
    __syncthreads();
    dot = (ctl->part[0][row] + ctl->part[1][row]) + (ctl->part[2][row] + ctl->part[3][row]);
    const float inverse = 1.0f / stat.y;

    float sum[OWN] = {};
    uint32_t parity = 0;
    for (uint32_t j0 = 0;; parity ^= 1u) {
        kp.store_k_major(k_tile, kt);
        kp.store_mn_major(kn_tile, kt);
        vp.store_k_major(v_tile, kt);
        const uint32_t counts = __ballot_sync(0xffffffffu, mine != 0.0f), here = min(kt, sh.s - j0);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (tid == 0) {
            after_sync();
            issue_scores(tmem + SCORES_AT, tmem + ROWS_A_HI, tc::smem_u32(k_tile), kt, (sh.d + 7) / 8);
            issue_scores(tmem + DP_AT, tmem + ROWS_B_HI, tc::smem_u32(v_tile), kt, (sh.d + 7) / 8);
            tc::mma_commit(tc::smem_u32(&ctl->bars[0]));
        }
        __syncwarp();
        const uint32_t next = j0 + kt;
        if (next < sh.s) fetch(next);
        bool alive = tc::warp_wait<1>(tc::smem_u32(&ctl->bars[0]), parity, &ctl->abort_flag, x.status);
        after_sync();
        const bool busy = part * 16 < kt;  // (the same for a warp)
        float ds[16];
        if (busy) {
            float p[16];
            load_sum16(lanes + SCORES_AT + part * 16, lanes + SCORES_AT + kt + part * 16, p);
            load_sum16(lanes + DP_AT + part * 16, lanes + DP_AT + kt + part * 16, ds);
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                p[i] = (counts >> i) & 1u ? expf(p[i] * sh.scale - stat.x) * inverse : 0.0f;
                ds[i] = p[i] * (ds[i] - dot) * sh.scale;
            }
        }
        before_sync();
        alive = __syncthreads_and(alive);  // every warp has its scores and dP: their columns are free
        after_sync();
        if (busy) {
            store_split(lanes + DP_AT + part * 16, lanes + DP_AT + 64 + part * 16, ds);
            tmem_stored();
        }
        before_sync();
        __syncthreads();
        if (tid == 0) {
            after_sync();
            issue_product<DP, BACKWARD_TILE / 8>(tmem + SCORES_AT, tmem + DP_AT, 64, tc::smem_u32(kn_tile), kt, here);
            tc::mma_commit(tc::smem_u32(&ctl->bars[1]));
        }
        __syncwarp();
        alive = tc::warp_wait<1>(tc::smem_u32(&ctl->bars[1]), parity, &ctl->abort_flag, x.status) && alive;
        after_sync();
        add_product(lanes + SCORES_AT + part * OWN, lanes + SCORES_AT + DP + part * OWN, sum);
        j0 = next;
        if (!__syncthreads_and(alive && j0 < sh.s)) break;
    }
    let_next_start();
    put_row<DP, VEC>(x.dq + q_at, sh.h, at.first + row, sh.l, part * OWN, sh.d, sum);
    finish(tmem);
}

template <int DP, bool VEC> __device__ __forceinline__ void backward_keys(char* smem, Control* ctl, const BackwardArgs& x, const Shape& sh) {
    constexpr uint32_t OWN = DP / 4, TILE = TILE_BYTES<DP>;
    char *const q_tile = smem, *const g_tile = smem + TILE, *const qn_tile = smem + 2 * TILE, *const gn_tile = smem + 3 * TILE;
    // Of the tile's queries: maximum, 1 / sum, O . G.
    float *const top = reinterpret_cast<float*>(ctl + 1), *const inverse = top + BACKWARD_TILE, *const dots = inverse + BACKWARD_TILE;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, quarter = warp & 3u, part = warp >> 2;
    const uint32_t row = quarter * 32 + lane;  // a key
    const Place at = place_of(sh, blockIdx.x, sh.key_tiles);
    const uint32_t kt = min(BACKWARD_TILE, (sh.l + 15) / 16 * 16);
    const uint64_t k_at = static_cast<uint64_t>(at.b) * sh.s * sh.h + at.a * sh.d, q_at = static_cast<uint64_t>(at.b) * sh.l * sh.h + at.a * sh.d;
    const float2* const stats = x.stats + (static_cast<uint64_t>(at.b) * sh.heads + at.a) * sh.l;

    Piece<DP, BACKWARD_TILE, VEC> qp, gp, op;
    float2 stat;
    auto fetch = [&](uint32_t i0) {
        const uint32_t queries = min(kt, sh.l - i0);
        const uint64_t from = q_at + static_cast<uint64_t>(i0) * sh.h;
        qp.fetch(x.q + from, sh.h, queries, sh.d);
        gp.fetch(x.g + from, sh.h, queries, sh.d);
        op.fetch(x.out + from, sh.h, queries, sh.d);
        stat = tid < queries ? load_global(stats + i0 + tid) : make_float2(0.f, 1.f);
    };
    const uint32_t tmem = begin(ctl), lanes = tmem + ((quarter * 32u) << 16);
    fetch(0);
    const bool counted = at.first + row < sh.s && load_global(x.mask + static_cast<uint64_t>(at.b) * sh.s + at.first + row) != 0.0f;
    float own[OWN];
    fetch_row<DP, VEC>(x.k + k_at, sh.h, at.first + row, sh.s, part * OWN, sh.d, own);
    store_split(lanes + ROWS_A_HI + part * OWN, lanes + ROWS_A_LO + part * OWN, own);
    fetch_row<DP, VEC>(x.v + k_at, sh.h, at.first + row, sh.s, part * OWN, sh.d, own);
    store_split(lanes + ROWS_B_HI + part * OWN, lanes + ROWS_B_LO + part * OWN, own);
    tmem_stored();
    before_sync();

    float dk[OWN] = {}, dv[OWN] = {};
    uint32_t parity = 0;
    for (uint32_t i0 = 0;; parity ^= 1u) {
        qp.store_k_major(q_tile, kt);
        qp.store_mn_major(qn_tile, kt);
        gp.store_k_major(g_tile, kt);
        gp.store_mn_major(gn_tile, kt);
        if (tid < kt) {
            top[tid] = stat.x;
            inverse[tid] = 1.0f / stat.y;
        }
#pragma unroll
        for (int i = 0; i < gp.COUNT; ++i) {
            const float4 o = op.v[i], g = gp.v[i];
            float dot = fmaf(o.x, g.x, fmaf(o.y, g.y, fmaf(o.z, g.z, o.w * g.w)));
#pragma unroll
            for (int away = DP / 8; away > 0; away >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, away);
            if (gp.column() == 0) dots[gp.row(i)] = dot;
        }
        const uint32_t here = min(kt, sh.l - i0);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (tid == 0) {
            after_sync();
            issue_scores(tmem + SCORES_AT, tmem + ROWS_A_HI, tc::smem_u32(q_tile), kt, (sh.d + 7) / 8);
            issue_scores(tmem + DP_AT, tmem + ROWS_B_HI, tc::smem_u32(g_tile), kt, (sh.d + 7) / 8);
            tc::mma_commit(tc::smem_u32(&ctl->bars[0]));
        }
        __syncwarp();
        const uint32_t next = i0 + kt;
        if (next < sh.l) fetch(next);
        bool alive = tc::warp_wait<1>(tc::smem_u32(&ctl->bars[0]), parity, &ctl->abort_flag, x.status);
        after_sync();
        const bool busy = part * 16 < kt;
        float p[16], ds[16];
        if (busy) {
            load_sum16(lanes + SCORES_AT + part * 16, lanes + SCORES_AT + kt + part * 16, p);
            load_sum16(lanes + DP_AT + part * 16, lanes + DP_AT + kt + part * 16, ds);
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const uint32_t c = part * 16 + i;  // queries past the tile's last: zeros
                p[i] = counted && c < here ? expf(p[i] * sh.scale - top[c]) * inverse[c] : 0.0f;
                ds[i] = counted && c < here ? p[i] * (ds[i] - dots[c]) * sh.scale : 0.0f;
            }
        }
        before_sync();
        alive = __syncthreads_and(alive);
        after_sync();
        if (x.dv) {
            if (busy) {
                store_split(lanes + SCORES_AT + part * 16, lanes + SCORES_AT + 64 + part * 16, p);
                tmem_stored();
            }
            before_sync();
            __syncthreads();
            if (tid == 0) {
                after_sync();
                issue_product<DP, BACKWARD_TILE / 8>(tmem + DP_AT, tmem + SCORES_AT, 64, tc::smem_u32(gn_tile), kt, here);
                tc::mma_commit(tc::smem_u32(&ctl->bars[1]));
            }
            __syncwarp();
            alive = tc::warp_wait<1>(tc::smem_u32(&ctl->bars[1]), parity, &ctl->abort_flag, x.status) && alive;
            after_sync();
            add_product(lanes + DP_AT + part * OWN, lanes + DP_AT + DP + part * OWN, dv);
        }
        if (x.dk) {
            if (busy) {
                store_split(lanes + SCORES_AT + part * 16, lanes + SCORES_AT + 64 + part * 16, ds);
                tmem_stored();
            }
            before_sync();
            __syncthreads();
            if (tid == 0) {
                after_sync();
                issue_product<DP, BACKWARD_TILE / 8>(tmem + DP_AT, tmem + SCORES_AT, 64, tc::smem_u32(qn_tile), kt, here);
                tc::mma_commit(tc::smem_u32(&ctl->bars[2]));
            }
            __syncwarp();
            alive = tc::warp_wait<1>(tc::smem_u32(&ctl->bars[2]), parity, &ctl->abort_flag, x.status) && alive;
            after_sync();
            add_product(lanes + DP_AT + part * OWN, lanes + DP_AT + DP + part * OWN, dk);
        }
        i0 = next;
        if (!__syncthreads_and(alive && i0 < sh.l)) break;
    }
    let_next_start();
    if (x.dk) put_row<DP, VEC>(x.dk + k_at, sh.h, at.first + row, sh.s, part * OWN, sh.d, dk);
    if (x.dv) put_row<DP, VEC>(x.dv + k_at, sh.h, at.first + row, sh.s, part * OWN, sh.d, dv);
    finish(tmem);
}

template <int DP, bool VEC>
__global__ void __launch_bounds__(THREADS, 1) attention_f32_backward_kernel(const __grid_constant__ BackwardArgs args, const __grid_constant__ Shape sh) {
    extern __shared__ __align__(1024) char smem[];
    Control* const ctl = reinterpret_cast<Control*>(smem + 4 * TILE_BYTES<DP>);
    // (the blocks that take longer go first)
    if (blockIdx.x < sh.key_blocks) backward_keys<DP, VEC>(smem, ctl, args, sh);
    else backward_queries<DP, VEC>(smem, ctl, args, sh);
}

Shape shape_of(AttentionShape sh) {
    Shape s;
    s.l = sh.q_len; s.s = sh.k_len; s.heads = sh.heads; s.d = sh.head_dim; s.h = sh.heads * sh.head_dim;
    s.tiles = (sh.q_len + QUERIES - 1) / QUERIES;
    s.key_tiles = (sh.k_len + QUERIES - 1) / QUERIES;
    s.key_blocks = 0;
    s.scale = 1.0f / sqrtf(static_cast<float>(sh.head_dim));
    s.p_vec = 0;
    return s;
}
bool on_16_bytes(std::initializer_list<const void*> pointers) {
    for (const void* p : pointers)
        if (reinterpret_cast<uintptr_t>(p) % 16 != 0) return false;
    return true;
}

}  // namespace

bool attention_f32_supported(AttentionShape sh) {
    return sh.head_dim >= 1 && sh.head_dim <= 64 && sh.k_len >= 1 && sh.k_len <= 512 && sh.q_len >= 1 &&
           static_cast<uint64_t>(sh.batch) * sh.heads * ((sh.q_len + QUERIES - 1) / QUERIES + 4) < (1ull << 31);
}

// Which way is the sooner one inside a step's graph, in us. The kernels here: their blocks in waves, each with a start
// and, per tile, some 7 to 8 us for 64 columns (the most of it the tile's products), and 1.5 for code that is cold where
// the products' is not. The batched products: three launches forward and four backward of a tile or two each, and
// what the work adds, its tiles padded; more where rows off 16 bytes keep them from TMA. Measured (a launch alone less
// the 2 us that it costs outside of a graph; these kernels, the products), forward: 64 heads of 128 x 64 10.7, 14.6; 16
// heads 10.7, 11.1 (in a step 2 us slower than the products); 128 heads 12.3, 17.7; 96 of 40 x 24 6.4, 10.5; 768 of 16 x 64 35,
// 26; 384 of 512 x 64 320, 390; off 16 bytes, 15 heads of 77 x 33 9.3, 11.6. Backward: 64 heads of 128 x 64 18.6, 20.7; 16 heads
// 18.6, 17.7; 128 heads 32.9, 26.9; 96 of 40 x 24 10.4, 16.7; 240 of 64 x 32 26.8, 22.8; 8 of 256 x 64 31, 23; 15 of 77 x 33 17.7, 25.4.
AttentionWay attention_f32_way(AttentionShape sh, bool gradients) {
    if (!attention_f32_supported(sh)) return AttentionWay::Products;
    auto up = [](uint64_t x, uint64_t to) { return (x + to - 1) / to; };
    const uint64_t heads = static_cast<uint64_t>(sh.batch) * sh.heads, longest = std::max(sh.q_len, sh.k_len);
    const bool aligned = sh.head_dim % 4 == 0 && sh.k_len % 4 == 0, narrow = sh.head_dim <= 32;
    const uint64_t pad = longest <= 64 ? 64 : 128;
    const double work = 1e-6 * static_cast<double>(heads * up(sh.q_len, pad) * up(sh.k_len, pad) * pad * pad * up(sh.head_dim, 32) * 32);
    const double keys = static_cast<double>(up(sh.k_len, FORWARD_KEYS)) * std::min(1.0, up(sh.k_len, 16) * 16 / 128.0);
    const double forward = 1.5 + static_cast<double>(up(heads * up(sh.q_len, QUERIES), SMS)) * (3.5 + keys * (narrow ? 4.0 : 7.5));
    const double forward_products = aligned ? 10.5 + (longest <= 64 ? 0.10 : 0.06) * work : 13.0 + 0.09 * work;
    if (!gradients) return forward < forward_products ? AttentionWay::Forward : AttentionWay::Products;
    const double tile = 2.0 + (narrow ? 4.0 : 5.0) * std::min(1.0, up(longest, 16) * 16 / 64.0);
    const double backward = 1.5 + static_cast<double>(up(heads * (up(sh.q_len, QUERIES) + up(sh.k_len, QUERIES)), SMS)) *
                                      (3.5 + static_cast<double>(up(longest, BACKWARD_TILE)) * tile);
    const double backward_products = aligned ? 17.0 + (longest <= 64 ? 0.17 : 0.07) * work : 23.0 + 0.16 * work;
    // (the probabilities that the gradients' products read are left by the forward kernel where one tile holds a row)
    const bool leaves = sh.k_len <= FORWARD_KEYS && forward < forward_products;
    if (forward + backward < (leaves ? forward : forward_products) + backward_products) return AttentionWay::Both;
    return leaves ? AttentionWay::Forward : AttentionWay::Products;
}

uint64_t attention_f32_stats_floats(AttentionShape sh) { return 2ull * sh.batch * sh.heads * sh.q_len; }

void attention_f32_forward(cudaStream_t s, const float* q, const float* k, const float* v, const float* mask, float* out, float* stats, float* p,
                           AttentionShape sh, uint32_t* status) {
    if (sh.batch == 0) return;
    Shape shape = shape_of(sh);
    shape.p_vec = sh.k_len % 4 == 0 && on_16_bytes({p});
    const bool vec = sh.head_dim % 4 == 0 && on_16_bytes({q, k, v, out});
    auto go = [&](auto kernel, int bytes, std::atomic<int>& configured_device) {
        set_shared_memory(kernel, bytes, configured_device);
        kernel<<<sh.batch * sh.heads * shape.tiles, THREADS, bytes, s>>>(q, k, v, mask, out, reinterpret_cast<float2*>(stats), p, shape, status);
    };
    static std::atomic<int> configured[4] = {{-1}, {-1}, {-1}, {-1}};
    if (sh.head_dim <= 32) vec ? go(attention_f32_forward_kernel<32, true>, forward_bytes<32>(), configured[0])
                               : go(attention_f32_forward_kernel<32, false>, forward_bytes<32>(), configured[1]);
    else vec ? go(attention_f32_forward_kernel<64, true>, forward_bytes<64>(), configured[2])
             : go(attention_f32_forward_kernel<64, false>, forward_bytes<64>(), configured[3]);
    check_launch("attention_f32_forward");
}

void attention_f32_backward(cudaStream_t s, const float* q, const float* k, const float* v, const float* mask, const float* g, const float* out,
                            const float* stats, float* dq, float* dk, float* dv, AttentionShape sh, uint32_t* status) {
    if (sh.batch == 0 || (!dq && !dk && !dv)) return;
    Shape shape = shape_of(sh);
    const uint32_t heads = sh.batch * sh.heads;
    shape.key_blocks = dk || dv ? heads * shape.key_tiles : 0;
    const uint32_t blocks = shape.key_blocks + (dq ? heads * shape.tiles : 0);
    const bool vec = sh.head_dim % 4 == 0 && on_16_bytes({q, k, v, g, out, dq, dk, dv});
    const BackwardArgs args = {q, k, v, mask, g, out, reinterpret_cast<const float2*>(stats), dq, dk, dv, status};
    auto go = [&](auto kernel, int bytes, std::atomic<int>& configured_device) {
        set_shared_memory(kernel, bytes, configured_device);
        kernel<<<blocks, THREADS, bytes, s>>>(args, shape);
    };
    static std::atomic<int> configured[4] = {{-1}, {-1}, {-1}, {-1}};
    if (sh.head_dim <= 32) vec ? go(attention_f32_backward_kernel<32, true>, backward_bytes<32>(), configured[0])
                               : go(attention_f32_backward_kernel<32, false>, backward_bytes<32>(), configured[1]);
    else vec ? go(attention_f32_backward_kernel<64, true>, backward_bytes<64>(), configured[2])
             : go(attention_f32_backward_kernel<64, false>, backward_bytes<64>(), configured[3]);
    check_launch("attention_f32_backward");
}

}  // namespace k
}  // namespace msx
