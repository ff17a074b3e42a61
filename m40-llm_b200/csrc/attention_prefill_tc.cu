// Prompt attention on the 5th-generation tensor cores: CTA = one or two tiles of 128 query rows of one sequence and kv head, keys in
// tiles of 128.
//
//   scores   S[128 q rows][128 keys] = Qhi K^T + Qlo K^T   A = queries (f16 hi and lo, shared memory), B = the key tile, K-major;
//   softmax  thread = query row = accumulator lane, so a row needs no exchange;
//   values   O[128][HD + 16] += P [V | 1]                   A = the weights in tensor memory (f16, over the scores they came from),
//                                                           B = the value tile, MN-major, and behind it a chunk of ones, whose
//                                                           columns add up the weights that the values were multiplied with.
//
// A row's reference is its running maximum, so its strongest key weighs exactly 1, and numerator and denominator share the
// rounding of all others: relative error 0.96 to 1.01 of what the mma.sync form gives, for queries scaled by 1 to 8. (A reference
// that moves only with every 2^8 of growth saves most of the rescaling, 9 of 273 us and 18 of 221 us at head size 64,
// but its strongest weight is rounded: 1.05 times that error for flat scores, 3.3 times for peaked ones. Adding up the rounded
// weights in the rows' registers took 12 us more.)
//
// With one tile warps 0..3 are the query rows, warp 4 loads K and V by TMA (a ring of four tiles, three with two row tiles of 128
// dimensions), warp 5 issues the MMAs: S(j + 1) runs while the rows work on S(j). With two, warps 0..7 are the rows, which add up their rounded
// weights themselves: there is no chunk of ones. A 128 x 128 tile of HD 128 is 24 MMAs (1600 cycles at the tensor rate) beside 1024
// cycles of exponentials per scheduler; one set of rows per SM leaves part of either idle, so that two row tiles share a CTA (TILES) where there are enough CTAs to
// balance (prompt_cost.cuh). Four packed prompts of 509 to 2048 tokens, 32 / 8 heads of 128: 245 us, with one tile 280, against 438 us with
// mma.sync fragments (attention_prefill.cu), which stay for short segments; 220 since the call no longer copies its lengths back.
// Rows behind a sequence's last key are whatever the cache holds there; the issuing warp clears them in the value tile, since
// zero weights do not cancel a NaN. Values of tokens that only some rows see are dealt with at the end (attend_row()): looking
// through the one or two tiles in question beforehand, in shared memory or with a warp of its own, cost 8 to 22 us of 273, this 5.
//
// Every wait is bounded: a wait that runs out raises status bit 4; nothing waits any more from then on, copies in flight are drained
// and tensor memory is freed.
#include <atomic>

#include "attention.cuh"
#include "attention_mma.cuh"
#include "attention_prefill_tc.cuh"
#include "gemm_tc.cuh"
#include "stack_math.cuh"
#include "tc_ptx.cuh"

namespace {

using namespace tc;
using attn_mma::attend_row;
using attn_mma::fast_exp2;
using attn_mma::is_finite;
using attn_mma::LOG2E;
using attn_mma::pack_h2;
using attn_mma::split_h2;

constexpr uint32_t ROWS = 128, KEYS = 128, CHUNK = 128 * 128;  // a chunk: 128 rows of 64 f16
constexpr uint32_t IDESC_B_MN = 1u << 16;

template <int HD, int TILES>
struct Smem {
    static constexpr uint32_t CH = HD / 64, TILE = CH * CHUNK;
    static constexpr uint32_t SLOTS = HD == 128 && TILES == 2 ? 3 : 4;   // ring of key and value tiles in turn
    static constexpr uint32_t ONES = TILES == 1 ? CHUNK : 0;             // 128 rows of ones behind a value tile's slot
    static constexpr uint32_t Q_LO = TILE, Q_PITCH = 2 * TILE, RING = TILES * Q_PITCH;
    static constexpr uint32_t END = RING + SLOTS * TILE + SLOTS / 2 * ONES;
    __device__ static constexpr uint32_t slot(uint32_t s) { return RING + s * TILE + (TILES == 1 ? (s >> 1) * ONES : 0u); }
    // staged output: per warp 32 rows of HD + 4 floats, over the dead tiles
    static constexpr uint32_t OUT_ROW = HD + 4;
    static_assert(TILES * 4 * 32 * OUT_ROW * 4 <= END, "output staging");
    // one CTA per SM: 512 columns of tensor memory are all there is
    static constexpr uint32_t BYTES = (END < 116 * 1024 ? 116 * 1024 : END) + 1024;
};

// MN-major, 128-byte-swizzled operand: 64-element chunks along MN are lbo bytes apart, groups of 8 along K 1024 bytes.
__device__ __forceinline__ uint64_t make_desc_mn(uint32_t smem_addr, uint32_t lbo) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)(lbo >> 4) << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

template <int HD, bool CACHE, int TILES>
__global__ void __launch_bounds__(128 * TILES + 64, 1) prefill_tc_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                                                            M40PrefillTcArgs a) {
    using L = Smem<HD, TILES>;
    extern __shared__ unsigned char smem_unaligned[];
    unsigned char* smem = smem_unaligned + ((1024u - (smem_u32(smem_unaligned) & 1023u)) & 1023u);
    __shared__ uint64_t full[L::SLOTS], empty[L::SLOTS], s_full[2], o_done[2], p_ready[2], q_ready;
    __shared__ uint32_t tmem_slot;
    __shared__ volatile uint32_t abort_flag;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const M40PrefillCall& pc = a.c;
    // Two tiles are the same rows of two q heads that share their keys, or, where a group has an odd number of heads, rows that follow
    // one another. The last rows of a sequence see the most keys: they come first, over all heads and sequences.
    const bool heads2 = TILES == 2 && a.pair_heads;
    const uint32_t b = blockIdx.y, cta_rows = TILES == 2 && !heads2 ? 2 * ROWS : ROWS, cta_r0 = (gridDim.z - 1u - blockIdx.z) * cta_rows;
    const uint32_t mine = TILES == 2 ? threadIdx.x >> 7 : 0u;  // this row thread's tile
    const uint32_t qh = heads2 ? 2u * blockIdx.x + (mine & 1u) : blockIdx.x, r0 = cta_r0 + (TILES == 2 && !heads2 ? mine * ROWS : 0u);
    if (CACHE) pdl_wait();
    const uint32_t q_len = CACHE ? pc.seg[4 * b + 1] : a.q_lens[b];
    const uint32_t kv_len = CACHE ? pc.seg[4 * b + 3] + q_len : a.kv_lens[b];
    if (cta_r0 >= q_len || q_len == 0 || kv_len == 0 || q_len > kv_len) return;
    const uint32_t kvh = (heads2 ? 2u * blockIdx.x : blockIdx.x) / (pc.q_heads / pc.kv_heads);
    const uint32_t slot = CACHE ? pc.seg[4 * b + 2] * pc.slot_mul + pc.slot_add : 0u;
    if (CACHE && (slot >= pc.slots || kv_len > pc.max_seq_len || (uint64_t)pc.seg[4 * b] + q_len > pc.rows)) {
        if (threadIdx.x == 0) atomicOr(a.status, 1u);
        return;
    }
    const size_t q_row0 = (size_t)(CACHE ? pc.seg[4 * b] : a.q_offsets[b]) + r0;
    const int kv_row = (int)(CACHE ? (slot * pc.kv_heads + kvh) * pc.max_seq_len : a.kv_offsets[b]);
    const int kv_col = CACHE ? 0 : (int)(kvh * HD);
    const uint32_t shift = kv_len - q_len;                              // q row i sees keys 0 .. shift + i
    const uint32_t kv_end = shift + min(cta_r0 + cta_rows, q_len);
    const uint32_t n_tiles = (kv_end + KEYS - 1) / KEYS;

    if (threadIdx.x == 0) {
        for (uint32_t i = 0; i < L::SLOTS; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        // [tile of keys % 2], with two tiles of rows [tile]
        for (int i = 0; i < 2; ++i) {
            mbar_init(&s_full[i], 1);
            // One tile: a row waits for a value product now and then only, by parity. Two barriers in turn keep that unambiguous: s_full of
            // tile j says that product j - 2 is done, and product j + 1 cannot be before the row has handed over tile j.
            mbar_init(&o_done[i], 1);
            // S(j + 1) is there before all rows have handed over tile j: a fast warp's next arrival needs a barrier of its own
            mbar_init(&p_ready[i], 128);
        }
        mbar_init(&q_ready, 128 * TILES);
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 4 * TILES + 1) tmem_alloc(&tmem_slot, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (CACHE) pdl_trigger();  // only now: see m40_launch_dependent()
    const uint32_t tmem_s = tmem_slot, tmem_o = tmem_s + 2 * KEYS;
    auto wait = [&](uint64_t* bar, uint32_t parity) {
        if (abort_flag) return false;
        if (mbar_wait(bar, parity)) return true;
        abort_flag = 1;
        atomicOr(a.status, 4u);
        return false;
    };

    uint32_t sent = 0;  // tiles that the loading thread has requested: keys 0, values 0, keys 1, ...
    if (warp == 4 * TILES) {
        if (lane == 0) {
            for (uint32_t s = 0, round = 0; sent < 2u * n_tiles; ++sent) {
                if (round > 0 && !wait(&empty[s], (round - 1u) & 1u)) break;
                mbar_expect_tx(&full[s], L::TILE);
                const CUtensorMap* map = sent & 1u ? &tmV : &tmK;
                for (uint32_t c = 0; c < L::CH; ++c)
                    tma_load_2d(smem + L::slot(s) + c * CHUNK, map, &full[s], kv_col + (int)(c * 64u), kv_row + (int)((sent >> 1) * KEYS));
                if (++s == L::SLOTS) s = 0, ++round;
            }
        }
        __syncwarp();
    } else if (warp == 4 * TILES + 1) {
        // the warp walks the loop converged (see elect_one()), one lane issues
        const uint32_t idesc_s = make_idesc(KEYS), idesc_o = make_idesc(HD + (TILES == 1 ? 16 : 0)) | IDESC_B_MN;
        const uint32_t base_at = smem_u32(smem);
        auto tile_there = [&](uint32_t i) { return (bool)__all_sync(0xffffffffu, wait(&full[i % L::SLOTS], (i / L::SLOTS) & 1u)); };
        // scores of row tile t and key tile j, which is in shared memory; `last`: nothing else reads it
        auto scores = [&](uint32_t t, uint32_t j, bool last) {
            const uint32_t buf = TILES == 2 ? t : j & 1u, k_at = base_at + L::slot(2u * j % L::SLOTS), q_at = base_at + t * L::Q_PITCH;
            tc_fence_after();
            if (elect_one()) {
#pragma unroll
                for (uint32_t k = 0; k < HD / UMMA_K; ++k) {
                    const uint32_t at = (k >> 2) * CHUNK + (k & 3u) * 32u;
                    const uint64_t dk = make_desc_sw128(k_at + at);
                    umma_f16(tmem_s + buf * KEYS, make_desc_sw128(q_at + at), dk, idesc_s, k);
                    umma_f16(tmem_s + buf * KEYS, make_desc_sw128(q_at + L::Q_LO + at), dk, idesc_s, 1u);
                }
                if (last) umma_commit(&empty[2u * j % L::SLOTS]);
                umma_commit(&s_full[buf]);
            }
            __syncwarp();
        };
        bool ok = __all_sync(0xffffffffu, wait(&q_ready, 0));
        // keys of the first tile; one tile of rows works ahead into the second score buffer
        for (uint32_t j = 0; j < (TILES == 1 ? min(n_tiles, 2u) : 1u) && ok; ++j) {
            ok = tile_there(2u * j);
            for (uint32_t t = 0; t < TILES && ok; ++t) scores(t, j, t + 1u == TILES);
        }
        for (uint32_t j = 0; j < n_tiles && ok; ++j) {
            const uint32_t vs = (2u * j + 1u) % L::SLOTS, next = TILES == 1 ? j + 2u : j + 1u;
            ok = tile_there(2u * j + 1u);
            if (!ok) break;
            if ((j + 1) * KEYS > kv_end) {
                const uint32_t first = kv_end - j * KEYS;
                for (uint32_t i = first * 8u + lane; i < KEYS * 8u; i += 32u)
                    for (uint32_t c = 0; c < L::CH; ++c)
                        *reinterpret_cast<uint4*>(smem + L::slot(vs) + c * CHUNK + i * 16u) = make_uint4(0u, 0u, 0u, 0u);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
            }
            for (uint32_t t = 0; t < TILES; ++t) {
                const uint32_t buf = TILES == 2 ? t : j & 1u;
                ok = __all_sync(0xffffffffu, wait(&p_ready[buf], (TILES == 2 ? j : j >> 1) & 1u));
                if (!ok) break;
                tc_fence_after();
                if (elect_one()) {
#pragma unroll
                    for (uint32_t k = 0; k < KEYS / UMMA_K; ++k)
                        umma_f16_ts(tmem_o + t * HD, tmem_s + buf * KEYS + k * 8u, make_desc_mn(base_at + L::slot(vs) + k * 2048u, CHUNK), idesc_o, j | k);
                    if (t + 1u == TILES) umma_commit(&empty[vs]);
                    if (TILES == 1 || j + 1u == n_tiles) umma_commit(&o_done[buf]);
                }
                __syncwarp();
                if (next < n_tiles) {  // into the buffer whose weights the MMAs above read first
                    if (t == 0) ok = tile_there(2u * next);
                    if (!ok) break;
                    scores(t, next, t + 1u == TILES);
                }
            }
        }
    } else {
        const uint32_t tid = threadIdx.x & 127u, quarter = warp & 3u, row = r0 + tid;
        const uint32_t lane_addr = (quarter * 32u) << 16, my_o = tmem_o + mine * HD + lane_addr;
        unsigned char* my_q = smem + mine * L::Q_PITCH;
        // ---- the queries, scaled to base 2, as f16 hi and lo
        {
            const float qs = pc.scale * LOG2E;
            constexpr uint32_t PIECES = HD / 8;
#pragma unroll 8
            for (uint32_t i = tid; i < ROWS * PIECES; i += 128u) {
                const uint32_t r = i / PIECES, p = i % PIECES;
                float4 x0 = make_float4(0.f, 0.f, 0.f, 0.f), x1 = x0;
                if (r0 + r < q_len && p * 8u < pc.q_dim) {
                    const float4* q = reinterpret_cast<const float4*>(pc.q + (q_row0 + r) * pc.q_ld + qh * pc.q_dim + p * 8u);
                    x0 = q[0], x1 = q[1];
                }
                uint32_t hi[4], lo[4];
                split_h2(x0.x * qs, x0.y * qs, &hi[0], &lo[0]);
                split_h2(x0.z * qs, x0.w * qs, &hi[1], &lo[1]);
                split_h2(x1.x * qs, x1.y * qs, &hi[2], &lo[2]);
                split_h2(x1.z * qs, x1.w * qs, &hi[3], &lo[3]);
                unsigned char* dst = my_q + (p >> 3) * CHUNK + r * 128u + (((p & 7u) ^ (r & 7u)) << 4);
                *reinterpret_cast<uint4*>(dst) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                *reinterpret_cast<uint4*>(dst + L::Q_LO) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
            }
            if constexpr (L::ONES > 0) {
                const uint4 ones = make_uint4(0x3c003c00u, 0x3c003c00u, 0x3c003c00u, 0x3c003c00u);
                for (uint32_t i = tid * 16u; i < L::ONES; i += 128u * 16u)
                    for (uint32_t v = 1; v < 4; v += 2) *reinterpret_cast<uint4*>(smem + L::slot(v) + L::TILE + i) = ones;
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            mbar_arrive(&q_ready);
        }
        const uint32_t lim = shift + min(row, q_len - 1u);  // last key this row sees
        float ref = -INFINITY, l = 0.0f;  // l: the denominator; with one tile only the sink's part of it
        if (CACHE && pc.sink) {  // a sink is a key whose score is known from the start and whose value is zero
            ref = pc.sink[qh] * LOG2E;
            l = 1.0f;
        }
        bool ok = true;
        for (uint32_t j = 0; j < n_tiles && ok; ++j) {
            const uint32_t base = j * KEYS, buf = TILES == 2 ? mine : j & 1u, phase = (TILES == 2 ? j : j >> 1) & 1u, s_at = tmem_s + buf * KEYS + lane_addr;
            ok = __all_sync(0xffffffffu, wait(&s_full[buf], phase));  // tensor-memory loads are warp-collective
            if (!ok) break;
            tc_fence_after();
            const bool all_seen = base + KEYS - 1u <= shift + min(r0 + quarter * 32u, q_len - 1u);  // by every row of the warp
            // One tile keeps the scores in registers; two leave fewer registers, and fetch them again for the weights.
            constexpr uint32_t HELD = TILES == 1 ? KEYS : 64;
            uint32_t raw[HELD];
            float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (uint32_t h = 0; h < KEYS; h += HELD) {
#pragma unroll
                for (uint32_t i = 0; i < HELD; i += 64) tmem_ld_x64(s_at + h + i, raw + i);
                tmem_ld_wait();
                if (!all_seen) {
#pragma unroll
                    for (uint32_t i = 0; i < HELD; ++i)
                        if (base + h + i > lim) raw[i] = 0xff800000u;
                }
#pragma unroll
                for (uint32_t i = 0; i < HELD; ++i) mx[i & 3u] = fmaxf(mx[i & 3u], __uint_as_float(raw[i]));
            }
            const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
            const bool grow = top > ref;
            float corr = 1.0f;
            if (grow) {
                corr = fast_exp2(ref - top);
                ref = top;
                l *= corr;
            }
            const bool rescale = j > 0 && __any_sync(0xffffffffu, grow);
            if (TILES == 1 && rescale) {  // two tiles: these scores were issued behind the value product, and are there
                ok = __all_sync(0xffffffffu, wait(&o_done[(j - 1u) & 1u], ((j - 1u) >> 1) & 1u));
                tc_fence_after();
            }
            const float use = ref == -INFINITY ? 0.0f : ref;
            float sum[4] = {};
            // The outputs so far are rescaled: by two tiles piece by piece while the exponentials are computed, fetched before, stored behind
            // them; by one tile first of all, so that its exponentials are one straight run (130 rows over 4000 keys, 32 / 8 heads of 128: 56.5
            // us, piece by piece 59.3; two tiles with the exponentials in a run of their own for either case: 126 -> 164 us for 640 rows there).
            constexpr uint32_t PIECES = KEYS / 32, O_COLS = HD / PIECES;
            if (TILES == 1 && rescale) {
#pragma unroll
                for (uint32_t c = 0; c < HD + 16; c += 16) {
                    uint32_t r[16];
                    tmem_ld_x16(my_o + c, r);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 16; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * corr);
                    tmem_st_x16(my_o + c, r);
                }
            }
#pragma unroll
            for (uint32_t c = 0; c < PIECES; ++c) {
                uint32_t o[O_COLS], again[32], p[16];
                if (TILES == 2) tmem_ld_x32(s_at + 32u * c, again);
                if (TILES == 2) tmem_ld_wait();
                if (TILES == 2 && rescale) {
#pragma unroll
                    for (uint32_t i = 0; i < O_COLS; i += 16) tmem_ld_x16(my_o + c * O_COLS + i, o + i);
                }
#pragma unroll
                for (uint32_t i = 0; i < 16; ++i) {
                    float s0, s1;
                    if (TILES == 1) {
                        s0 = __uint_as_float(raw[(32u * c + 2u * i) % HELD]), s1 = __uint_as_float(raw[(32u * c + 2u * i + 1u) % HELD]);
                    } else {
                        s0 = __uint_as_float(again[2 * i]), s1 = __uint_as_float(again[2 * i + 1]);
                        if (!all_seen) {
                            if (base + 32u * c + 2u * i > lim) s0 = -INFINITY;
                            if (base + 32u * c + 2u * i + 1u > lim) s1 = -INFINITY;
                        }
                    }
                    p[i] = pack_h2(fast_exp2(s0 - use), fast_exp2(s1 - use));
                    if (TILES == 2) {  // the rounded weights, which the values are multiplied with
                        const float2 w = __half22float2(*reinterpret_cast<const __half2*>(&p[i]));
                        sum[(2 * i) & 3] += w.x, sum[(2 * i + 1) & 3] += w.y;
                    }
                }
                if (TILES == 2 && rescale) {
                    tmem_ld_wait();
#pragma unroll
                    for (uint32_t i = 0; i < O_COLS; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * corr);
#pragma unroll
                    for (uint32_t i = 0; i < O_COLS; i += 16) tmem_st_x16(my_o + c * O_COLS + i, o + i);
                }
                tmem_st_x16(s_at + 16u * c, p);
            }
            tmem_st_wait();
            tc_fence_before();
            if (TILES == 2) l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
            mbar_arrive(&p_ready[buf]);
        }
        if (TILES == 1) {
            ok = ok && __all_sync(0xffffffffu, wait(&o_done[(n_tiles - 1u) & 1u], ((n_tiles - 1u) >> 1) & 1u));
        } else {  // both: the output is staged over tiles of either
            ok = ok && __all_sync(0xffffffffu, wait(&o_done[0], 0u) && wait(&o_done[1], 0u));
        }
        if (ok) {
            tc_fence_after();
            float o[HD];
            {
                uint32_t r[HD];
                tmem_ld_x64(my_o, r);
                if (HD == 128) tmem_ld_x64(my_o + 64u, r + HD - 64);
                uint32_t weights[4] = {};  // equal columns
                if (TILES == 1) tmem_ld_x4(my_o + HD, weights);
                tmem_ld_wait();
                l += __uint_as_float(weights[0]);
#pragma unroll
                for (int i = 0; i < HD; ++i) o[i] = __uint_as_float(r[i]);
            }
            float* stage = reinterpret_cast<float*>(smem) + warp * 32u * L::OUT_ROW;  // nothing reads or writes a tile any more
            float* mine = stage + lane * L::OUT_ROW;
            float nan[4] = {};
#pragma unroll
            for (int i = 0; i < HD; ++i) nan[i & 3] = fmaf(o[i], 0.0f, nan[i & 3]);
            uint32_t again = __ballot_sync(0xffffffffu, row < q_len && !is_finite((nan[0] + nan[1]) + (nan[2] + nan[3])));
            if (again) {
#pragma unroll
                for (int i = 0; i < HD; ++i) mine[i] = o[i];
                __syncwarp();
                const size_t pitch = CACHE ? HD : (size_t)pc.kv_heads * HD, at = (size_t)kv_row * pitch + kv_col;
                for (; again; again &= again - 1u) {
                    const uint32_t r = __ffs(again) - 1u, t = quarter * 32u + r;
                    const float from = __shfl_sync(0xffffffffu, ref, r);
                    const float4 v = attend_row<HD>(pc.q + (q_row0 + t) * pc.q_ld + qh * pc.q_dim, pc.q_dim, pc.scale * LOG2E, pc.K + at,
                                                    pc.V + at, pitch, shift + r0 + t + 1u, from == -INFINITY ? 0.0f : from);
                    float* d = stage + r * L::OUT_ROW + 2u * lane;
                    if (!is_finite(d[0])) d[0] = v.x;
                    if (!is_finite(d[1])) d[1] = v.y;
                    if (HD == 128 && !is_finite(d[64])) d[64] = v.z;
                    if (HD == 128 && !is_finite(d[65])) d[65] = v.w;
                }
                __syncwarp();
#pragma unroll
                for (int i = 0; i < HD; ++i) o[i] = mine[i];
            }
            float inv = 1.0f / (l > 0.0f ? l : 1.0f);
            if (CACHE && pc.turn_back) {
                const float4* t = reinterpret_cast<const float4*>(pc.turn_back + (q_row0 - r0 + min(row, q_len - 1u)) * (HD / 2));
#pragma unroll
                for (int i = 0; i < HD / 4; ++i) {
                    const float4 cs = t[i];
                    const float u0 = o[2 * i], v0 = o[2 * i + HD / 2], u1 = o[2 * i + 1], v1 = o[2 * i + 1 + HD / 2];
                    o[2 * i] = u0 * cs.x + v0 * cs.y;
                    o[2 * i + HD / 2] = v0 * cs.x - u0 * cs.y;
                    o[2 * i + 1] = u1 * cs.z + v1 * cs.w;
                    o[2 * i + 1 + HD / 2] = v1 * cs.z - u1 * cs.w;
                }
            }
            if (CACHE && pc.gate && row < q_len) inv *= m40_sigmoid(pc.gate[(q_row0 + tid) * pc.gate_ld + qh]);
            // rows leave through shared memory, whole lines at a time
#pragma unroll
            for (int i = 0; i < HD; i += 4)
                *reinterpret_cast<float4*>(mine + i) =
                    make_float4(o[i] * inv, o[i + 1] * inv, o[i + 2] * inv, o[i + 3] * inv);
            __syncwarp();
            constexpr uint32_t PER = HD / 4;  // float4 per row
            for (uint32_t i = lane; i < 32u * PER; i += 32u) {
                const uint32_t r = i / PER, c = (i % PER) * 4u;
                if (r0 + quarter * 32u + r < q_len && c < pc.v_dim)
                    *reinterpret_cast<float4*>(pc.out + (q_row0 + quarter * 32u + r) * pc.out_ld + qh * pc.v_dim + c) =
                        *reinterpret_cast<const float4*>(stage + r * L::OUT_ROW + c);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (abort_flag && warp == 4 * TILES && lane == 0)  // copies in flight land (bounded) before the CTA goes away
        for (uint32_t i = sent > L::SLOTS ? sent - L::SLOTS : 0u; i < sent; ++i) {
            const uint32_t s = i % L::SLOTS;
            mbar_wait(&full[s], (i / L::SLOTS) & 1u);
        }
    if (warp == 4 * TILES + 1) {
        tc_fence_after();
        tmem_dealloc(tmem_slot, 512);
    }
}

template <int HD, bool CACHE, int TILES>
int launch(M40llmCudaContext* ctx, cudaStream_t s, const CUtensorMap& mk, const CUtensorMap& mv, const M40PrefillTcArgs& a) {
    // contexts on several threads may set it at the same time: setting it twice is harmless, losing another device's bit is not
    static std::atomic<unsigned long long> configured{0ull};
    const unsigned long long bit = 1ull << (ctx->device_id & 63);
    if (!(configured.load(std::memory_order_acquire) & bit)) {
        if (cudaFuncSetAttribute(prefill_tc_kernel<HD, CACHE, TILES>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Smem<HD, TILES>::BYTES) !=
            cudaSuccess)
            return -4;
        configured.fetch_or(bit, std::memory_order_release);
    }
    const uint32_t rows = TILES == 2 && !a.pair_heads ? 2 * ROWS : ROWS;
    const dim3 grid(TILES == 2 && a.pair_heads ? a.c.q_heads / 2 : a.c.q_heads, a.c.segments, (a.c.max_segment_rows + rows - 1) / rows);
    cudaError_t e;
    if (CACHE) {
        e = m40_launch_dependent(prefill_tc_kernel<HD, CACHE, TILES>, grid, dim3(128 * TILES + 64), Smem<HD, TILES>::BYTES, s, mk, mv, a);
    } else {
        prefill_tc_kernel<HD, CACHE, TILES><<<grid, 128 * TILES + 64, Smem<HD, TILES>::BYTES, s>>>(mk, mv, a);
        e = cudaSuccess;
    }
    M40_COUNT_LAUNCH(ctx);
    return e == cudaSuccess && cudaGetLastError() == cudaSuccess ? 0 : -4;
}

}  // namespace

int m40_attention_prefill_tc(M40llmCudaContext* ctx, cudaStream_t s, const M40PrefillTcArgs& call, uint64_t kv_rows) {
    M40PrefillTcArgs a = call;
    const M40PrefillCall& c = a.c;
    const bool cache = c.seg != nullptr;
    if (c.hd != 64 && c.hd != 128) return 1;
    if (c.max_segment_rows < M40_PREFILL_TC_MIN_ROWS) return 1;
    if (((((uintptr_t)c.q) | ((uintptr_t)c.out) | ((uintptr_t)c.K) | ((uintptr_t)c.V) | ((uintptr_t)c.turn_back)) & 15u) != 0u) return 1;
    if (c.q_dim % 8 != 0 || c.v_dim % 4 != 0 || c.q_ld % 4 != 0 || c.out_ld % 4 != 0 || kv_rows >= 0x7fffffffull) return 1;
    CUtensorMap mk, mv;
    const uint64_t cols = cache ? c.hd : (uint64_t)c.kv_heads * c.hd;
    if (!m40_tc_map(&mk, c.K, kv_rows, cols, KEYS, false) || !m40_tc_map(&mv, c.V, kv_rows, cols, KEYS, false)) return 1;
    a.pair_heads = c.q_heads / c.kv_heads % 2 == 0 ? 1u : 0u;
    const bool two = a.two_tiles != 0u;
    if (c.hd == 128)
        return cache ? (two ? launch<128, true, 2>(ctx, s, mk, mv, a) : launch<128, true, 1>(ctx, s, mk, mv, a))
                     : (two ? launch<128, false, 2>(ctx, s, mk, mv, a) : launch<128, false, 1>(ctx, s, mk, mv, a));
    return cache ? (two ? launch<64, true, 2>(ctx, s, mk, mv, a) : launch<64, true, 1>(ctx, s, mk, mv, a))
                 : (two ? launch<64, false, 2>(ctx, s, mk, mv, a) : launch<64, false, 1>(ctx, s, mk, mv, a));
}
