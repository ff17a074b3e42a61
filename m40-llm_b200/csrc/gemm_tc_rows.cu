// Projections of 2 to 32 activation rows on tcgen05 in ONE launch: f32 activations in, finished result out.
//
// C[m][n] = sum_k X[m][k] W[n][k] is computed "swapped": a tile of 128 weight rows is the MMA's A operand and the activation rows,
// padded to a multiple of 16, are the B operand, so that the tensor core runs at full height however few rows there are and every
// weight byte is read from HBM once. The f32 activations are split into 16-bit hi + lo parts, which lie one behind the other as one
// operand of 2 * M_pad rows: one MMA per k-step, the two halves of the accumulator are added when it is read. The tensor core truncates
// as it adds up, by more the longer a sum grows, so a CTA's k-blocks go in two runs with accumulators of their own: 16 sums for K where
// there are 8 splits (256 x 8192: an error of 6e-7 of the norm against 64 bits, with one run 1.2e-6).
//
//   warp 0      weight tiles by TMA into a ring of 64-deep stages; those of the first pass are requested before the dependency wait
//   warp 1      issues the MMAs
//   warps 2..5  make the activation operand: f32 values, prefetched in registers, -> hi and lo -> swizzled
//               shared memory, a k-block per warp; then they take the accumulator out of tensor memory
//   all         add the K splits and finish the result
//
// K is split over the CTAs of a cluster (up to 8), each of which finishes its share of the tile's rows: a CTA leaves its sums over its ring
// and sends every other CTA that one's rows (a bulk copy each, counted by the receiver's mbarrier). Sums are added in a fixed order; then
// bias, norm, residual, soft cap, gate or RoPE with cache append.
//
// At this few rows a call is a chain of latencies beside a stream of weights, and the split, the sums and the epilogue as launches of
// their own cost more than their work: 16 rows of 4096 x 4096 took 12.8 us with them and take 8.8, 4096 x 14336 32.5 and 22.0, 32 rows of
// 2048 x 2048 9.2 and 6.2. A norm or activation of x is not applied here: every tile's CTA would do it again (a dynamic tanh of
// 16 x 4096 values in each of 224 CTAs: 87 us against 39 with a split kernel); calls with one, calls whose result lies over x and calls of more
// than 16 rows with more tiles than SMs come split already (M40_ROWS_SPLIT).
//
// Every wait is bounded: a wait that runs out raises status bit 4; all threads still meet at the barriers, copies in flight land
// (bounded) and tensor memory is freed.
#include <atomic>

#include "gemm_tc_rows.cuh"
#include "tc_ptx.cuh"

namespace {

using namespace tc;

constexpr uint32_t THREADS = 192, A_BYTES = BLOCK_N * BLOCK_K * 2;
// ring and sums; two CTAs per SM, of whose 114 KB each 1 KB is the system's and less than 1 KB control data
constexpr uint32_t SMEM_BYTES = 112u * 1024u, MIN_STAGES = 4, MAX_STAGES = 8, MAX_SPLITS = 8;

template <int SRC>
struct Part {
    using T = __half;
};
template <>
struct Part<M40_ROWS_BF16> {
    using T = __nv_bfloat16;
};
__device__ __forceinline__ void split1(float v, __half* h, __half* l) {
    *h = __float2half_rn(v);
    *l = __float2half_rn(v - __half2float(*h));
}
__device__ __forceinline__ void split1(float v, __nv_bfloat16* h, __nv_bfloat16* l) {
    *h = __float2bfloat16_rn(v);
    *l = __float2bfloat16_rn(v - __bfloat162float(*h));
}
// The arrivals order no data: they say that a CTA's barriers are in place, and later that it will not be read or written any more. (With
// .release a thread waits about 0.6 us for its writes.)
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void copy_to_cluster(uint32_t dst, uint32_t src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "r"(src), "r"(bytes),
                 "r"(bar)
                 : "memory");
}

// Behind ring and sums.
struct Control {
    M40RowsArgs tail;  // parameters that are first needed at the end would be fetched one miss after the other there
    uint64_t w_full[MAX_STAGES], x_full[MAX_STAGES], empty[MAX_STAGES], accum, received;
    uint32_t tmem_slot;
    uint32_t abort_flag;
};

// The activation operand, by four warps: each takes every fourth k-block as a whole, so that the fence that hands one to the tensor core
// (hundreds of cycles) is waited for by one warp while the others work. A lane owns column chunk lane % 8 (16 bytes of 16-bit values) of
// rows lane / 8 + 4 i. Sixteen rows are a step; PF steps are on their way from L2 while one is converted.
template <int SRC, int UNITS>
__device__ __forceinline__ void make_operand(const M40RowsArgs& a, unsigned char* ring, uint32_t stage_bytes, uint64_t* x_full, uint64_t* empty,
                                             volatile uint32_t* abort_flag, uint32_t kb0, uint32_t n_kb) {
    using T = typename Part<SRC>::T;
    constexpr int PF = 3;
    const uint32_t w = (threadIdx.x >> 5) - 2u, lane = threadIdx.x & 31u, c = lane & 7u, r0 = lane >> 3;
    const uint32_t steps = n_kb > w ? (n_kb - w + 3u) / 4u * UNITS : 0u;
    float4 x[PF][8];
    auto fetch = [&](uint32_t t, int at) {  // every load is unconditional: clamped here, masked below
        const uint32_t col = (kb0 + w + t / UNITS * 4u) * BLOCK_K + c * 8u, row = t % UNITS * 16u + r0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float4* p = reinterpret_cast<const float4*>(a.x + (size_t)min(row + 4u * i, a.M - 1u) * a.ldx + (col < a.K ? col : 0u));
            x[at][2 * i] = p[0], x[at][2 * i + 1] = p[1];
        }
    };
#pragma unroll
    for (int j = 0; j < PF; ++j)
        if ((uint32_t)j < steps) fetch(j, j);
    uint32_t s = w % a.stages, round = w / a.stages;
    bool ok = true;
    for (uint32_t t0 = 0; t0 < steps && ok; t0 += PF) {
#pragma unroll
        for (int j = 0; j < PF; ++j) {
            const uint32_t t = t0 + j, half = t % UNITS;
            if (t >= steps || !ok) continue;
            // A parity wait only tells adjacent uses of a stage apart. The use after the one waited for is this k-block's own. The use
            // before it is over, since this warp has waited for a later one, four k-blocks ago: the ring has at least MIN_STAGES = 4.
            if (half == 0 && round > 0) ok = __all_sync(0xffffffffu, !*abort_flag && mbar_wait(&empty[s], (round - 1u) & 1u));
            if (!ok) continue;
            const bool in = (kb0 + w + t / UNITS * 4u) * BLOCK_K + c * 8u < a.K;
            unsigned char* dst = ring + s * stage_bytes + A_BYTES;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t row = half * 16u + r0 + 4u * i;
                const float4 p = x[j][2 * i], q = x[j][2 * i + 1];
                const float v[8] = {p.x, p.y, p.z, p.w, q.x, q.y, q.z, q.w};
                const bool live = in && row < a.M;
                T h[8], l[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) split1(live ? v[e] : 0.0f, &h[e], &l[e]);
                const uint32_t at = row * 128u + ((c ^ (row & 7u)) << 4);
                *reinterpret_cast<uint4*>(dst + at) = *reinterpret_cast<const uint4*>(h);
                *reinterpret_cast<uint4*>(dst + UNITS * 2048u + at) = *reinterpret_cast<const uint4*>(l);
            }
            if (t + PF < steps) fetch(t + PF, j);
            if (half + 1u < UNITS) continue;
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&x_full[s]);
            s += 4u;
            if (s >= a.stages) s -= a.stages, ++round;
        }
    }
    if (!ok) *abort_flag = 1;
}

// grid (tiles, K splits), the K splits of a tile are a cluster. SRC: M40_ROWS_*. UNITS: sixteens of rows.
template <int SRC, int UNITS>
__global__ void __launch_bounds__(THREADS, 2) gemm_tc_rows_kernel(const __grid_constant__ CUtensorMap tmW0, const __grid_constant__ CUtensorMap tmW1,
                                                                  const __grid_constant__ CUtensorMap tmW2,
                                                                  const __grid_constant__ CUtensorMap tmXh,
                                                                  const __grid_constant__ CUtensorMap tmXl, const __grid_constant__ M40RowsArgs a) {
    constexpr uint32_t M_pad = 16 * UNITS, b_bytes = M_pad * BLOCK_K * 2, stage_bytes = A_BYTES + 2 * b_bytes;
    constexpr uint32_t acc_cols = 2 * M_pad, tmem_cols = 2 * acc_cols;  // two runs of k-blocks; 64 or 128
    extern __shared__ __align__(1024) unsigned char ring[];  // swizzled tiles start on 1024-byte boundaries
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t tile = blockIdx.x, ks = gridDim.y, split = blockIdx.y;
    // this CTA finishes rows m0 .. m1 - 1; their sums arrive as [split][row][128] behind the ring, or lie over every CTA's ring
    const uint32_t share = (a.M + ks - 1u) / ks, m0 = min(split * share, a.M), m1 = min(m0 + share, a.M);
    unsigned char* sums = ks > 1 ? ring + a.stages * stage_bytes : ring;
    Control& ctl = *reinterpret_cast<Control*>(ring + a.stages * stage_bytes + (ks > 1 ? ks * share * BLOCK_N * 4u : 0u));
    uint64_t *w_full = ctl.w_full, *x_full = ctl.x_full, *empty = ctl.empty;
    volatile uint32_t& abort_flag = ctl.abort_flag;

    uint32_t problem = 0;
    while (problem + 1 < a.problems && tile >= a.tile_begin[problem + 1]) ++problem;
    const CUtensorMap* tmW = problem == 0 ? &tmW0 : (problem == 1 ? &tmW1 : &tmW2);
    const uint32_t n_rows = a.paired ? BLOCK_N / 2 : BLOCK_N, row0 = (tile - a.tile_begin[problem]) * n_rows;
    const uint32_t kb0 = split * a.kb_per_split, kb1 = min(kb0 + a.kb_per_split, a.kblocks);
    const uint32_t n_kb = kb1 > kb0 ? kb1 - kb0 : 0u, run = (n_kb + 1u) / 2u;  // blocks of the first run; the second has run or one less

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < a.stages; ++s) {
            mbar_init(&w_full[s], 1);
            mbar_init(&x_full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(&ctl.accum, 1);
        mbar_init(&ctl.received, 1);
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (ks > 1) mbar_expect_tx(&ctl.received, ks * (m1 - m0) * BLOCK_N * 4u);
    }
    if (warp == 1) tmem_alloc(&ctl.tmem_slot, tmem_cols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = ctl.tmem_slot;
    pdl_trigger();
    if (ks > 1) cluster_arrive();  // the others' barriers are in place once this has been waited for

    uint32_t sent = 0;  // stages that the loading thread has requested
    if (warp == 0) {
        if (lane == 0) {
            auto load_w = [&](uint32_t i, uint32_t s) {
                unsigned char* st = ring + s * stage_bytes;
                const int kx = (int)((kb0 + i) * BLOCK_K);
                mbar_expect_tx(&w_full[s], SRC == M40_ROWS_SPLIT ? stage_bytes : A_BYTES);
                tma_load_2d(st, tmW, &w_full[s], kx, (int)row0);
                if (a.paired) tma_load_2d(st + A_BYTES / 2, &tmW1, &w_full[s], kx, (int)row0);
            };
            auto load_x = [&](uint32_t i, uint32_t s) {
                unsigned char* st = ring + s * stage_bytes + A_BYTES;
                const int kx = (int)((kb0 + i) * BLOCK_K);
                tma_load_2d(st, &tmXh, &w_full[s], kx, 0);
                tma_load_2d(st + b_bytes, &tmXl, &w_full[s], kx, 0);
            };
            const uint32_t pre = min(n_kb, a.stages);
            for (; sent < pre; ++sent) load_w(sent, sent);
            if (SRC == M40_ROWS_SPLIT) {
                pdl_wait();
                for (uint32_t i = 0; i < pre; ++i) load_x(i, i);
            }
            for (uint32_t i = pre, s = 0, round = 1; i < n_kb; ++i) {
                if (abort_flag || !mbar_wait(&empty[s], (round - 1) & 1u)) { abort_flag = 1; break; }
                load_w(i, s);
                if (SRC == M40_ROWS_SPLIT) load_x(i, s);
                ++sent;
                if (++s == a.stages) s = 0, ++round;
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // the warp walks the loop converged (see elect_one()), one lane issues
        const uint32_t idesc = make_idesc(2u * M_pad) | a.fmt_bits;
        uint32_t s = 0, phase = 0;
        for (uint32_t i = 0; i < n_kb; ++i) {
            bool there = !abort_flag && mbar_wait(&w_full[s], phase);
            if (SRC != M40_ROWS_SPLIT) there = there && mbar_wait(&x_full[s], phase);
            if (!__all_sync(0xffffffffu, there)) { abort_flag = 1; break; }
            tc_fence_after();
            const uint32_t sa = smem_u32(ring + s * stage_bytes), sb = sa + A_BYTES;
            const uint32_t acc = tmem_base + (i < run ? 0u : acc_cols), older = i < run ? i : i - run;
            if (elect_one()) {
#pragma unroll
                for (uint32_t k = 0; k < BLOCK_K / UMMA_K; ++k)
                    umma_f16(acc, make_desc_sw128(sa + k * UMMA_K * 2), make_desc_sw128(sb + k * UMMA_K * 2), idesc, older | k);
                umma_commit(&empty[s]);              // frees the stage once these MMAs have read it
                if (i + 1 == n_kb) umma_commit(&ctl.accum);
            }
            __syncwarp();
            if (++s == a.stages) s = 0, phase ^= 1u;
        }
    } else {
        for (uint32_t i = threadIdx.x - 64u; i < sizeof(M40RowsArgs) / 4u; i += 128u)
            reinterpret_cast<uint32_t*>(&ctl.tail)[i] = reinterpret_cast<const uint32_t*>(&a)[i];
        pdl_wait();
        if constexpr (SRC != M40_ROWS_SPLIT) {
            make_operand<SRC, UNITS>(a, ring, stage_bytes, x_full, empty, &abort_flag, kb0, n_kb);
        }
        bool ok = n_kb > 0;
        if (ok && !mbar_wait(&ctl.accum, 0)) { abort_flag = 1; ok = false; }
        ok = __all_sync(0xffffffffu, ok);  // tcgen05.ld is warp-collective
        tc_fence_after();
        const uint32_t n = (warp & 3u) * 32u + lane, at = tmem_base + (((warp & 3u) * 32u) << 16);
        float* acc = reinterpret_cast<float*>(ring) + n;  // [M][128]: every MMA has read the ring
        float v[M_pad] = {};
        uint32_t z[64];
#pragma unroll
        for (uint32_t c = 0; c < tmem_cols; c += 64) {  // both runs at 16 rows, a run at 32; in pieces of 16 columns: 0.35 us a piece
            if (!ok) continue;
            tmem_ld_x64(at + c, z);
            tmem_ld_wait();
#pragma unroll
            for (uint32_t r = 0; r < 64; r += acc_cols) {
                if (c + r > 0 && n_kb == 1u) continue;  // there is no second run: those columns may hold anything
#pragma unroll
                for (uint32_t j = 0; j < M_pad; ++j) v[j] += __uint_as_float(z[r + j]) + __uint_as_float(z[r + M_pad + j]);
            }
        }
#pragma unroll
        for (uint32_t j = 0; j < M_pad; ++j)
            if (j < a.M) acc[j * BLOCK_N] = v[j];
        tc_fence_before();
        if (ks > 1) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("bar.sync 1, 128;" ::: "memory");
            cluster_wait();
            const uint32_t first = lane * share, bytes = min(share, a.M - min(first, a.M)) * (BLOCK_N * 4u);
            if (warp == 2 && lane < ks && bytes > 0)
                copy_to_cluster(map_to_rank(smem_u32(sums) + split * bytes, lane), smem_u32(ring) + first * (BLOCK_N * 4u), bytes,
                                map_to_rank(smem_u32(&ctl.received), lane));
            __syncwarp();
        }
    }
    if (ks > 1 && warp < 2u) cluster_wait();
    pdl_wait();  // the residual, and whatever earlier kernels still read of the result's memory
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, tmem_cols);
    }
    if (ks > 1) {
        if (!mbar_wait_cluster(&ctl.received, 0)) abort_flag = 1;
        __syncwarp();
        cluster_arrive();  // the second time: this CTA has what it was sent
    }

    // ---- sums and tail of rows m0 .. m1 - 1, four adjacent outputs a time
    const M40RowsArgs& ta = ctl.tail;
    const uint32_t per_row = n_rows / 4u, N = ta.N[problem];
    auto total = [&](uint32_t m, uint32_t col) {
        float4 v[MAX_SPLITS], t = make_float4(0.f, 0.f, 0.f, 0.f);
        if (ks == 1) return *reinterpret_cast<const float4*>(sums + (m * BLOCK_N + col) * 4u);
#pragma unroll
        for (uint32_t k = 0; k < MAX_SPLITS; ++k) {  // unconditional, so that all are on their way together
            const uint32_t j = min(k, ks - 1u);
            v[k] = *reinterpret_cast<const float4*>(sums + ((j * (m1 - m0) + m - m0) * BLOCK_N + col) * 4u);
        }
#pragma unroll
        for (uint32_t k = 0; k < MAX_SPLITS; ++k)
            if (k < ks) t.x += v[k].x, t.y += v[k].y, t.z += v[k].z, t.w += v[k].w;
        return t;
    };
    float* out = ta.out[problem];
    for (uint32_t u = m0 * per_row + threadIdx.x; u < m1 * per_row; u += THREADS) {
        const uint32_t m = u / per_row, n4 = (u % per_row) * 4u, n = row0 + n4;
        if (n >= N) continue;
        const size_t at = (size_t)m * N + n;
        const uint32_t live = min(N - n, 4u);
        float y[4];
        if (ta.paired) {
            const float4 t = total(m, n4), up = total(m, BLOCK_N / 2 + n4);
            const float g[4] = {t.x, t.y, t.z, t.w}, z[4] = {up.x, up.y, up.z, up.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) y[j] = m40_act(ta.act, g[j]) * z[j];
        } else {
            const float *bias = ta.bias[problem], *residual = ta.residual[problem];
            float add[4], res[4], pw[4], pb[4];
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) {
                const uint32_t i = j < live ? j : 0u;
                res[j] = residual ? residual[at + i] : 0.0f;
                add[j] = bias ? bias[n + i] : 0.0f;
                pw[j] = ta.post_w ? ta.post_w[n + i] : 1.0f;
                pb[j] = ta.post_b ? ta.post_b[n + i] : 0.0f;
            }
            const float4 t = total(m, n4);
            const float v[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) y[j] = m40_tail(ta.tail, v[j], add[j], pw[j], pb[j], res[j]);
        }
        if (ta.rope_on) {
            // q | k | v: RoPE on adjacent pairs of q and k, then q to its buffer and k, v as f16 into the cache row of this position
            const M40TcRopeAppend& ra = ta.rope;
            const uint32_t seq = ra.seq_ids[m], pos = ra.positions[m];
            if (seq >= ra.max_batch || pos >= ra.max_seq_len) {
                if (problem == 0 && n == 0) atomicOr(ra.status, 2u);
                continue;
            }
#pragma unroll
            for (uint32_t h = 0; h < 2; ++h) {
                const uint32_t d = (n + 2 * h) % ra.head_dim, head = (n + 2 * h) / ra.head_dim;
                if (problem < 2) {
                    float c, sn;
                    rope_cs(pos, d >> 1, ra.head_dim, ra.freq_base, ra.freq_scale, &c, &sn, ra.inv_freq);
                    const float p = y[2 * h], q = y[2 * h + 1];
                    y[2 * h] = p * c - q * sn;
                    y[2 * h + 1] = p * sn + q * c;
                }
                if (problem == 0) continue;
                const size_t to = kv_row_offset(seq, head, pos, ra.kv_heads, ra.max_seq_len, ra.head_dim) + d;
                *reinterpret_cast<__half2*>((problem == 1 ? ra.d_k : ra.d_v) + to) = __floats2half2_rn(y[2 * h], y[2 * h + 1]);
            }
            if (problem > 0) {
                if (problem == 1 && n == 0) ra.d_seq_map[seq] = pos + 1u;
                continue;
            }
        }
        if (ta.vec_out >> problem & 1u) {
            *reinterpret_cast<float4*>(out + at) = make_float4(y[0], y[1], y[2], y[3]);
        } else {
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j)
                if (j < live) out[at + j] = y[j];
        }
    }
    if (ks > 1) {  // no CTA leaves while its copies are under way
        __syncwarp();
        cluster_wait();
    }
    if (threadIdx.x == 0 && abort_flag) {
        atomicOr(a.status, 4u);
        for (uint32_t i = sent > a.stages ? sent - a.stages : 0u; i < sent; ++i) mbar_wait(&w_full[i % a.stages], (i / a.stages) & 1u);
    }
}

// Stands in for the above where the occupancy is asked for: of a kernel that takes tensor memory the runtime says that one CTA fits an
// SM, whatever it takes.
__global__ void __launch_bounds__(THREADS, 2) footprint_kernel(uint32_t* p) {
    extern __shared__ __align__(1024) unsigned char ring[];
    if (p) p[threadIdx.x] = ring[threadIdx.x];
}

using Kernel = void (*)(CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, M40RowsArgs);

template <int SRC, int UNITS>
Kernel prepared(const M40llmCudaContext* ctx) {
    // contexts on several threads may set it at the same time: setting it twice is harmless, losing another device's bit is not
    static std::atomic<unsigned long long> configured{0ull};
    const unsigned long long bit = 1ull << (ctx->device_id & 63);
    if (!(configured.load(std::memory_order_acquire) & bit)) {
        if (cudaFuncSetAttribute(gemm_tc_rows_kernel<SRC, UNITS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 SMEM_BYTES + sizeof(Control)) != cudaSuccess)
            return nullptr;
        configured.fetch_or(bit, std::memory_order_release);
    }
    return gemm_tc_rows_kernel<SRC, UNITS>;
}
template <int SRC>
Kernel pick(const M40llmCudaContext* ctx, uint32_t M) {
    return M <= 16 ? prepared<SRC, 1>(ctx) : prepared<SRC, 2>(ctx);
}

// Clusters of `ks` CTAs that fit the device at once, two CTAs per SM. Contexts on several threads may ask at the same time: each finds out
// for itself and all store the same.
uint32_t resident_clusters(const M40llmCudaContext* ctx, uint32_t ks) {
    static std::atomic<uint32_t> known[64][MAX_SPLITS + 1];  // clusters + 1, per device
    std::atomic<uint32_t>& slot = known[ctx->device_id & 63][ks];
    const uint32_t have = slot.load(std::memory_order_acquire);
    if (have) return have - 1u;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = ks;
    attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1, ks);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = SMEM_BYTES + sizeof(Control);
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaFuncSetAttribute(footprint_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES + sizeof(Control)) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&clusters, footprint_kernel, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    slot.store((uint32_t)clusters + 1u, std::memory_order_release);
    return (uint32_t)clusters;
}
uint32_t stage_size(uint32_t M) { return A_BYTES + 2u * ((M + 15) / 16 * 16) * BLOCK_K * 2; }
// Sums that a CTA is sent.
uint32_t sums_size(uint32_t M, uint32_t ks) { return ks > 1 ? ks * ((M + ks - 1) / ks) * BLOCK_N * 4 : 0u; }
// K splits: as many as leave all clusters resident at once, with at least four k-blocks each and, where the kernel splits x, MIN_STAGES of
// the ring beside the sums. (48 tiles: six splits would be 288 CTAs of 296, but only 45 clusters of six fit, and the last three took a
// second wave: 24 us instead of 15.)
uint32_t rows_splits(const M40llmCudaContext* ctx, const M40RowsArgs& a, uint32_t tiles, bool own_split) {
    for (uint32_t ks = min(min(2u * (uint32_t)ctx->sm_count / tiles, a.kblocks / 4u), MAX_SPLITS); ks > 1; --ks) {
        const uint32_t per = (a.kblocks + ks - 1) / ks, real = (a.kblocks + per - 1) / per;
        if (tiles <= resident_clusters(ctx, real) && (!own_split || sums_size(a.M, real) + MIN_STAGES * stage_size(a.M) <= SMEM_BYTES)) return real;
    }
    return 1;
}
}  // namespace

int m40_rows_launch(M40llmCudaContext* ctx, cudaStream_t s, int source, const CUtensorMap* w, const CUtensorMap& xh,
                    const CUtensorMap& xl, M40RowsArgs a) {
    a.kblocks = (a.K + BLOCK_K - 1) / BLOCK_K;
    a.status = ctx->d_status;
    uint32_t tiles = 0;
    const uint32_t n_rows = a.paired ? BLOCK_N / 2 : BLOCK_N;
    for (uint32_t p = 0; p < (a.paired ? 1u : a.problems); ++p) {
        a.tile_begin[p] = tiles;
        tiles += (a.N[p] + n_rows - 1) / n_rows;
    }
    if (a.paired) a.problems = 1;
    for (uint32_t p = a.problems; p < 4; ++p) a.tile_begin[p] = tiles;
    for (uint32_t p = 0; p < a.problems; ++p)
        if (a.N[p] % 4 == 0 && ((uintptr_t)a.out[p] & 15u) == 0) a.vec_out |= 1u << p;
    const uint32_t stage_bytes = stage_size(a.M), ks = rows_splits(ctx, a, tiles, source != M40_ROWS_SPLIT), sums = sums_size(a.M, ks);
    a.kb_per_split = (a.kblocks + ks - 1) / ks;
    const uint32_t fit = (SMEM_BYTES - sums) / stage_bytes;
    a.stages = fit < MAX_STAGES ? fit : MAX_STAGES;
    if (source != M40_ROWS_SPLIT && a.stages < MIN_STAGES) return -2;
    const Kernel k = source == M40_ROWS_SPLIT ? pick<M40_ROWS_SPLIT>(ctx, a.M)
                                              : (source == M40_ROWS_F16 ? pick<M40_ROWS_F16>(ctx, a.M) : pick<M40_ROWS_BF16>(ctx, a.M));
    if (!k) return -2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(tiles, ks);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = (size_t)a.stages * stage_bytes + sums + sizeof(Control);
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    uint32_t n = 0;
    if (m40_pdl_enabled()) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (ks > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = 1;
        attr[n].val.clusterDim.y = ks;
        attr[n++].val.clusterDim.z = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, k, w[0], w[1], w[2], xh, xl, a);
    M40_COUNT_LAUNCH(ctx);
    return e == cudaSuccess && cudaGetLastError() == cudaSuccess ? 0 : -2;
}
