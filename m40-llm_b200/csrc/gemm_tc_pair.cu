// Projections of many activation rows (prompts): persistent tcgen05 GEMM on CTA pairs (cta_group::2).
//
// With both parts (hi and lo) of the activations a call is 2 x M x N x K multiply-adds, so it is bound by the tensor cores once
// the tiles arrive fast enough. A 128 x 128 tile per CTA (gemm_tc.cu) asks L2 for 48 KB per 512 cycles of MMAs on every SM,
// more than L2 gives: it ran at half of the tensor rate. Here two SMs share a tile of 256 weight rows x up to 256 activation
// rows: each CTA holds 128 weight rows (operand A) and half of the activation rows (operand B, hi and lo), 48 KB per 1024 cycles.
//   D[256 x width] (f32, 128 lanes of tensor memory in each CTA)  +=  W[256 x 64] * (Xh + Xl)[64 x width]
// A ring of 48 KB stages (four at full width) is filled by one TMA thread per CTA; the even CTA issues all MMAs; two
// accumulators let the epilogue warps take a sum out while the next one is computed. In a gate | up call each CTA's 128 weight
// rows are 64 gate rows over 64 up rows, and the two warps that hold a gate row and its up row trade halves of their columns
// through shared memory. (Two accumulators of half the width in place of that need no trade, but an MMA of 128 columns takes as
// long as its weight operand does: 1600 cycles per 64-deep step against 1100.)
// Work units (weight tile x row tile x K split) are dealt round robin over the resident pairs; gemm_tc_pair_plan.cuh picks the
// width and the split.
//
// Precision: the tensor core cuts its f32 sums off where f32 multiply-adds round, so that the error grows with the number of
// additions to one accumulator (relative 8e-6 at K = 14336 with hi and lo added to the same one, 4e-6 with one each). Sums are
// therefore only SEG k-blocks long; the epilogue warps add them up in registers, rounding, while the MMAs fill the other
// accumulator.
//
// Every wait is bounded: a wait that runs out winds down both CTAs (give_up()): they stop issuing work, raise bit 2 of the
// device status word, wait for their copies in flight, free tensor memory and return. The barrier of two trading warps
// (finish_gated()) has no bound of its own, so both come to it equally often whatever their waits gave.
#include <atomic>
#include <type_traits>

#include "gemm_tc_pair.cuh"
#include "tc_ptx.cuh"

namespace {

using namespace tc;

constexpr uint32_t A_BYTES = BLOCK_N * BLOCK_K * 2;  // 16 KB
constexpr uint32_t RING_BYTES = 192u * 1024u;
constexpr uint32_t TRADE_BYTES = 32u * 1024u;  // gate | up: [2][4 warp pairs][2 directions][16][32] floats
constexpr uint32_t MAX_STAGES = 8;
constexpr uint32_t SEG = 4;  // k-blocks that are summed in tensor memory

struct PairArgs {
    uint32_t* status;
    uint32_t M, kblocks, stages;
    uint32_t units, k_splits, kb_per_split, m_tiles, width, tiles;
    uint32_t tile_begin[4];
    uint32_t problems, fmt_bits;
    float* partial;
    float* out;
    uint32_t n_out;
    const float* bias;
    const float* residual;
    const float* post_w;
    const float* post_b;
    int act;
    M40Tail tail;
};

struct Unit {
    uint32_t split, m_base, tile, problem, row0, kb0, n_kb;
};
template <bool PAIRED>
__device__ __forceinline__ Unit unit_of(const PairArgs& a, uint32_t u) {
    Unit r;
    r.split = u % a.k_splits;
    const uint32_t t = u / a.k_splits;
    r.m_base = (t % a.m_tiles) * a.width;  // row tiles of one weight tile are neighbours: its weights are read from L2
    r.tile = t / a.m_tiles;
    r.problem = 0;
    while (r.problem + 1 < a.problems && r.tile >= a.tile_begin[r.problem + 1]) ++r.problem;
    r.row0 = (r.tile - a.tile_begin[r.problem]) * (PAIRED ? M40_PAIR_ROWS / 2 : M40_PAIR_ROWS);
    r.kb0 = r.split * a.kb_per_split;
    r.n_kb = min(a.kb_per_split, a.kblocks - r.kb0);
    return r;
}

// Stores rows 0 .. live - 1 of a column. The full case has no guards, so that the elements' work interleaves.
template <uint32_t N, typename F>
__device__ __forceinline__ void store_column(const F& value, float* dst, uint32_t pitch, uint32_t live) {
    if (live >= N) {
#pragma unroll
        for (uint32_t i = 0; i < N; ++i, dst += pitch) *dst = value(i);
    } else {
#pragma unroll
        for (uint32_t i = 0; i < N; ++i, dst += pitch)
            if (i < live) *dst = value(i);
    }
}

// 16 activation rows of one output column: sum -> result. An epilogue warp has its scheduler nearly to itself, so a branch per
// element costs its full latency each time (50 000 cycles per tile, as long as the tile's MMAs): what a call asks for is
// decided once, outside of the loops.
__device__ __forceinline__ void finish_columns(const PairArgs& a, const float* v, uint32_t m, uint32_t n, uint32_t live) {
    const bool n_ok = n < a.n_out;
    const uint32_t n_ld = n_ok ? n : 0u;
    float* dst = a.out + (size_t)m * a.n_out + n_ld;
    float res[16];
    const float bias = a.bias ? a.bias[n_ld] : 0.0f;
    if (a.residual) {
        const float* r = a.residual + (size_t)m * a.n_out + n_ld;
#pragma unroll
        for (uint32_t i = 0; i < 16; ++i) {  // unconditional (the last row repeats): all under way together
            res[i] = *r;
            if (i + 1 < live) r += a.n_out;
        }
    } else {
        if (n_ok && a.tail.post == (int)M40LLM_NORM_NONE && !(a.tail.soft_cap > 0.0f)) {
            store_column<16>([&](uint32_t i) { return v[i] + bias; }, dst, a.n_out, live);
            return;
        }
#pragma unroll
        for (uint32_t i = 0; i < 16; ++i) res[i] = 0.0f;
    }
    if (!n_ok) return;
    if (a.tail.post == (int)M40LLM_NORM_NONE && !(a.tail.soft_cap > 0.0f)) {
        store_column<16>([&](uint32_t i) { return v[i] + bias + res[i]; }, dst, a.n_out, live);
        return;
    }
    const float pw = a.post_w ? a.post_w[n_ld] : 1.0f, pb = a.post_b ? a.post_b[n_ld] : 0.0f;
    if (a.tail.soft_cap > 0.0f) {
        store_column<16>([&](uint32_t i) { return m40_tail(a.tail, v[i], bias, pw, pb, res[i]); }, dst, a.n_out, live);
        return;
    }
    const M40Tail dyt = {(int)M40LLM_NORM_DYT, a.tail.post_alpha, 0.0f};
    store_column<16>([&](uint32_t i) { return m40_tail(dyt, v[i], bias, pw, pb, res[i]); }, dst, a.n_out, live);
}

// The same for gate | up and 32 activation rows: this warp holds gate rows (lane group 0, 1) or the up rows of the same outputs
// (2, 3) and finishes 16 of the activation rows with what the other warp hands over. `trade` is used by this pair of warps
// only; two halves of it take turns, so one barrier per call is enough.
__device__ __forceinline__ void finish_gated(const PairArgs& a, const float (&v)[32], uint32_t m, uint32_t n, uint32_t live,
                                             bool gate, uint32_t barrier, float* trade) {
    const uint32_t lane = threadIdx.x & 31u;
    float *give = trade + (gate ? 512u : 0u) + lane, *take = trade + (gate ? 0u : 512u) + lane;
    float mine[16], other[16];
#pragma unroll
    for (uint32_t i = 0; i < 16; ++i) {
        give[i * 32u] = gate ? v[16 + i] : v[i];
        mine[i] = gate ? v[i] : v[16 + i];
    }
    asm volatile("bar.sync %0, 64;" ::"r"(barrier) : "memory");
#pragma unroll
    for (uint32_t i = 0; i < 16; ++i) other[i] = take[i * 32u];
    const uint32_t skip = gate ? 0u : 16u;
    if (n >= a.n_out || live <= skip) return;
    float* dst = a.out + (size_t)(m + skip) * a.n_out + n;
    const auto gated = [&](auto act) {
        store_column<16>([&](uint32_t i) { return m40_act(decltype(act)::value, gate ? mine[i] : other[i]) * (gate ? other[i] : mine[i]); },
                         dst, a.n_out, live - skip);
    };
    if (a.act == (int)M40LLM_ACT_GELU_TANH) gated(std::integral_constant<int, (int)M40LLM_ACT_GELU_TANH>{});
    else if (a.act == (int)M40LLM_ACT_GELU_ERF) gated(std::integral_constant<int, (int)M40LLM_ACT_GELU_ERF>{});
    else gated(std::integral_constant<int, (int)M40LLM_ACT_SILU>{});
}

template <bool PAIRED>
__global__ void __launch_bounds__(384, 1) gemm_tc_pair_kernel(const __grid_constant__ CUtensorMap tmW0,
                                                              const __grid_constant__ CUtensorMap tmW1,
                                                              const __grid_constant__ CUtensorMap tmW2,
                                                              const __grid_constant__ CUtensorMap tmXh,
                                                              const __grid_constant__ CUtensorMap tmXl, PairArgs a) {
    extern __shared__ unsigned char smem_unaligned[];
    unsigned char* smem = smem_unaligned + ((1024u - (smem_u32(smem_unaligned) & 1023u)) & 1023u);
    __shared__ uint64_t full[MAX_STAGES], empty[MAX_STAGES], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_slot;
    __shared__ volatile uint32_t abort_flag;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t rank = cluster_rank(), pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const uint32_t part_bytes = (a.width / 2) * BLOCK_K * 2;  // half of the activation rows, hi or lo
    const uint32_t stage_bytes = A_BYTES + 2 * part_bytes;

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < a.stages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (uint32_t b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 16);  // eight epilogue warps of each CTA
        }
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tmem_alloc_pair(&tmem_slot, 512);
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();
    tc_fence_after();
    const uint32_t tmem_base = tmem_slot;
    pdl_trigger();
    const auto give_up = [&] {
        abort_flag = 1;
        st_cluster(map_to_rank(smem_u32(const_cast<uint32_t*>(&abort_flag)), rank ^ 1u), 1u);
    };
    uint32_t it = 0;  // stages that the loading thread has filled

    // Registers: launched with 3 x 168 per lane of the three warpgroups; the first keeps 40, the epilogue's two take 232 each.
    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
        if (warp == 0 && lane == 0) {
            // ---------------- TMA producer of this CTA. The weights of the first ring pass do not depend on the previous
            // kernel; everything else waits for it.
            uint32_t s = 0, round = 0;
            bool waited = false, ok = true;
            for (uint32_t u = pair; u < a.units && ok; u += pairs) {
                const Unit w = unit_of<PAIRED>(a, u);
                const CUtensorMap* tmW = w.problem == 0 ? &tmW0 : (w.problem == 1 ? &tmW1 : &tmW2);
                const int wrow = (int)(w.row0 + rank * (PAIRED ? BLOCK_N / 2 : BLOCK_N)), xrow = (int)(w.m_base + rank * (a.width / 2));
                uint32_t ahead = 0;  // stages of this unit whose weights were requested before the dependency wait
                if (!waited) {
                    ahead = min(w.n_kb, a.stages);
                    for (uint32_t i = 0; i < ahead; ++i) {
                        unsigned char* st = smem + i * stage_bytes;
                        const uint32_t bar = map_to_rank(smem_u32(&full[i]), 0);
                        if (rank == 0) mbar_expect_tx(&full[i], 2 * stage_bytes);
                        tma_load_2d_pair(st, tmW, bar, (int)((w.kb0 + i) * BLOCK_K), wrow);
                        if (PAIRED) tma_load_2d_pair(st + A_BYTES / 2, &tmW1, bar, (int)((w.kb0 + i) * BLOCK_K), wrow);
                    }
                    pdl_wait();
                    waited = true;
                }
                for (uint32_t i = 0; i < w.n_kb; ++i, ++it) {
                    if (round > 0 && (abort_flag || !mbar_wait(&empty[s], (round - 1) & 1u))) {
                        give_up();
                        ok = false;
                        break;
                    }
                    unsigned char* st = smem + s * stage_bytes;
                    const uint32_t bar = map_to_rank(smem_u32(&full[s]), 0);
                    const int kx = (int)((w.kb0 + i) * BLOCK_K);
                    if (i >= ahead) {
                        if (rank == 0) mbar_expect_tx(&full[s], 2 * stage_bytes);
                        tma_load_2d_pair(st, tmW, bar, kx, wrow);
                        if (PAIRED) tma_load_2d_pair(st + A_BYTES / 2, &tmW1, bar, kx, wrow);
                    }
                    tma_load_2d_pair(st + A_BYTES, &tmXh, bar, kx, xrow);
                    tma_load_2d_pair(st + A_BYTES + part_bytes, &tmXl, bar, kx, xrow);
                    if (++s == a.stages) s = 0, ++round;
                }
            }
        } else if (warp == 1 && rank == 0) {
            // ---------------- MMA issuer of the pair: the whole warp walks the loop, so that addresses and descriptors stay in
            // uniform registers; one lane issues
            const uint32_t idesc = make_idesc_pair(a.width) | a.fmt_bits;
            uint32_t s = 0, phase = 0, seg = 0;
            bool ok = true;
            for (uint32_t u = pair; u < a.units && ok; u += pairs) {
                const Unit w = unit_of<PAIRED>(a, u);
                for (uint32_t k0 = 0; k0 < w.n_kb && ok; k0 += SEG, ++seg) {
                    const uint32_t d = tmem_base + (seg & 1u) * 256u, k1 = min(k0 + SEG, w.n_kb);
                    if (seg >= 2) ok = __all_sync(0xffffffffu, mbar_wait_cluster(&acc_empty[seg & 1u], ((seg >> 1) & 1u) ^ 1u));
                    for (uint32_t i = k0; i < k1 && ok; ++i) {
                        ok = __all_sync(0xffffffffu, mbar_wait_cluster(&full[s], phase));
                        if (!ok) break;
                        tc_fence_after();
                        const uint32_t sa = smem_u32(smem + s * stage_bytes), sb = sa + A_BYTES;
                        if (elect_one()) {
#pragma unroll
                            for (uint32_t k = 0; k < BLOCK_K / UMMA_K; ++k) {
                                const uint32_t step = k * UMMA_K * 2;
                                const uint64_t da = make_desc_sw128(sa + step);
                                umma_f16_pair(d, da, make_desc_sw128(sb + step), idesc, (i - k0) | k);
                                umma_f16_pair(d, da, make_desc_sw128(sb + part_bytes + step), idesc, 1u);
                            }
                            umma_commit_pair(&empty[s]);
                            if (i + 1 == k1) umma_commit_pair(&acc_full[seg & 1u]);
                        }
                        __syncwarp();
                        if (++s == a.stages) s = 0, phase ^= 1u;
                    }
                }
            }
            if (!ok) give_up();
        }
        __syncwarp();
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 232;");
        // ---------------- epilogue: warp w owns lanes 32 * (w % 4) .. + 31 of this CTA's half of the tile and every second
        // run of 32 activation rows
        const uint32_t lane_group = warp & 3u;
        const uint32_t empty0 = map_to_rank(smem_u32(&acc_empty[0]), 0), empty1 = map_to_rank(smem_u32(&acc_empty[1]), 0);
        const uint32_t half = (warp - 4u) >> 2, warp_pair = half * 2u + (lane_group & 1u);
        float* trade = reinterpret_cast<float*>(smem + RING_BYTES);
        uint32_t seg = 0, traded = 0;
        bool ok = true;
        pdl_wait();
        for (uint32_t u = pair; u < a.units && (PAIRED || ok); u += pairs) {
            const Unit w = unit_of<PAIRED>(a, u);
            const uint32_t m_live = min(a.width, a.M - w.m_base);
            float acc[4][32];
#pragma unroll
            for (uint32_t e = 0; e < 128; ++e) acc[e / 32][e % 32] = 0.0f;
            for (uint32_t i = 0; i < w.n_kb && ok; i += SEG, ++seg) {
                const uint32_t b = seg & 1u;
                ok = __all_sync(0xffffffffu, mbar_wait(&acc_full[b], (seg >> 1) & 1u));
                if (!ok) {
                    give_up();
                    break;
                }
                tc_fence_after();
                const uint32_t taddr = tmem_base + b * 256u + ((lane_group * 32u) << 16) + half * 32u;
#pragma unroll
                for (uint32_t q = 0; q < 4; ++q) {
                    if (q * 64u + half * 32u >= m_live) continue;
                    uint32_t v[32];
                    tmem_ld_x32(taddr + q * 64u, v);
                    tmem_ld_wait();
#pragma unroll
                    for (uint32_t e = 0; e < 32; ++e) acc[q][e] += __uint_as_float(v[e]);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(b ? empty1 : empty0);
            }
            if (!PAIRED && !ok) break;
            const uint32_t in_tile = rank * BLOCK_N + lane_group * 32u + lane;
            const uint32_t n = PAIRED ? w.row0 + rank * (BLOCK_N / 2) + (lane_group & 1u) * 32u + lane : w.row0 + in_tile;
            const uint32_t pitch = a.tiles * M40_PAIR_ROWS;
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q) {
                const uint32_t c = q * 64u + half * 32u;
                if (c >= m_live) continue;
                const uint32_t live = ok ? min(32u, m_live - c) : 0u;
                if (PAIRED) {
                    finish_gated(a, acc[q], w.m_base + c, n, live, lane_group < 2u, 1u + warp_pair,
                                 trade + ((traded++ & 1u) * 4u + warp_pair) * 1024u);
                } else if (a.partial) {
                    store_column<32>([&](uint32_t i) { return acc[q][i]; },
                                     a.partial + ((size_t)w.split * a.M + w.m_base + c) * pitch + w.tile * M40_PAIR_ROWS + in_tile,
                                     pitch, live);
                } else {
                    finish_columns(a, acc[q], w.m_base + c, n, live);
                    if (live > 16u) finish_columns(a, acc[q] + 16, w.m_base + c + 16u, n, live - 16u);
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();  // neither CTA leaves while the other's MMAs or barriers still use its memory
    if (abort_flag) {    // the same in both CTAs by now
        if (threadIdx.x == 0 && rank == 0) {
            atomicOr(a.status, 4u);
            for (uint32_t s = 0; s < a.stages && s < it; ++s)  // copies of either CTA that are still under way land
                mbar_wait_cluster(&full[s], ((it - 1u - s) / a.stages) & 1u);
        }
        cluster_sync_all();
    }
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, 512);
    }
}

cudaLaunchConfig_t pair_config(cudaLaunchAttribute* attr, uint32_t ctas, bool paired, cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(384);
    cfg.dynamicSmemBytes = RING_BYTES + 1024u + (paired ? TRADE_BYTES : 0u);
    cfg.stream = s;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = m40_pdl_enabled() ? 2 : 1;
    return cfg;
}

// CTA pairs that fit the device at once, 0 where it takes none. Contexts on several threads may ask at the same time: each finds out
// for itself and all store the same. A query that fails is not remembered.
uint32_t resident_pairs(const M40llmCudaContext* ctx) {
    static std::atomic<uint32_t> known[64];  // pairs + 1, per device
    std::atomic<uint32_t>& slot = known[ctx->device_id & 63];
    const uint32_t have = slot.load(std::memory_order_acquire);
    if (have) return have - 1u;
    int clusters = 0;
    cudaLaunchAttribute attr[2];
    cudaLaunchConfig_t cfg = pair_config(attr, 2, true, nullptr);
    cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(gemm_tc_pair_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, RING_BYTES + 1024) != cudaSuccess ||
        cudaFuncSetAttribute(gemm_tc_pair_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, RING_BYTES + 1024 + TRADE_BYTES) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&clusters, gemm_tc_pair_kernel<true>, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    slot.store((uint32_t)clusters + 1u, std::memory_order_release);
    return (uint32_t)clusters;
}

}  // namespace

bool m40_pair_available(const M40llmCudaContext* ctx) { return resident_pairs(ctx) > 0; }

bool m40_pair_plan(const M40llmCudaContext* ctx, uint32_t M, uint32_t kblocks, uint32_t problems, const int* N, bool gate_up,
                   bool partial_only, M40PairPlan* plan) {
    return m40_pair_cut_best(resident_pairs(ctx), M, kblocks, problems, N, gate_up, partial_only, plan);
}

int m40_pair_launch(M40llmCudaContext* ctx, cudaStream_t s, const M40PairCall& c, const M40PairPlan& p) {
    const uint32_t pairs = resident_pairs(ctx);
    if (pairs == 0) return -2;
    PairArgs a = {};
    a.status = ctx->d_status;
    a.M = c.M;
    a.kblocks = c.kblocks;
    const uint32_t stage_bytes = A_BYTES + p.width * BLOCK_K * 2;
    a.stages = RING_BYTES / stage_bytes < MAX_STAGES ? RING_BYTES / stage_bytes : MAX_STAGES;
    a.units = p.tiles * p.m_tiles * p.k_splits;
    a.k_splits = p.k_splits;
    a.kb_per_split = p.kb_per_split;
    a.m_tiles = p.m_tiles;
    a.width = p.width;
    a.tiles = p.tiles;
    for (int i = 0; i < 4; ++i) a.tile_begin[i] = p.tile_begin[i];
    a.problems = p.paired ? 1u : c.problems;
    a.fmt_bits = c.fmt_bits;
    a.partial = c.partial;
    a.out = c.out;
    a.n_out = c.n_out;
    a.bias = c.bias;
    a.residual = c.residual;
    a.post_w = c.post_w;
    a.post_b = c.post_b;
    a.act = c.act;
    a.tail = c.tail;
    cudaLaunchAttribute attr[2];
    const cudaLaunchConfig_t cfg = pair_config(attr, 2u * (a.units < pairs ? a.units : pairs), p.paired, s);
    const cudaError_t e = cudaLaunchKernelEx(&cfg, p.paired ? gemm_tc_pair_kernel<true> : gemm_tc_pair_kernel<false>, c.w[0], c.w[1],
                                             c.w[2], c.xh, c.xl, a);
    M40_COUNT_LAUNCH(ctx);
    return e == cudaSuccess && cudaGetLastError() == cudaSuccess ? 0 : -2;
}
