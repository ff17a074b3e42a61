// Generalised delta rule: a recurrent mixer whose state is one matrix per head,
//   S <- diag(w) S - (a * u) (u^T S) + k v^T,   o = S^T r,
// with a decay w and a removal rate a per head and key channel, u the unit key. All of it is f32.
//
// With k = n u (n the key's length) the update of one value column s of S is
//   d = u . s,   s_i <- w_i s_i + u_i (n v - a_i d),   o = r . s,
// so columns are independent. A column's key dimension is shared by a few lanes (16-byte pieces dealt round-robin) and stays in
// registers; the only serial chain is d: a dot product over the lanes, then two multiply-adds per element. (With one, on
// w_i s_i + u_i n v from before, a state whose keys come back loses twice as much: n v - a d must cancel before it is rounded to the
// size of either.)
//
//   portions of several tokens, in passes of rows whose records stay in L2:
//     delta_prepare_kernel  warp = (row, head): gates, decays, unit key -> one record [w | u | a | r | n v | c] per (head, row);
//     delta_scan_kernel     CTA = (16 to 64 columns, head, segment) walks the tokens in pairs; the records of 16 tokens arrive by
//                           one bulk copy (cp.async.bulk + mbarrier) several chunks ahead. Reads of the records from shared memory
//                           are the limit, so a lane holds few keys of several columns and every piece serves all of them;
//     delta_finish_kernel   the per-head norm and the output gate.
//   delta_decode_kernel     one token per sequence: CTA = (head, row) does everything, the low-rank decay projection
//                           included, in one launch; bound by reading and writing the state once.
//
// Two tokens share one trip over the lanes. With s1 the column after the first of a pair,
//   d1 = u1 . s1 = (w0 u1) . s0 + c1 n0 v0 - c2 d0,   c1 = u1 . u0,   c2 = u1 . (a0 u0),
// so both dot products start from s0, and c1 and c2 are the same for all columns and come with the record. The terms are those of
// u1 . s1 added up in another order, in f32 like everything here. A longer chunked (matrix-product) form is not used: its products of
// decays would have to leave f32.
//
// The scan's waits are bounded like the tensor-core kernels': a wait that runs out raises status bit 4, the CTA stops,
// waits (bounded) for its copies in flight and returns.
#include <atomic>

#include "common.cuh"
#include "delta_scan_plan.cuh"
#include "stack_math.cuh"
#include "state_cache.cuh"
#include "tc_ptx.cuh"

namespace {

constexpr int LANES = 4;          // decode: lanes per column
constexpr int SCAN_THREADS = M40_SCAN_THREADS;
constexpr size_t PASS_BYTES = (size_t)96 << 20;  // records of one pass: inside L2
constexpr int SCAN_CHUNK = 16;    // tokens per bulk copy (even: pairs do not cross chunks)
constexpr uint32_t SCAN_MAX_STAGES = 8;
constexpr int SCAN_SMEM = 196608;
// A record: w | u | a | r | n v, DP floats each, then c1, c2 and two floats of padding.
__host__ __device__ constexpr uint32_t rec_floats(int dp) { return 5u * dp + 4u; }
__host__ __device__ constexpr size_t scan_stage_bytes(int dp) { return (size_t)SCAN_CHUNK * rec_floats(dp) * sizeof(float); }

struct DeltaArgs {
    const float* packed;
    const void* w2;
    const float* w0;
    const float* a_bias;
    const float* norm;
    const float* decay_in;
    float* out;
    float* state;
    uint32_t* status;
    const uint32_t* row_seq;
    const uint32_t* row_pos;
    const uint32_t* seg;
    uint32_t ld, rank, w2_dtype, w2_wide, heads, dim, slots, slot_mul, slot_add, rows;
    float decay_scale, unit_eps, eps;
};

__device__ __forceinline__ float w2_elem(const DeltaArgs& a, size_t i) {
    if (a.w2_dtype == M40LLM_DT_BF16) return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(a.w2)[i]);
    if (a.w2_dtype == M40LLM_DT_F16) return __half2float(reinterpret_cast<const __half*>(a.w2)[i]);
    return reinterpret_cast<const float*>(a.w2)[i];
}
__device__ __forceinline__ float decay_of(const DeltaArgs& a, float z) { return expf(a.decay_scale * m40_sigmoid(z)); }

// State of one column: elements 4 (l4 + LANES i) .. + 3 of the key dimension.
template <int NI, int LANES>
__device__ __forceinline__ void load_column(const float* col, uint32_t dim, uint32_t l4, bool zero, float4 (&s)[NI]) {
#pragma unroll
    for (int i = 0; i < NI; ++i) {
        const uint32_t k = 4u * (l4 + LANES * i);
        s[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (zero || k >= dim) continue;
        if (dim % 4u == 0u) {
            s[i] = *reinterpret_cast<const float4*>(col + k);
        } else {
            s[i].x = col[k];
            if (k + 1 < dim) s[i].y = col[k + 1];
            if (k + 2 < dim) s[i].z = col[k + 2];
            if (k + 3 < dim) s[i].w = col[k + 3];
        }
    }
}
template <int NI, int LANES>
__device__ __forceinline__ void store_column(float* col, uint32_t dim, uint32_t l4, const float4 (&s)[NI]) {
#pragma unroll
    for (int i = 0; i < NI; ++i) {
        const uint32_t k = 4u * (l4 + LANES * i);
        if (k >= dim) continue;
        if (dim % 4u == 0u) {
            *reinterpret_cast<float4*>(col + k) = s[i];
        } else {
            col[k] = s[i].x;
            if (k + 1 < dim) col[k + 1] = s[i].y;
            if (k + 2 < dim) col[k + 2] = s[i].z;
            if (k + 3 < dim) col[k + 3] = s[i].w;
        }
    }
}

// One token on one column: vec = [w | u | a | r], each DP floats (zero beyond dim); nv = n * v of this column. Returns o,
// the same in all LANES lanes.
template <int NI>
__device__ __forceinline__ float delta_token(const float* vec, uint32_t l4, float nv, float4 (&s)[NI]) {
    constexpr int DP = NI * LANES * 4;
    const float4* w = reinterpret_cast<const float4*>(vec) + l4;
    const float4* u = reinterpret_cast<const float4*>(vec + DP) + l4;
    const float4* a = reinterpret_cast<const float4*>(vec + 2 * DP) + l4;
    const float4* r = reinterpret_cast<const float4*>(vec + 3 * DP) + l4;
    float4 uu[NI];
    float d0 = 0.f, d1 = 0.f, d2 = 0.f, d3 = 0.f;
#pragma unroll
    for (int i = 0; i < NI; ++i) {
        uu[i] = u[LANES * i];
        d0 = fmaf(uu[i].x, s[i].x, d0), d1 = fmaf(uu[i].y, s[i].y, d1);
        d2 = fmaf(uu[i].z, s[i].z, d2), d3 = fmaf(uu[i].w, s[i].w, d3);
    }
    float d = (d0 + d1) + (d2 + d3);
    d += __shfl_xor_sync(0xffffffffu, d, 1);
    d += __shfl_xor_sync(0xffffffffu, d, 2);
    float o0 = 0.f, o1 = 0.f, o2 = 0.f, o3 = 0.f;
#pragma unroll
    for (int i = 0; i < NI; ++i) {
        const float4 wi = w[LANES * i], ai = a[LANES * i], ri = r[LANES * i];
        s[i].x = fmaf(uu[i].x, fmaf(-ai.x, d, nv), wi.x * s[i].x);
        s[i].y = fmaf(uu[i].y, fmaf(-ai.y, d, nv), wi.y * s[i].y);
        s[i].z = fmaf(uu[i].z, fmaf(-ai.z, d, nv), wi.z * s[i].z);
        s[i].w = fmaf(uu[i].w, fmaf(-ai.w, d, nv), wi.w * s[i].w);
        o0 = fmaf(ri.x, s[i].x, o0), o1 = fmaf(ri.y, s[i].y, o1);
        o2 = fmaf(ri.z, s[i].z, o2), o3 = fmaf(ri.w, s[i].w, o3);
    }
    float o = (o0 + o1) + (o2 + o3);
    o += __shfl_xor_sync(0xffffffffu, o, 1);
    o += __shfl_xor_sync(0xffffffffu, o, 2);
    return o;
}

// Rows [base, base + count) of every segment (relative to its start) -> records. One warp per (row, head); `rec` holds, per
// head, n_rec records, the record of row r of the step at r - base. c1 and c2 look back at the row before, whatever sequence it
// belongs to: the scan uses them within a segment only.
template <int DP>
__global__ void __launch_bounds__(256) delta_prepare_kernel(DeltaArgs a, float* __restrict__ rec, uint32_t n_rec, uint32_t base,
                                                            uint32_t count) {
    constexpr int CPL = DP / 32;  // channels per lane
    pdl_wait();
    pdl_trigger();
    const uint32_t wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31u;
    if (wid >= count * a.heads) return;
    const uint32_t head = wid % a.heads, row = base + wid / a.heads, D = a.dim, HD = a.heads * D;
    const float* p = a.packed + (size_t)row * a.ld + head * D;
    const float* before = p - (row > 0u ? a.ld : 0u);
    float r[CPL], k[CPL], v[CPL], rate[CPL], z[CPL], k0[CPL], rate0[CPL], ss = 0.0f, ss0 = 0.0f;
#pragma unroll
    for (int i = 0; i < CPL; ++i) {
        const uint32_t ch = lane + 32u * i, cc = ch < D ? ch : D - 1u;  // clamped: every load is unconditional
        r[i] = p[cc];
        k[i] = p[HD + cc];
        v[i] = p[2 * (size_t)HD + cc];
        rate[i] = p[4 * (size_t)HD + cc] + a.a_bias[head * D + cc];
        z[i] = (a.decay_in ? a.decay_in[(size_t)row * HD + head * D + cc] : 0.0f) + a.w0[head * D + cc];
        k0[i] = before[HD + cc];
        rate0[i] = before[4 * (size_t)HD + cc] + a.a_bias[head * D + cc];
    }
    if (!a.decay_in) {
        const float* zp = a.packed + (size_t)row * a.ld + 5 * (size_t)HD;
#pragma unroll
        for (int i = 0; i < CPL; ++i) {
            const uint32_t ch = lane + 32u * i, cc = ch < D ? ch : D - 1u;
            float acc = 0.0f;
            for (uint32_t q = 0; q < a.rank; ++q) acc = fmaf(w2_elem(a, (size_t)(head * D + cc) * a.rank + q), tanhf(zp[q]), acc);
            z[i] += acc;
        }
    }
#pragma unroll
    for (int i = 0; i < CPL; ++i) {
        ss = lane + 32u * i < D ? fmaf(k[i], k[i], ss) : ss;
        ss0 = lane + 32u * i < D ? fmaf(k0[i], k0[i], ss0) : ss0;
    }
    const float len = sqrtf(warp_sum(ss) + a.unit_eps), inv = 1.0f / len;
    const float inv0 = 1.0f / sqrtf(warp_sum(ss0) + a.unit_eps);
    float* dst = rec + ((size_t)head * n_rec + (row - base)) * rec_floats(DP);
    float c1 = 0.0f, c2 = 0.0f;
#pragma unroll
    for (int i = 0; i < CPL; ++i) {
        const uint32_t ch = lane + 32u * i;
        const bool in = ch < D;
        const float u = k[i] * inv, u0 = k0[i] * inv0;
        dst[ch] = in ? decay_of(a, z[i]) : 0.0f;
        dst[DP + ch] = in ? u : 0.0f;
        dst[2 * DP + ch] = in ? m40_sigmoid(rate[i]) : 0.0f;
        dst[3 * DP + ch] = in ? r[i] : 0.0f;
        dst[4 * DP + ch] = in ? len * v[i] : 0.0f;
        c1 = in ? fmaf(u, u0, c1) : c1;
        c2 = in ? fmaf(u, u0 * m40_sigmoid(rate0[i]), c2) : c2;
    }
    c1 = warp_sum(c1), c2 = warp_sum(c2);
    if (lane == 0) *reinterpret_cast<float4*>(dst + 5 * DP) = make_float4(c1, c2, 0.0f, 0.0f);
}

// Two f32 in one register pair: one instruction works on both (rounded like the scalar ones).
struct F2 {
    unsigned long long v;
};
__device__ __forceinline__ F2 f2(float lo, float hi) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float f2_sum(F2 a) {
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a.v));
    return lo + hi;
}
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b) {
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
// This lane's pieces of one vector of a record.
template <int NI, int LANES>
__device__ __forceinline__ void load_pieces(const float* vec, uint32_t l, F2 (&x)[2 * NI]) {
#pragma unroll
    for (int i = 0; i < NI; ++i) {
        const ulonglong2 t = *(reinterpret_cast<const ulonglong2*>(vec) + l + LANES * i);
        x[2 * i].v = t.x, x[2 * i + 1].v = t.y;
    }
}
// One trip over LANES lanes: every lane gets the sums of d and e, and of the V values o by halving the one of index held_sum<V>(l),
// in o[0]. The shuffles of a level are independent of each other and stand next to each other: the compiler keeps their order, and
// one value after the other would pay for each shuffle's latency (16 instead of 4: 300 instead of 241 us for 2048 tokens of 32 x 64).
template <int COLS, int V, int LANES, int BIT = 1>
__device__ __forceinline__ void sums_over_lanes(float (&d)[COLS], float (&e)[COLS], float (&o)[V], uint32_t l) {
    constexpr uint32_t FULL = 0xffffffffu;
    if constexpr (BIT < LANES) {
        constexpr int H = V > 1 ? V / 2 : 1;
        const bool upper = l & BIT;
        float td[COLS], te[COLS], to[H], half[H];
#pragma unroll
        for (int c = 0; c < COLS; ++c) td[c] = __shfl_xor_sync(FULL, d[c], BIT), te[c] = __shfl_xor_sync(FULL, e[c], BIT);
#pragma unroll
        for (int i = 0; i < H; ++i) to[i] = __shfl_xor_sync(FULL, V > 1 && !upper ? o[V > 1 ? H + i : 0] : o[i], BIT);
#pragma unroll
        for (int c = 0; c < COLS; ++c) d[c] += td[c], e[c] += te[c];
#pragma unroll
        for (int i = 0; i < H; ++i) half[i] = (V > 1 && upper ? o[V > 1 ? H + i : 0] : o[i]) + to[i];
        sums_over_lanes<COLS, H, LANES, BIT * 2>(d, e, half, l);
        o[0] = half[0];
    }
}
template <int V>
__device__ __forceinline__ uint32_t held_sum(uint32_t l) {
    uint32_t at = 0;
#pragma unroll
    for (int half = V / 2, bit = 0; half > 0; half /= 2, ++bit) at += (l >> bit & 1u) * half;
    return at;
}

// COLS adjacent values.
template <int COLS>
__device__ __forceinline__ void load_values(const float* p, float (&v)[COLS]) {
    static_assert(COLS == 2 || COLS == 4, "vector loads");
    if constexpr (COLS == 2)
        *reinterpret_cast<float2*>(v) = *reinterpret_cast<const float2*>(p);
    else
        *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(p);
}

// grid (column blocks, heads, segments). Rows [base, base + count) of the segment, counted from its start. LANES lanes hold COLS
// columns of LANES * NI * 4 keys; which of them a call takes: delta_scan_plan.cuh. A pair's chain of shuffles and multiply-adds takes most
// of the time. The whole call for 2048 tokens of one sequence, 32 heads of 64: 301 us (368 a token at a time, 32 columns per CTA); 1504
// tokens of 16 sequences, 64 heads: 187 us (300).
template <int NI, int LANES, int COLS>
__global__ void __launch_bounds__(SCAN_THREADS) delta_scan_kernel(DeltaArgs a, const float* __restrict__ rec, uint32_t n_rec,
                                                                  uint32_t rec_base, uint32_t base, uint32_t count, uint32_t stages) {
    constexpr int DP = NI * LANES * 4;
    constexpr uint32_t REC = rec_floats(DP), CHUNK = SCAN_CHUNK;
    extern __shared__ __align__(128) float ring[];
    __shared__ uint64_t full[SCAN_MAX_STAGES];
    __shared__ uint32_t stop;
    const uint32_t tid = threadIdx.x;
    if (tid == 0) {
        for (uint32_t s = 0; s < stages; ++s) tc::mbar_init(&full[s], 1);
        stop = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    pdl_wait();
    pdl_trigger();
    const uint32_t head = blockIdx.y, col0 = blockIdx.x * (SCAN_THREADS / LANES * COLS), D = a.dim, HD = a.heads * D;
    // last segments first: a step has its single tokens before its prompts, whose chains take longest
    const uint32_t z = gridDim.z - 1u - blockIdx.z;
    const uint32_t seg0 = a.seg[4 * z], seg_n = a.seg[4 * z + 1];
    const uint32_t slot = a.seg[4 * z + 2] * a.slot_mul + a.slot_add, pos0 = a.seg[4 * z + 3];
    if (slot >= a.slots || (uint64_t)seg0 + seg_n > a.rows) {
        if (tid == 0 && blockIdx.x == 0 && head == 0) atomicOr(a.status, 2u);
        return;
    }
    if (base >= seg_n) return;
    const uint32_t n = seg_n - base < count ? seg_n - base : count, row0 = seg0 + base;
    const float* src = rec + ((size_t)head * n_rec + (row0 - rec_base)) * REC;
    const uint32_t chunks = (n + CHUNK - 1) / CHUNK;
    auto request = [&](uint32_t ch, uint32_t s) {  // thread 0
        const uint32_t m = n - ch * CHUNK < CHUNK ? n - ch * CHUNK : CHUNK, bytes = m * REC * 4u;
        tc::mbar_expect_tx(&full[s], bytes);
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                     ::"r"(tc::smem_u32(ring + (size_t)s * CHUNK * REC)), "l"(src + (size_t)ch * CHUNK * REC), "r"(bytes),
                     "r"(tc::smem_u32(&full[s])) : "memory");
    };
    if (tid == 0)
        for (uint32_t ch = 0; ch < chunks && ch < stages; ++ch) request(ch, ch);

    const uint32_t l = tid % LANES, first = col0 + tid / LANES * COLS;
    const uint32_t nv_at = 4 * DP + (first < DP ? first : 0u);  // a block may reach beyond the padded columns
    float* state = a.state + ((size_t)slot * a.heads + head) * D * D;
    F2 s[COLS][2 * NI];
    const bool fresh = pos0 == 0 && base == 0;
#pragma unroll
    for (int c = 0; c < COLS; ++c) {
        float4 t[NI];
        const uint32_t col = first + c;
        load_column<NI, LANES>(state + (size_t)(col < D ? col : 0u) * D, D, l, fresh || col >= D, t);
#pragma unroll
        for (int i = 0; i < NI; ++i) s[c][2 * i] = f2(t[i].x, t[i].y), s[c][2 * i + 1] = f2(t[i].z, t[i].w);
    }
    // lanes 0 .. 2 COLS - 1 store: outputs o[column][token] of a pair
    constexpr uint32_t V = 2 * COLS;
    const uint32_t token = held_sum<V>(l) % 2u, mine = first + held_sum<V>(l) / 2u;
    float* out = a.out + (size_t)(row0 + token) * HD + head * D + (mine < D ? mine : 0u);
    const bool store = l < V && mine < D;

    const F2 zero = f2(0.0f, 0.0f);
    float o[V] = {};  // the outputs of the pair before, still spread over the lanes: summed together with this pair's products
    bool held = false;
    uint32_t ch = 0, slot_at = 0, phase = 0;
    for (; ch < chunks; ++ch) {
        if (!tc::mbar_wait(&full[slot_at], phase)) stop = 1u;
        const float* buf = ring + (size_t)slot_at * CHUNK * REC;
        const uint32_t m = n - ch * CHUNK < CHUNK ? n - ch * CHUNK : CHUNK;
        F2 u0[2 * NI], q1[2 * NI], w0[2 * NI];  // of the pair at hand: u0, w0 and w0 u1
        load_pieces<NI, LANES>(buf, l, w0);
        load_pieces<NI, LANES>(buf + DP, l, u0);
        load_pieces<NI, LANES>(buf + (m > 1u ? REC : 0u) + DP, l, q1);
#pragma unroll
        for (int i = 0; i < 2 * NI; ++i) q1[i] = f2_mul(q1[i], w0[i]);
        for (uint32_t t = 0; t < m; t += 2u) {
            const float* va = buf + (size_t)t * REC;
            const bool two = t + 1u < m;
            const float* vb = va + (two ? REC : 0u);
            float d[COLS], e[COLS];
#pragma unroll
            for (int c = 0; c < COLS; ++c) {
                F2 x = f2_mul(u0[0], s[c][0]), y = f2_mul(q1[0], s[c][0]);
#pragma unroll
                for (int i = 1; i < 2 * NI; ++i) x = f2_fma(u0[i], s[c][i], x), y = f2_fma(q1[i], s[c][i], y);
                d[c] = f2_sum(x), e[c] = f2_sum(y);
            }
            // the rest of this pair's records and the start of the next pair's are on their way during the shuffles
            F2 a0[2 * NI], r[2 * NI], u1[2 * NI], w1[2 * NI], a1[2 * NI], r1[2 * NI];
            load_pieces<NI, LANES>(va + 2 * DP, l, a0);
            load_pieces<NI, LANES>(va + 3 * DP, l, r);
            load_pieces<NI, LANES>(vb, l, w1);
            load_pieces<NI, LANES>(vb + DP, l, u1);
            load_pieces<NI, LANES>(vb + 2 * DP, l, a1);
            load_pieces<NI, LANES>(vb + 3 * DP, l, r1);
            const float2 cc = *reinterpret_cast<const float2*>(vb + 5 * DP);
            float nv0[COLS], nv1[COLS];
            load_values<COLS>(va + nv_at, nv0);
            load_values<COLS>(vb + nv_at, nv1);
            sums_over_lanes<COLS, V, LANES>(d, e, o, l);
            if (held) {
                if (store) out[0] = o[0];
                out += 2 * (size_t)HD;
            }
            held = two;
#pragma unroll
            for (int c = 0; c < COLS; ++c) {
                const F2 n0 = f2(nv0[c], nv0[c]), d0 = f2(-d[c], -d[c]);
                F2 x = zero;
#pragma unroll
                for (int i = 0; i < 2 * NI; ++i) {
                    s[c][i] = f2_fma(u0[i], f2_fma(a0[i], d0, n0), f2_mul(w0[i], s[c][i]));
                    x = f2_fma(r[i], s[c][i], x);
                }
                o[2 * c] = f2_sum(x);
            }
            if (!two) break;  // the last token of the segment
#pragma unroll
            for (int c = 0; c < COLS; ++c) {
                const float d1 = fmaf(-cc.y, d[c], fmaf(cc.x, nv0[c], e[c]));
                const F2 n1 = f2(nv1[c], nv1[c]), dd = f2(-d1, -d1);
                F2 x = zero;
#pragma unroll
                for (int i = 0; i < 2 * NI; ++i) {
                    s[c][i] = f2_fma(u1[i], f2_fma(a1[i], dd, n1), f2_mul(w1[i], s[c][i]));
                    x = f2_fma(r1[i], s[c][i], x);
                }
                o[2 * c + 1] = f2_sum(x);
            }
            const float* vn = va + (t + 2u < m ? 2u * REC : 0u);
            load_pieces<NI, LANES>(vn, l, w0);
            load_pieces<NI, LANES>(vn + DP, l, u0);
            load_pieces<NI, LANES>(vn + (t + 3u < m ? REC : 0u) + DP, l, q1);
#pragma unroll
            for (int i = 0; i < 2 * NI; ++i) q1[i] = f2_mul(q1[i], w0[i]);
        }
        __syncthreads();  // everyone is done with this slot
        if (stop) break;
        if (tid == 0 && ch + stages < chunks) request(ch + stages, slot_at);
        if (++slot_at == stages) slot_at = 0, phase ^= 1u;
    }
    if (ch < chunks) {  // a wait ran out: the copies still in flight must land before this CTA's memory goes away
        if (tid == 0) {
            atomicOr(a.status, 4u);
            for (uint32_t i = ch; i < chunks && i < ch + stages; ++i) tc::mbar_wait(&full[i % stages], (i / stages) & 1u);
        }
        return;
    }
    if (!held) {  // an odd number of tokens: the last one has no partner
#pragma unroll
        for (int c = 0; c < COLS; ++c) o[2 * c + 1] = 0.0f;
    }
    float none[COLS] = {};
    sums_over_lanes<COLS, V, LANES>(none, none, o, l);
    if (store && (held || token == 0u)) out[0] = o[0];
#pragma unroll
    for (int c = 0; c < COLS; ++c) {
        float4 t[NI];
#pragma unroll
        for (int i = 0; i < NI; ++i) {
            asm("mov.b64 {%0, %1}, %2;" : "=f"(t[i].x), "=f"(t[i].y) : "l"(s[c][2 * i].v));
            asm("mov.b64 {%0, %1}, %2;" : "=f"(t[i].z), "=f"(t[i].w) : "l"(s[c][2 * i + 1].v));
        }
        if (first + c < D) store_column<NI, LANES>(state + (size_t)(first + c) * D, D, l, t);
    }
}

// out <- (out / rms per head) * norm * sigmoid(g). One warp per (row, head).
__global__ void __launch_bounds__(256) delta_finish_kernel(DeltaArgs a) {
    pdl_wait();
    pdl_trigger();
    const uint32_t wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31u;
    if (wid >= a.rows * a.heads) return;
    const uint32_t row = wid / a.heads, head = wid % a.heads, D = a.dim, HD = a.heads * D;
    float* o = a.out + (size_t)row * HD + head * D;
    const float* g = a.packed + (size_t)row * a.ld + 3 * (size_t)HD + head * D;
    float v[8], ss = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint32_t ch = lane + 32u * i;
        v[i] = ch < D ? o[ch] : 0.0f;
        ss = fmaf(v[i], v[i], ss);
    }
    const float inv = 1.0f / sqrtf(warp_sum(ss) / (float)D + a.eps);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint32_t ch = lane + 32u * i;
        if (ch < D) o[ch] = v[i] * inv * a.norm[head * D + ch] * m40_sigmoid(g[ch]);
    }
}

// grid (heads, rows), block = dim * LANES rounded up to a warp.
template <int NI>
__global__ void __launch_bounds__(NI * LANES * 4 * LANES, NI <= 4 ? 16 / NI : 1) delta_decode_kernel(DeltaArgs a) {
    constexpr int DP = NI * LANES * 4;
    __shared__ __align__(16) float vec[4 * DP];
    __shared__ __align__(16) float sz[1024];
    __shared__ float sv[DP], so[DP];
    const uint32_t head = blockIdx.x, row = blockIdx.y, D = a.dim, HD = a.heads * D, tid = threadIdx.x;
    const uint32_t lane = tid & 31u, col = tid / LANES, l4 = tid % LANES;
    const uint32_t cc = head * D + (col < D ? col : D - 1u);  // this thread's channel (clamped)
    // The low-rank rows of this channel do not depend on the previous kernel: 16-byte pieces l4, l4 + 4, ... of a 16-bit
    // row, up to four per lane, are requested before the dependency wait.
    const bool wide = a.w2_wide != 0u;
    uint4 wq[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint32_t q8 = l4 + LANES * j;
        wq[j] = make_uint4(0u, 0u, 0u, 0u);
        if (wide && q8 < a.rank / 8u)
            wq[j] = *reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(a.w2) + (size_t)cc * a.rank + 8u * q8);
    }
    const float w0 = a.w0[cc], ab = a.a_bias[cc];
    pdl_wait();
    pdl_trigger();
    const uint32_t slot = a.row_seq[row] * a.slot_mul + a.slot_add;
    if (slot >= a.slots) {
        if (tid == 0 && head == 0) atomicOr(a.status, 2u);
        for (uint32_t ch = tid; ch < D; ch += blockDim.x) a.out[(size_t)row * HD + head * D + ch] = 0.0f;
        return;
    }
    float* colp = a.state + (((size_t)slot * a.heads + head) * D + (col < D ? col : 0u)) * D;
    float4 s[NI];
    load_column<NI, LANES>(colp, D, l4, a.row_pos[row] == 0 || col >= D, s);
    const float* prow = a.packed + (size_t)row * a.ld;
    const float* p = prow + head * D;
    const float pr = prow[cc], pk = prow[HD + cc], pv = prow[2 * (size_t)HD + cc], pa = prow[4 * (size_t)HD + cc];
    float z = a.decay_in ? a.decay_in[(size_t)row * HD + cc] : 0.0f;
    float ss = 0.0f;
    for (uint32_t ch = lane; ch < D; ch += 32u) ss = fmaf(p[HD + ch], p[HD + ch], ss);
    if (!a.decay_in) {
        const float* zp = prow + 5 * (size_t)HD;
        for (uint32_t q = tid; q < a.rank; q += blockDim.x) sz[q] = tanhf(zp[q]);
    }
    const float len = sqrtf(warp_sum(ss) + a.unit_eps), inv = 1.0f / len;  // every warp, redundantly
    if (!a.decay_in) {
        __syncthreads();
        // the low-rank product: LANES lanes per channel
        if (wide) {
            const bool bf = a.w2_dtype == M40LLM_DT_BF16;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t q8 = l4 + LANES * j;
                if (q8 >= a.rank / 8u) break;
                const uint32_t u[4] = {wq[j].x, wq[j].y, wq[j].z, wq[j].w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float2 h = __half22float2(*reinterpret_cast<const __half2*>(&u[i]));
                    z = fmaf(bf ? __uint_as_float(u[i] << 16) : h.x, sz[8u * q8 + 2 * i], z);
                    z = fmaf(bf ? __uint_as_float(u[i] & 0xffff0000u) : h.y, sz[8u * q8 + 2 * i + 1], z);
                }
            }
        } else {
            for (uint32_t q = l4; q < a.rank; q += LANES) z = fmaf(w2_elem(a, (size_t)cc * a.rank + q), sz[q], z);
        }
        z += __shfl_xor_sync(0xffffffffu, z, 1);
        z += __shfl_xor_sync(0xffffffffu, z, 2);
    }
    if (l4 == 0 && col < DP) {
        const bool in = col < D;
        vec[col] = in ? decay_of(a, z + w0) : 0.0f;
        vec[DP + col] = in ? pk * inv : 0.0f;
        vec[2 * DP + col] = in ? m40_sigmoid(pa + ab) : 0.0f;
        vec[3 * DP + col] = in ? pr : 0.0f;
        sv[col] = in ? len * pv : 0.0f;
    }
    const float gate = m40_sigmoid(prow[3 * (size_t)HD + cc]) * a.norm[cc];
    // channels beyond the block's columns (block = dim * LANES rounded up to a warp, vectors padded to DP)
    for (uint32_t ch = blockDim.x / LANES + tid; ch < DP; ch += blockDim.x)
        vec[ch] = vec[DP + ch] = vec[2 * DP + ch] = vec[3 * DP + ch] = 0.0f;
    __syncthreads();
    const float o = delta_token<NI>(vec, l4, col < DP ? sv[col] : 0.0f, s);
    if (col < D) store_column<NI, LANES>(colp, D, l4, s);
    if (l4 == 0 && col < D) so[col] = o;
    __syncthreads();
    ss = 0.0f;
    for (uint32_t ch = lane; ch < D; ch += 32u) ss = fmaf(so[ch], so[ch], ss);
    const float rs = 1.0f / sqrtf(warp_sum(ss) / (float)D + a.eps);
    if (l4 == 0 && col < D) a.out[(size_t)row * HD + cc] = so[col] * rs * gate;
}

template <int NI>
int run_decode(M40llmCudaContext* ctx, const DeltaArgs& a) {
    const uint32_t threads = (a.dim * LANES + 31u) & ~31u;
    const cudaError_t e =
        m40_launch_dependent(delta_decode_kernel<NI>, dim3(a.heads, a.rows), dim3(threads), 0, ctx->decode_stream, a);
    M40_COUNT_LAUNCH(ctx);
    return e == cudaSuccess && cudaGetLastError() == cudaSuccess ? 0 : -6;
}

template <int NI, int LANES, int COLS>
int launch_scan(M40llmCudaContext* ctx, const DeltaArgs& a, const float* rec, uint32_t n_rec, uint32_t base, uint32_t pass, uint32_t segments,
                uint32_t stages) {
    constexpr int DP = NI * LANES * 4, BLOCK_COLS = SCAN_THREADS / LANES * COLS;
    const size_t smem = stages * scan_stage_bytes(DP);
    // contexts on several threads may set it at the same time: setting it twice is harmless, losing another device's bit is not
    static std::atomic<unsigned long long> configured{0ull};
    const unsigned long long bit = 1ull << (ctx->device_id & 63);
    if (!(configured.load(std::memory_order_acquire) & bit)) {
        if (cudaFuncSetAttribute(delta_scan_kernel<NI, LANES, COLS>, cudaFuncAttributeMaxDynamicSharedMemorySize, SCAN_SMEM) != cudaSuccess)
            return -6;
        configured.fetch_or(bit, std::memory_order_release);
    }
    const dim3 grid((a.dim + BLOCK_COLS - 1) / BLOCK_COLS, a.heads, segments);
    const cudaError_t e = m40_launch_dependent(delta_scan_kernel<NI, LANES, COLS>, grid, dim3(SCAN_THREADS), smem, ctx->decode_stream, a, rec,
                                               n_rec, base, base, pass, stages);
    M40_COUNT_LAUNCH(ctx);
    return e == cudaSuccess ? 0 : -6;
}

// P: 32-key pieces of a column. The forms that delta_scan_plan.cuh chooses from.
template <int P>
int launch_planned(M40llmCudaContext* ctx, const DeltaArgs& a, const float* rec, uint32_t n_rec, uint32_t base, uint32_t pass, uint32_t segments,
                   uint32_t stages, const M40ScanPlan& plan) {
    if constexpr (P % 2 == 0)
        if (plan.lanes == 16) return launch_scan<P / 2, 16, 2>(ctx, a, rec, n_rec, base, pass, segments, stages);
    if constexpr (P <= 4)
        if (plan.cols == 4) return launch_scan<P, 8, 4>(ctx, a, rec, n_rec, base, pass, segments, stages);
    return launch_scan<P, 8, 2>(ctx, a, rec, n_rec, base, pass, segments, stages);
}

template <int P>
int run_scan(M40llmCudaContext* ctx, const DeltaArgs& a, uint32_t segments, uint32_t max_segment_rows) {
    constexpr int DP = P * 32;
    constexpr uint32_t CHUNK = SCAN_CHUNK;
    cudaStream_t s = ctx->decode_stream;
    static_assert(2 * scan_stage_bytes(DP) <= SCAN_SMEM, "the ring needs two slots");
    // One segment is walked in passes of rows whose records fit PASS_BYTES; several segments take one pass.
    const size_t per_row = (size_t)a.heads * rec_floats(DP) * sizeof(float);
    uint32_t pass = max_segment_rows;
    if (segments == 1) {
        const size_t fit = PASS_BYTES / per_row / CHUNK * CHUNK;
        pass = fit < CHUNK ? CHUNK : (fit < pass ? (uint32_t)fit : pass);
    }
    const uint32_t n_rec = segments == 1 ? pass : a.rows;
    float* rec = (float*)m40_ensure_scratch(ctx, 1, n_rec * per_row, 1);
    if (!rec) return -5;
    const M40ScanPlan plan = m40_scan_plan(a.dim, a.heads, segments, segments == 1 ? max_segment_rows : a.rows, max_segment_rows, (uint32_t)ctx->sm_count);
    const uint32_t fit = (uint32_t)(SCAN_SMEM / plan.per_sm / scan_stage_bytes(DP));
    const uint32_t stages = fit < 2u ? 2u : (fit > SCAN_MAX_STAGES ? SCAN_MAX_STAGES : fit);
    cudaError_t e;
    for (uint32_t base = 0; base < max_segment_rows; base += pass) {
        // `rows` of the step from `base` on: with one segment the pass's rows, with several all of them
        const uint32_t rows = segments == 1 ? (a.rows - base < pass ? a.rows - base : pass) : a.rows;
        e = m40_launch_dependent(delta_prepare_kernel<DP>, dim3((rows * a.heads + 7) / 8), dim3(256), 0, s, a, rec, n_rec, base, rows);
        M40_COUNT_LAUNCH(ctx);
        if (e != cudaSuccess) return -6;
        const int rc = launch_planned<P>(ctx, a, rec, n_rec, base, pass, segments, stages, plan);
        if (rc != 0) return rc;
    }
    e = m40_launch_dependent(delta_finish_kernel, dim3((a.rows * a.heads + 7) / 8), dim3(256), 0, s, a);
    M40_COUNT_LAUNCH(ctx);
    return e == cudaSuccess && cudaGetLastError() == cudaSuccess ? 0 : -6;
}

}  // namespace

extern "C" {

int m40llm_delta_rule_async(M40llmCudaContext* ctx, M40llmStateCache* st, const M40llmDeltaRule* c,
                            const M40llmStepRows* rows) {
    if (!ctx || !st || !c || !rows || !c->packed || !c->w0 || !c->a_bias || !c->norm || !c->out) return -1;
    if (!c->decay_in && (!c->w2 || c->rank == 0 || c->rank > 1024)) return -2;
    if (st->dim == 0) return -3;  // a cache of plain values
    if (rows->rows == 0 || rows->segments == 0 || rows->max_segment_rows == 0) return -2;
    if (rows->max_segment_rows == 1 ? (!rows->row_seq || !rows->row_pos) : !rows->seg) return -1;
    if (c->w_dtype > M40LLM_DT_BF16) return -3;
    const uint64_t need = 5ull * st->heads * st->dim + (c->decay_in ? 0u : c->rank);
    if (c->ld < need) return -2;
    if (m40_ensure_device(ctx) != 0) return -1;
    DeltaArgs a = {};
    a.packed = (const float*)c->packed;
    a.w2 = c->w2;
    a.w0 = (const float*)c->w0;
    a.a_bias = (const float*)c->a_bias;
    a.norm = (const float*)c->norm;
    a.decay_in = (const float*)c->decay_in;
    a.out = (float*)c->out;
    a.state = st->d_state;
    a.status = ctx->d_status;
    a.row_seq = rows->row_seq;
    a.row_pos = rows->row_pos;
    a.seg = rows->seg;
    a.ld = c->ld;
    a.rank = c->rank;
    a.w2_dtype = c->w_dtype;
    a.w2_wide = !c->decay_in && c->w_dtype != M40LLM_DT_F32 && c->rank % 8 == 0 && c->rank <= 128 && ((uintptr_t)c->w2 & 15u) == 0;
    a.heads = st->heads;
    a.dim = st->dim;
    a.slots = st->slots;
    a.slot_mul = rows->slot_mul;
    a.slot_add = rows->slot_add;
    a.rows = rows->rows;
    a.decay_scale = c->decay_scale;
    a.unit_eps = c->unit_eps;
    a.eps = c->eps;
    if (rows->max_segment_rows > 1) {
        // rows outside the segment's range must not be prepared: with one segment it must start at row 0 and span the step
        const uint32_t sg = rows->segments, mx = rows->max_segment_rows;
        if (sg == 1 && mx != rows->rows) return -2;
        switch ((st->dim + 31) / 32) {  // 32-channel pieces per lane group
            case 1: return run_scan<1>(ctx, a, sg, mx);
            case 2: return run_scan<2>(ctx, a, sg, mx);
            case 3: return run_scan<3>(ctx, a, sg, mx);
            case 4: return run_scan<4>(ctx, a, sg, mx);
            case 5: case 6: return run_scan<6>(ctx, a, sg, mx);
            default: return run_scan<8>(ctx, a, sg, mx);
        }
    }
    switch ((st->dim + 15) / 16) {  // 16-channel pieces per lane group
        case 1: return run_decode<1>(ctx, a);
        case 2: return run_decode<2>(ctx, a);
        case 3: return run_decode<3>(ctx, a);
        case 4: return run_decode<4>(ctx, a);
        case 5: return run_decode<5>(ctx, a);
        case 6: return run_decode<6>(ctx, a);
        case 7: case 8: return run_decode<8>(ctx, a);
        case 9: case 10: case 11: case 12: return run_decode<12>(ctx, a);
        default: return run_decode<16>(ctx, a);
    }
}

}  // extern "C"
