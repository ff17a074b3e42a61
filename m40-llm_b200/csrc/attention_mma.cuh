// Warp-level building blocks shared by the attention kernels: cp.async, ldmatrix, mma.sync m16n8k16 (f16 inputs,
// f32 accumulate), fast exp2 and the f32 -> (hi, lo) f16 split.
#pragma once
#include <cuda_fp16.h>
#include <stdint.h>

namespace attn_mma {

constexpr float LOG2E = 1.4426950408889634f;
constexpr float LN2 = 0.6931471805599453f;

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N)); }

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], const void* smem) {
    const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(s));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], const void* smem) {
    const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(s));
}
// D (f32, m16n8) += A (f16, m16k16) * B (f16, k16n8)
__device__ __forceinline__ void mma16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                         uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ uint32_t pack_h2(float lo, float hi) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}
// f32 pair -> (hi, lo) f16 pairs with hi + lo == the f32 value to ~2^-22 relative
__device__ __forceinline__ void split_h2(float x, float y, uint32_t* hi, uint32_t* lo) {
    const __half hx = __float2half_rn(x), hy = __float2half_rn(y);
    const __half2 h = __halves2half2(hx, hy);
    *hi = *reinterpret_cast<const uint32_t*>(&h);
    *lo = pack_h2(x - __half2float(hx), y - __half2float(hy));
}

// Zero weights do not cancel an infinity or a NaN: in a tile that a row sees in part, the value product hands the row what later
// tokens hold. The prompt kernels therefore look at what comes out, and a row with something that is not finite in it gets those
// dimensions once more from the keys that it sees, in plain f32. One warp; row of q with q_dim values, weights relative to `ref` in
// base 2, not normalised. Lane l returns dimensions d, d + 1 (x, y) and d + 64, d + 65 (z, w; HD 128) with d = 2 l.
__device__ __forceinline__ bool is_finite(float v) { return fabsf(v) <= 3.402823466e38f; }
template <int HD>
__device__ __noinline__ float4 attend_row(const float* q, uint32_t q_dim, float scale, const __half* K, const __half* V, size_t pitch,
                                          uint32_t n, float ref) {
    const uint32_t d = 2u * (threadIdx.x & 31u);
    const auto q_at = [&](uint32_t i) { return i < q_dim ? q[i] * scale : 0.0f; };
    const float4 x = make_float4(q_at(d), q_at(d + 1u), HD == 128 ? q_at(d + 64u) : 0.0f, HD == 128 ? q_at(d + 65u) : 0.0f);
    float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 4
    for (uint32_t t = 0; t < n; ++t, K += pitch, V += pitch) {
        const float2 k0 = __half22float2(*reinterpret_cast<const __half2*>(K + d)), v0 = __half22float2(*reinterpret_cast<const __half2*>(V + d));
        float2 k1 = make_float2(0.0f, 0.0f), v1 = k1;
        if (HD == 128) {
            k1 = __half22float2(*reinterpret_cast<const __half2*>(K + d + 64));
            v1 = __half22float2(*reinterpret_cast<const __half2*>(V + d + 64));
        }
        float s = x.x * k0.x + x.y * k0.y + x.z * k1.x + x.w * k1.y;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        const float p = fast_exp2(s - ref);
        acc.x += p * v0.x, acc.y += p * v0.y, acc.z += p * v1.x, acc.w += p * v1.y;
    }
    return acc;
}

}  // namespace attn_mma
