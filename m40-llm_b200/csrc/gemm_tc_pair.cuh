// Tensor-core GEMM for many activation rows on CTA pairs; see gemm_tc_pair.cu.
#pragma once
#include <cuda.h>

#include "common.cuh"
#include "gemm_tc_pair_plan.cuh"
#include "stack_math.cuh"

struct M40PairCall {
    CUtensorMap w[3];     // boxes of 128 weight rows (plan.paired: 64)
    CUtensorMap xh, xl;   // boxes of width / 2 activation rows
    uint32_t M, kblocks, problems;
    uint32_t fmt_bits;    // operand type bits of the instruction descriptor
    float* partial;       // not null: [k_splits][M][tiles * 256] partial sums, nothing else is applied
    float* out;           // else: one problem (or plan.paired), finished and stored
    uint32_t n_out;
    const float* bias;
    const float* residual;
    const float* post_w;
    const float* post_b;
    int act;
    M40Tail tail;
};

bool m40_pair_available(const M40llmCudaContext* ctx);
// m40_pair_cut_best() for this device. `gate_up`: two problems of equal N, out = act(first) * second. False: the device takes no CTA
// pairs.
bool m40_pair_plan(const M40llmCudaContext* ctx, uint32_t M, uint32_t kblocks, uint32_t problems, const int* N, bool gate_up,
                   bool partial_only, M40PairPlan* plan);
int m40_pair_launch(M40llmCudaContext* ctx, cudaStream_t s, const M40PairCall& call, const M40PairPlan& plan);
