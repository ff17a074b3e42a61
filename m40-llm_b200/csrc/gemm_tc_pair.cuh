// Tensor-core GEMM for many activation rows on CTA pairs; see gemm_tc_pair.cu.
#pragma once
#include <cuda.h>

#include "common.cuh"
#include "stack_math.cuh"

constexpr uint32_t M40_PAIR_ROWS = 256;  // weight rows of a tile: 128 per CTA of the pair

// How a call is cut; made by m40_pair_plan().
struct M40PairPlan {
    uint32_t m_tiles, width;        // activation rows per tile (multiple of 32)
    uint32_t k_splits, kb_per_split;
    uint32_t tiles;                 // weight tiles of all problems
    uint32_t tile_begin[4];
};

struct M40PairCall {
    CUtensorMap w[3];     // boxes of 128 weight rows (paired: 64)
    CUtensorMap xh, xl;   // boxes of width / 2 activation rows
    uint32_t M, kblocks, problems;
    uint32_t fmt_bits;    // operand type bits of the instruction descriptor
    uint32_t paired;      // problems 0 | 1 are gate | up of equal N: out = act(gate) * up
    float* partial;       // not null: [k_splits][M][tiles * 256] partial sums, nothing else is applied
    float* out;           // else: one problem (or paired), finished and stored
    uint32_t n_out;
    const float* bias;
    const float* residual;
    const float* post_w;
    const float* post_b;
    int act;
    M40Tail tail;
};

// Cuts `M` rows against problems of N[p] weight rows. `partial_only`: the caller's epilogue kernel finishes the sums whatever
// the split. False: the device takes no CTA pairs.
bool m40_pair_plan(const M40llmCudaContext* ctx, uint32_t M, uint32_t kblocks, uint32_t problems, const int* N, bool paired,
                   bool partial_only, M40PairPlan* plan);
int m40_pair_launch(M40llmCudaContext* ctx, cudaStream_t s, const M40PairCall& call, const M40PairPlan& plan);
