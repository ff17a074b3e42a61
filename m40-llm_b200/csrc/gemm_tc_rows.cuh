// Tensor-core GEMM for up to 32 activation rows, one launch from the f32 activations to the finished result; see gemm_tc_rows.cu.
#pragma once
#include <cuda.h>

#include "common.cuh"
#include "gemm_tc.cuh"
#include "stack_math.cuh"

constexpr uint32_t M40_ROWS_MAX = 32;

// What the kernel makes its activation operand from. With the f32 sources the result must not lie over x.
enum {
    M40_ROWS_SPLIT = 0,  // hi and lo copies that another kernel has made
    M40_ROWS_F16 = 1,    // f32 rows, split into f16 hi + lo on the way
    M40_ROWS_BF16 = 2,   // the same in bf16
};

struct M40RowsArgs {
    const float* x;          // not for M40_ROWS_SPLIT: [M][ldx], 16-byte aligned, ldx a multiple of 4
    uint32_t ldx;
    uint32_t* status;
    uint32_t M, K;
    uint32_t problems, paired;  // paired: problems 0 and 1 share tiles of 64 + 64 rows, out = act(first) * second
    uint32_t fmt_bits;          // operand type bits of the instruction descriptor
    uint32_t N[3];
    float* out[3];
    const float* bias[3];
    const float* residual[3];
    const float* post_w;     // tail.post == DYT: problem 0 only
    const float* post_b;
    int act;
    M40Tail tail;
    uint32_t rope_on;
    M40TcRopeAppend rope;
    // filled in by the launch
    uint32_t kblocks, kb_per_split, stages, vec_out;
    uint32_t tile_begin[4];
};

// w: boxes of 128 weight rows (paired: 64); xh, xl: boxes of M rows, padded to a multiple of 16, for M40_ROWS_SPLIT only.
int m40_rows_launch(M40llmCudaContext* ctx, cudaStream_t s, int source, const CUtensorMap* w, const CUtensorMap& xh,
                    const CUtensorMap& xl, M40RowsArgs a);
