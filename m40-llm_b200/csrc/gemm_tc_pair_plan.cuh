// How a projection of many rows is cut for the CTA-pair kernel (gemm_tc_pair.cu). Host arithmetic only.
#pragma once
#include <stdint.h>

constexpr uint32_t M40_PAIR_ROWS = 256;  // weight rows of a tile: 128 per CTA of the pair

struct M40PairPlan {
    uint32_t m_tiles, width;        // activation rows per tile (multiple of 32)
    uint32_t k_splits, kb_per_split;
    uint32_t tiles;                 // weight tiles of all problems
    uint32_t tile_begin[4];
    bool paired;                    // gate | up: a tile holds gate and up rows of the same outputs
    uint32_t n_sum;                 // weight rows of all problems
};

// One way to cut `M` rows against problems of N[p] weight rows for `pairs` resident CTA pairs. `paired`: problems 0 | 1 share tiles and
// K is not split. `partial_only`: a second kernel finishes the sums whatever the split.
inline bool m40_pair_cut(uint32_t pairs, uint32_t M, uint32_t kblocks, uint32_t problems, const int* N, bool paired, bool partial_only,
                         M40PairPlan* plan) {
    if (pairs == 0 || M == 0) return false;
    constexpr double A_BYTES = 128.0 * 64.0 * 2.0;
    uint32_t tiles = 0, n_sum = 0;
    for (uint32_t p = 0; p < (paired ? 1u : problems); ++p) {
        plan->tile_begin[p] = tiles;
        const uint32_t rows = paired ? M40_PAIR_ROWS / 2 : M40_PAIR_ROWS;
        tiles += ((uint32_t)N[p] + rows - 1) / rows;
        n_sum += (uint32_t)N[p];
    }
    for (uint32_t p = paired ? 1u : problems; p < 4; ++p) plan->tile_begin[p] = tiles;
    plan->tiles = tiles;
    plan->paired = paired;
    // Cycles of a call: full waves of units, each kb_per_split k-blocks long, paced by the MMAs (4 cycles per activation row and
    // k-block, and at least the 90 cycles per MMA that its weight operand takes) or by L2 (about 50 bytes a cycle and SM); then
    // the last tile's stores, and, where partial sums are needed, their way to L2 and back.
    plan->n_sum = n_sum;
    double best = 0.0;
    for (uint32_t width = 32; width <= 256u; width += 32) {
        const uint32_t m_tiles = (M + width - 1) / width;
        if (m_tiles > 1 && ((M + m_tiles - 1) / m_tiles + 31) / 32 * 32 != width) continue;  // a narrower tile gives as few
        if (m_tiles == 1 && width >= M + 32) continue;
        const double mma = 4.0 * width > 720.0 ? 4.0 * width : 720.0, load = (A_BYTES + 128.0 * width) / 50.0;
        for (uint32_t ks = 1; ks <= (paired ? 1u : 16u) && (ks == 1 || kblocks / ks >= 4); ++ks) {
            const uint32_t per = (kblocks + ks - 1) / ks, real = (kblocks + per - 1) / per;
            if (real != ks) continue;
            const uint64_t units = (uint64_t)tiles * m_tiles * ks;
            const double waves = (double)((units + pairs - 1) / pairs);
            double cost = waves * per * (mma > load ? mma : load) + 2000.0 + 12.0 * width;
            if (ks > 1 || partial_only) cost += 5000.0 + (double)ks * M * n_sum * 8.0 / (2.0 * pairs * 25.0);
            if (best == 0.0 || cost < best) {
                best = cost;
                plan->width = width;
                plan->m_tiles = m_tiles;
                plan->k_splits = ks;
                plan->kb_per_split = per;
            }
        }
    }
    return best > 0.0;
}

// Cycles of a gate | up call cut one way or the other. Unlike above, what a k-block takes at any width counts (a lone pair: 72 to 76 us
// for 128 of them at 129 as at 512 rows); with these numbers the choice below was within 7 % of the better way in each of 442 measured
// calls of 129 to 2048 rows, 64 to 8192 outputs and K of 64 to 8192, and within 0.03 % on average.
inline double m40_pair_gate_up_cycles(const M40PairPlan& p, uint32_t pairs, uint32_t M) {
    const double waves = (double)(((uint64_t)p.tiles * p.m_tiles * p.k_splits + pairs - 1) / pairs);
    double pace = (128.0 * 64.0 * 2.0 + 128.0 * p.width) / 50.0;
    if (pace < 4.0 * p.width) pace = 4.0 * p.width;
    if (pace < 1080.0) pace = 1080.0;
    const double sums = waves * p.kb_per_split * pace + 2000.0 + 12.0 * p.width;
    return p.paired ? sums : sums + 3500.0 + (double)p.k_splits * M * p.n_sum * 8.0 / (2.0 * pairs * 35.0);
}

// The cheapest way. Gate | up calls either share tiles, which finishes them in one kernel but leaves K whole, or run as two problems
// with K splits and a second kernel, the better way for narrow and deep ones: 200 rows, 2 x 640 outputs, K = 8192: 25 against 73 us;
// 2 x 4096, K = 2048: 25 against 29; 256 rows, 2 x 8192, K = 64: 27 against 14.
inline bool m40_pair_cut_best(uint32_t pairs, uint32_t M, uint32_t kblocks, uint32_t problems, const int* N, bool gate_up, bool partial_only,
                              M40PairPlan* plan) {
    if (!m40_pair_cut(pairs, M, kblocks, problems, N, false, partial_only || gate_up, plan)) return false;
    M40PairPlan shared;
    if (gate_up && m40_pair_cut(pairs, M, kblocks, problems, N, true, false, &shared) &&
        m40_pair_gate_up_cycles(shared, pairs, M) <= m40_pair_gate_up_cycles(*plan, pairs, M))
        *plan = shared;
    return true;
}
