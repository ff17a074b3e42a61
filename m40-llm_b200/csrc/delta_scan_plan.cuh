// How the scan of the delta rule (delta_rule.cu) is laid out for a call: lanes and columns of a group, and how many CTAs share an SM.
// Host arithmetic only; times from about 150 measured calls (head sizes 16 to 256, 4 to 300 heads, 1 to 32 segments of 2 to 2048 tokens).
//
// A CTA walks its tokens one pair after the other, so its time is tokens times what a pair takes, and that grows with the columns of a
// lane and with the CTAs beside it. 16 lanes with two columns are fastest alone, eight with four do most work per SM, and eight with two
// lie between: 64 heads of 64, 600 tokens of one sequence 132, 159 and 117 us; 48 heads, 12 sequences of 50 tokens 91, 62 and 71. A call
// goes to the form and the number of CTAs per SM whose waves take least by the table, which was at most 3 % over the best of all. The
// number per SM is imposed by the size of the ring: left to themselves, 128 CTAs that could share an SM do (32 heads of 64, 600 tokens: 115
// us instead of 91).
#pragma once
#include <stdint.h>

#include <algorithm>

constexpr uint32_t M40_SCAN_THREADS = 128;

struct M40ScanPlan {
    uint32_t lanes, cols, per_sm;
    double ns;  // estimate
};

// `rows` tokens in `segments` segments, the longest of `longest`.
inline M40ScanPlan m40_scan_plan(uint32_t dim, uint32_t heads, uint32_t segments, uint32_t rows, uint32_t longest, uint32_t sms) {
    // lanes, columns of a lane
    constexpr uint32_t FORMS[3][2] = {{16, 2}, {8, 2}, {8, 4}};
    // ns per token of a CTA that has its SM to itself, shares it with one, with two; by 32-key pieces of a column. 0: not built (an odd number
    // of pieces does not divide over 16 lanes, four columns of more than four pieces do not fit the registers) or too large for the SM.
    constexpr uint16_t NS[6][3][3] = {
        {{0, 0, 0}, {152, 279, 393}, {184, 331, 471}},
        {{118, 149, 189}, {124, 178, 248}, {181, 254, 343}},
        {{0, 0, 0}, {154, 242, 348}, {231, 352, 485}},
        {{137, 199, 0}, {195, 319, 0}, {305, 467, 0}},
        {{146, 0, 0}, {272, 0, 0}, {0, 0, 0}},  // five or six
        {{196, 0, 0}, {392, 0, 0}, {0, 0, 0}},  // seven or eight
    };
    constexpr uint32_t START = 16;  // what starting and ending a CTA takes, in tokens
    const uint32_t pieces = std::max((dim + 31) / 32, 1u), row = pieces <= 4 ? pieces - 1 : (pieces <= 6 ? 4 : 5);
    // segments as long as the longest that do as much work: single tokens beside a prompt are soon over
    const uint64_t units = (uint64_t)rows + (uint64_t)START * segments, most = longest + START;
    const uint64_t equal = std::max<uint64_t>((units + most - 1) / most, 1);
    M40ScanPlan best = {8, 2, 1, 1e30};
    for (uint32_t f = 0; f < 3; ++f) {
        // a CTA of few columns takes as long to start as another (33 tokens, 32 heads of 64: 12.1 and 11.5 us; 16 heads of 128: 13.1 and 15.6)
        if (FORMS[f][0] == 16 && pieces <= 2 && longest < 64) continue;
        const uint32_t cols = M40_SCAN_THREADS / FORMS[f][0] * FORMS[f][1];
        const uint64_t ctas = (uint64_t)((dim + cols - 1) / cols) * heads * equal;
        for (uint32_t per = 1; per <= 3; ++per) {
            const uint16_t* ns = NS[row][f];
            if (ns[per - 1] == 0) break;
            const uint64_t wave = (uint64_t)sms * per, full = ctas / wave, rest = ctas % wave;
            const double t = (double)most * ((double)full * ns[per - 1] + (rest ? ns[(rest + sms - 1) / sms - 1] : 0));
            if (t < best.ns) best = {FORMS[f][0], FORMS[f][1], per, t};
            if (full == 0) break;  // more per SM would change nothing
        }
    }
    return best;
}
