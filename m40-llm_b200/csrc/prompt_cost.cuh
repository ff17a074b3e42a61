// What attention over the rows of a prompt takes, in us on a B200, in each of the forms there are: the tcgen05 kernel (128 x 128 tiles,
// attention_prefill_tc.cu), the mma.sync kernel (64 x 64, attention_prefill.cu) and the decode kernels (every row reads its own
// context, attention_tiled.cu). Host arithmetic only; the numbers are fits to about 900 measured calls (1 to 32 segments of 16 to 1024
// rows at positions 0 to 8192; 32 / 8, 16 / 2 and 8 / 2 heads of 128, 32 / 4 and 8 / 8 of 64).
//
// The two prompt kernels walk a row tile's keys in one CTA. A CTA costs a fixed part and so much per key tile; the tcgen05 kernel has
// one CTA per SM, the mma.sync kernel two, which share it. So the former wins over long contexts (65 rows: 28 us against 33 at
// position 2048, 32 / 4 heads of 64; 33 against 59 with 32 / 8 of 128), the latter over short ones (32 segments of 65 rows at position 0:
// 65 against 50 us, 49 against 30) and where a call has short segments beside long ones, whose grid has many CTAs without rows (31
// segments of 16 rows and one of 300: 73 against 36 us). The decode form wins where few rows have a long context: 16 rows at 8192:
// 71 us against 210 (32 / 8 heads of 128), 26 against 114 (32 / 4 of 64). Choices by these estimates were at most 1 % slower than
// the decode form or the mma.sync form alone, where the worst of them would have been nine times as slow.
#pragma once
#include <stdint.h>

#include <algorithm>

// Calls whose longest segment is shorter than this stay on the mma.sync kernel: it fills one of its 64-row tiles and half of a
// 128-row tile of the other.
constexpr uint32_t M40_PREFILL_TC_MIN_ROWS = 65;

class M40PromptCost {
public:
    M40PromptCost(uint32_t head_dim, uint32_t q_heads, uint32_t kv_heads, uint32_t sms, uint32_t max_segment_rows)
        : hd_(head_dim), heads_(q_heads), kv_values_((double)kv_heads * head_dim), sms_(sms), max_rows_(max_segment_rows) {}

    // `times` segments of `rows` rows from position `pos` on.
    void add(uint32_t rows, uint32_t pos, uint32_t times = 1) {
        segments_ += times;
        rows_ += (double)times * rows;
        reads_ += (double)times * rows * (pos + 0.5 * rows);
        tc_.add(128, rows, pos, times);
        mma_.add(64, rows, pos, times);
    }

    double tc_tiles() const { return heads_ * tc_.ctas; }
    double tc_us() const {
        return hd_ == 128 ? tc_.us(*this, 8.5, 1.45, 8.5, 1.45, 0.9, false) : tc_.us(*this, 7.3, 1.25, 7.3, 1.25, 0.9, false);
    }
    double mma_us() const {
        return hd_ == 128 ? mma_.us(*this, 4.5, 1.6, 1.7, 1.27, 0.4, true) : mma_.us(*this, 3.3, 0.84, 1.1, 0.72, 0.35, true);
    }
    double prompt_us() const { return max_rows_ >= M40_PREFILL_TC_MIN_ROWS ? std::min(tc_us(), mma_us()) : mma_us(); }
    double decode_us() const { return 6.0 + rows_ * (0.08 + 1.7e-4 * kv_values_) + reads_ * kv_values_ * 4.0 / 1e7; }

private:
    struct Tiles {
        double ctas = 0.0, keys = 0.0, longest = 0.0;
        uint32_t size = 1;
        void add(uint32_t tile, uint32_t rows, uint32_t pos, uint32_t times) {
            size = tile;
            const double t = (rows + tile - 1) / tile, last = (pos + (uint64_t)rows + tile - 1) / tile;
            ctas += times * t;
            keys += times * (t > 1.0 ? t * ((pos + 0.5 * rows) / tile + 0.5) : last);
            longest = std::max(longest, last);
        }
        // A CTA that has an SM to itself: fixed + per_tile; one of several: shared_*; one without rows: empty.
        double us(const M40PromptCost& c, double fixed, double per_tile, double shared_fixed, double shared_tile, double empty, bool shares) const {
            const double all = c.heads_ * ctas, grid = (double)c.heads_ * c.segments_ * ((c.max_rows_ + size - 1) / size);
            const double waves = (double)(((uint64_t)all + c.sms_ - 1) / c.sms_);
            const double many = shares && waves <= 1.0 ? 0.0 : waves * (shared_fixed + shared_tile * keys / std::max(ctas, 1.0));
            return std::max(fixed + per_tile * longest, many) + empty * (grid - all) / c.sms_;
        }
    };
    Tiles tc_, mma_;
    uint32_t hd_, heads_;
    double kv_values_;
    uint32_t sms_, max_rows_, segments_ = 0;
    double rows_ = 0.0, reads_ = 0.0;
};
