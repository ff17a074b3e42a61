// What attention over the rows of a prompt takes, in us on a B200, in each of the forms there are: the tcgen05 kernel (attention_prefill_tc.cu)
// with one or two tiles of 128 rows per CTA, the mma.sync kernel (64 x 64, attention_prefill.cu) and the decode kernels (every row reads
// its own context, attention_tiled.cu). Host arithmetic only; the numbers are fits to measured calls: about 900 for the mma.sync and the
// decode form (1 to 32 segments of 16 to 1024 rows at positions 0 to 8192; 32 / 8, 16 / 2 and 8 / 2 heads of 128, 32 / 4 and 8 / 8 of 64), 210
// for either form of the tcgen05 kernel (1 to 16 segments of 65 to 2048 rows at positions 0 to 4000; also 33 / 11 of 128 and 40 / 40 of 64).
//
// The prompt kernels walk a row tile's keys in one CTA. A CTA costs a fixed part and so much per key tile; the tcgen05 kernel has
// one CTA per SM, the mma.sync kernel two, which share it. So the former wins over long contexts (65 rows: 28 us against 33 at
// position 2048, 32 / 4 heads of 64; 33 against 59 with 32 / 8 of 128), the latter over short ones (32 segments of 65 rows at position 0:
// 65 against 50 us, 49 against 30) and where a call has short segments beside long ones, whose grid has many CTAs without rows (31
// segments of 16 rows and one of 300: 73 against 36 us). The decode form wins where few rows have a long context: 16 rows at 8192:
// 71 us against 210 (32 / 8 heads of 128), 26 against 114 (32 / 4 of 64).
//
// Two row tiles per CTA take about twice as long a key tile as one, and save in all an eighth of the time, so they win where CTAs of either
// are enough to balance: 2048 rows of 32 / 8 heads of 128 68 against 76 us, but 1500 rows of 16 / 2 47 against 26 and 1000 of 32 / 8 35
// against 27. A group with an odd number of heads pairs rows that follow one another, and a short segment's second tile is empty: 16
// segments of 65 rows at position 2000, 40 / 40 heads of 64, 250 against 140.
//
// Choices by these estimates were at most 1 % slower in the calls measured than the kernel with one tile per CTA and the mma.sync kernel
// were by the estimates before there were two.
#pragma once
#include <stdint.h>

#include <algorithm>

// Calls whose longest segment is shorter than this stay on the mma.sync kernel: it fills one of its 64-row tiles and half of a
// 128-row tile of the other.
constexpr uint32_t M40_PREFILL_TC_MIN_ROWS = 65;

class M40PromptCost {
public:
    M40PromptCost(uint32_t head_dim, uint32_t q_heads, uint32_t kv_heads, uint32_t sms, uint32_t max_segment_rows)
        : hd_(head_dim), heads_(q_heads), kv_heads_(kv_heads), kv_values_((double)kv_heads * head_dim), sms_(sms), max_rows_(max_segment_rows) {}

    // `times` segments of `rows` rows from position `pos` on.
    void add(uint32_t rows, uint32_t pos, uint32_t times = 1) {
        segments_ += times;
        rows_ += (double)times * rows;
        reads_ += (double)times * rows * (pos + 0.5 * rows);
        one_.add(128, rows, pos, times);
        two_.add(heads_ / kv_heads_ % 2 == 0 ? 128 : 256, rows, pos, times);
        mma_.add(64, rows, pos, times);
    }

    double tc_one_us() const {
        return hd_ == 128 ? one_.us(heads_, sms_, max_rows_, segments_, 8.0, 1.47, 1.151, -2.88) : one_.us(heads_, sms_, max_rows_, segments_, 5.54, 1.329, 1.011, 2.19);
    }
    double tc_two_us() const {
        const uint32_t heads = two_.size == 128 ? heads_ / 2 : heads_;
        return hd_ == 128 ? two_.us(heads, sms_, max_rows_, segments_, 8.73, 3.175, 1.236, -1.59) : two_.us(heads, sms_, max_rows_, segments_, 6.3, 2.697, 1.11, 0.25);
    }
    bool tc_two() const { return tc_two_us() < tc_one_us(); }  // two row tiles per CTA
    double tc_us() const { return std::min(tc_one_us(), tc_two_us()); }
    double mma_us() const {
        return hd_ == 128 ? mma_.us(*this, 4.5, 1.6, 1.7, 1.27, 0.4) : mma_.us(*this, 3.3, 0.84, 1.1, 0.72, 0.35);
    }
    double prompt_us() const { return max_rows_ >= M40_PREFILL_TC_MIN_ROWS ? std::min(tc_us(), mma_us()) : mma_us(); }
    double decode_us() const { return 6.0 + rows_ * (0.08 + 1.7e-4 * kv_values_) + reads_ * kv_values_ * 4.0 / 1e7; }

private:
    // CTAs of one head (or pair of heads) of the tcgen05 kernel: `size` rows, tiles of 128 keys
    struct Ctas {
        double ctas = 0.0, keys = 0.0, longest = 0.0, shortest = 1e30;
        uint32_t size = 128;
        void add(uint32_t rows_per_cta, uint32_t rows, uint32_t pos, uint32_t times) {
            size = rows_per_cta;
            const double t = (rows + size - 1) / size, step = size / 128, before = (pos + 127) / 128, last = (pos + (uint64_t)rows + 127) / 128;
            ctas += times * t;
            keys += times * ((t - 1.0) * before + step * 0.5 * t * (t - 1.0) + last);
            longest = std::max(longest, last);
            shortest = std::min(shortest, t > 1.0 ? before + step : last);
        }
        // The longest CTA; or all of them spread over the SMs, by a factor and an offset for what the spreading leaves; or, longest first,
        // what an SM at least gets whose CTAs are one more than fit otherwise. 0.9 us per CTA without rows.
        double us(uint32_t heads, uint32_t sms, uint32_t max_rows, uint32_t segments, double fixed, double per_tile, double factor, double offset) const {
            const double all = heads * ctas, grid = (double)heads * segments * ((max_rows + size - 1) / size);
            const double waves = (double)(((uint64_t)all + sms - 1) / sms);
            double t = fixed + per_tile * longest;
            if (waves > 1.0) {
                const double nth = longest - (waves - 1.0) * sms / all * (longest - shortest);
                t = std::max({t, factor * (all * fixed + heads * keys * per_tile) / sms + offset, waves * (fixed + per_tile * nth)});
            }
            return t + 0.9 * (grid - all) / sms;
        }
    };
    // the mma.sync kernel's
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
        double us(const M40PromptCost& c, double fixed, double per_tile, double shared_fixed, double shared_tile, double empty) const {
            const double all = c.heads_ * ctas, grid = (double)c.heads_ * c.segments_ * ((c.max_rows_ + size - 1) / size);
            const double waves = (double)(((uint64_t)all + c.sms_ - 1) / c.sms_);
            const double many = waves <= 1.0 ? 0.0 : waves * (shared_fixed + shared_tile * keys / std::max(ctas, 1.0));
            return std::max(fixed + per_tile * longest, many) + empty * (grid - all) / c.sms_;
        }
    };
    Ctas one_, two_;
    Tiles mma_;
    uint32_t hd_, heads_, kv_heads_;
    double kv_values_;
    uint32_t sms_, max_rows_, segments_ = 0;
    double rows_ = 0.0, reads_ = 0.0;
};
