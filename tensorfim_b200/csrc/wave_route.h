// The automatic counter choice of a counting wave (tfim_count_wave), free of CUDA so that it can be
// compiled and checked by itself.
#pragma once
#include <cmath>
#include <cstdint>

namespace tfim {

// Share of 128-bit pieces that a one-item prefix leaves empty, the item taken with a probability in
// proportion to its support: what the CUDA-core tiles, which skip empty pieces, can leave unread.
inline float empty_pieces(const int32_t* support, int64_t n, int64_t n_bits) {
    double s1 = 0, s2 = 0;
    for (int64_t k = 0; k < n; k++) {
        s1 += support[k];
        s2 += (double)support[k] * support[k];
    }
    return s1 > 0 && n_bits > 0 ? (float)std::pow(1.0 - std::fmin(1.0, s2 / s1 / (double)n_bits), 128.0) : 0.f;
}

// Whether the tensor tiles (kind::mxf4) count a wave of `rows` prefixes x `cols` items over rows of
// `words` words.  They take from min_rows x min_cols on (the tuning table's i8_min_rows, 3, and
// i8_min_cols), up to two rows earlier where that pays and up to four rows later where it does not:
// their time hardly depends on the rows, about 36 us and 2.5 us per 10,000 words of every 128
// columns, while the CUDA-core tiles read what the prefixes leave of the columns' pieces.
// Lines from 125 shapes (8 to 6,162 items, 10,000 to 8.4M transactions, dense and long-tailed) x 1 to 32
// rows, us on the CUDA cores / on the tensor tiles:
//   1 row:  69 dense items x 262,144 tx 71 / 39, 6,162 long-tail items x 500,000 46 / 252
//   2 rows: 1,200 long-tail items x 130,000 82 / 51, 4,000 x 262,144 98 / 125
//   3 rows: 2,000 long-tail items x 500,000 142 / 110, 6,162 x 130,000 71 / 108, 16 dense x 8.4M 54 / 84
//   8 rows: 6,162 long-tail items x 500,000 237 / 254, every other shape in favour of the tensor tiles
constexpr int64_t kRouteShort = 10000;      // words of every 128 columns: the call is launch-bound
constexpr int64_t kRouteMid = 120000;       // ... and few rows still win
constexpr int64_t kRouteWords = 1 << 14;    // words per row up to which one or two rows can win
inline bool wave_on_tensor(int64_t rows, int64_t cols, int64_t words, float empty, int32_t min_rows, int32_t min_cols) {
    const int64_t r = rows - min_rows + 3;   // as if the table's line were 3 rows
    if (r < 1 || cols < min_cols) return false;
    if (r >= 8) return true;
    const int64_t work = (cols + 127) / 128 * words;
    if (r < 3) return work <= kRouteShort || (words <= kRouteWords && empty < (r == 1 ? 1e-6f : 0.3f));
    return work <= kRouteMid || (cols > 16 && empty < 0.5f);
}

}  // namespace tfim
