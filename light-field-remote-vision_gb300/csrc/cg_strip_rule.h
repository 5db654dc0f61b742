// cg_strip_rule.h -- which images k_cg_strip (kernels_cg.cu) takes, and how it cuts them: units of kStripCols x R pixels,
// kStripUnits of them a block, every block of a launch resident at once. `capacity` is the number of blocks that can be
// resident (0 where a block does not fit an SM); images beyond it run the streamed form.
#pragma once
#include <algorithm>
#include <cstddef>

namespace lfrv {

constexpr int kStripUnits = 4;  // spatial units per block
constexpr int kStripCols = 64;
constexpr int kStripClusterBlocks = 16, kStripClusterR = 8;
constexpr int kCgBatchMaxRows = 28;
constexpr int kStripRows[] = {4, 8, 16, kCgBatchMaxRows};

// Floats a unit exchanges per channel: top row, bottom row, left column, right column.
#ifdef __CUDACC__
__host__ __device__
#endif
constexpr int strip_border(int R) { return 2 * kStripCols + 2 * R; }

inline int strip_blocks(int W, int H, int R) {
    const int units = ((W + kStripCols - 1) / kStripCols) * ((H + R - 1) / R);
    return (units + kStripUnits - 1) / kStripUnits;
}

// Whether the borders of the units fit in dA and in dB (3 N floats each); very thin images do not.
inline bool strip_fits(int W, int H, int R) {
    return (size_t)((W + kStripCols - 1) / kStripCols) * ((H + R - 1) / R) * 3 * strip_border(R) <= (size_t)3 * W * H;
}

// Rows per unit for a W x H image: the smallest R of one cluster while R is at most kStripClusterR, else the smallest R
// that fits the grid (an iteration's arithmetic is proportional to R, its barrier is not); 0: the streamed form.
inline int strip_rows(int W, int H, int capacity) {
    for (int R : kStripRows)
        if (R <= kStripClusterR && strip_fits(W, H, R) &&
            strip_blocks(W, H, R) <= std::min(kStripClusterBlocks, capacity))
            return R;
    for (int R : kStripRows)
        if (strip_fits(W, H, R) && strip_blocks(W, H, R) <= capacity) return R;
    return 0;
}

}  // namespace lfrv
