// Which kernels a level runs, by its size: rules on whole numbers alone, checked
// without a GPU (tests/cpp/rules.cpp).
#pragma once

namespace rf {

// The tile of the two-pixel half-steps (rf_pair.cuh): a block has kPairW x kPairRows
// pixels, a warp per row.
constexpr int kPairRows = 4;
constexpr int kPairW = 64;

constexpr int kMaxGridY = 65535;

// rows whose pixel pairs and groups of four are aligned
inline bool pair_stride(int s) { return s % 4 == 0; }

// Whether a level of a single pair takes two pixels per thread.
inline bool use_pairs(int w, int h, int s) {
    // A 720p pair's level 0 (0.92 million pixels, under two waves of blocks, its
    // state in L2) takes as long either way (37.2 against 37.0 ms a solve), a
    // 1080p pair's (2.1 million) is faster by pairs (67.5 against 73.0 ms).
    constexpr long long kMinPixels = 1500000;
    // the one-pixel kernels' blocks have twice the rows, so a level can be too tall
    // for a grid of these alone
    return pair_stride(s) && (long long)w * h >= kMinPixels &&
           (h + kPairRows - 1) / kPairRows <= kMaxGridY;
}

}  // namespace rf
