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
    // A 1080p pair's level 0 (2.1 million pixels) is faster by pairs: 59.6 against
    // 68.9 ms a solve (6 levels, 5 x 100 iterations). The gain ends below: a 720p
    // pair's (0.92 million, under two waves of blocks, its state in L2) would take
    // 29.6 against 30.2.
    constexpr long long kMinPixels = 1500000;
    // the one-pixel kernels' blocks have twice the rows, so a level can be too tall
    // for a grid of these alone
    return pair_stride(s) && (long long)w * h >= kMinPixels &&
           (h + kPairRows - 1) / kPairRows <= kMaxGridY;
}

// A region of k_recon_tile (rf_tile.cuh): kTileW columns of `rows` rows, less two rings
// per iteration.
constexpr int kTileW = 32;
constexpr long long recon_tile_blocks(int w, int h, int rows, int k) {
    const int tw = kTileW - 4 * k, th = rows - 4 * k;
    return (long long)((w + tw - 1) / tw) * ((h + th - 1) / th);
}

// Which tile a level takes on a device of `sms` multiprocessors, 0 for none: the first
// of those below with no more than a block per SM.
inline int recon_tile_kind(int w, int h, int sms) {
    // An iteration of a block is bound by the instructions of its warps, so the
    // smallest tile is the fastest while every block has an SM to itself; two
    // blocks on one take twice as long.  Solves on 152 SMs, the level in question
    // with its tile and the next: 80x60 with 24 x 2 and 24 x 4: 2.55 and 2.66 ms
    // (of a 160x120 solve, 5 x 100); 112x83 with 24 x 4 and 20 x 8: 2.85 and 2.93
    // (451x333, 3 x 50); 160x120 with 20 x 8, three iterations, and 24 x 12, two:
    // 2.55 and 2.79; 225x166 with 24 x 12 and with two launches per iteration: 2.85
    // and 3.15.  320x240, 280 blocks of 24 x 12, is faster by two launches per
    // iteration (4.30 against 4.44, 640x480).
    if (recon_tile_blocks(w, h, 10, 2) <= sms) return 1;
    if (recon_tile_blocks(w, h, 12, 2) <= sms) return 2;
    if (recon_tile_blocks(w, h, 20, 3) <= sms) return 3;
    if (recon_tile_blocks(w, h, 20, 2) <= sms) return 4;
    return 0;
}

// Whether a direct convolution over `npos` positions takes 256 of them per block
// (`smem`: its shared memory then) rather than 128: where every SM gets one and two fit
// on it.  The larger tile loads the weights and the two rows around it half as often
// (64 images of 160 x 90: 0.53 ms against 0.65, eight 0.133 and 0.143); with too few
// of them SMs idle (one image: the same either way).
inline bool conv_wide_tile(long long npos, unsigned long long smem, int sms) {
    return npos >= 256ll * sms && smem <= 113 * 1024;
}

}  // namespace rf
