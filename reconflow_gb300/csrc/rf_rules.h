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
    // blocks on one take twice as long.  Solves of 96x72 .. 640x480, the level in
    // question with one tile and the next larger: 80x60 with 24 x 2 (10 rows) and
    // 24 x 8 (16): 2.44 and 2.56 ms (of a 160x120 solve); 112x83 with 24 x 4 and
    // 20 x 8: 3.74 and 3.82 (451x333); 160x120 with 20 x 8, three iterations, and
    // 24 x 12, two: 2.42 and 2.51; 225x166 with 24 x 12 and with two launches per
    // iteration: 3.52 and 3.75.  320x240, 280 blocks of 24 x 12, is as fast by two
    // launches per iteration (4.95 against 5.01, 640x480).
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
