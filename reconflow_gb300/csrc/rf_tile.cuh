// Several inner iterations of ReconFlow in one launch, for small levels.
//
// A level of 80x60 takes as long per launch as one of 320x240: the two launches
// of an iteration, their round trips to memory and their longest thread, 5.6 us.
// Here a block keeps a region's state in registers, 32 columns (a lane each) by
// ROWS rows (a warp each), and runs up to K iterations on it.  A reads p and the
// points one pixel around, B duhat and the triangulated points one pixel around,
// through shared memory and shuffles, so that each iteration uses up two rings
// of the region and the block's tile is what is left after K; rows in a ring that
// is used up sit out.  A tile's ring is other tiles' output: the state goes from
// one set of planes to another and, after an even number of launches, is back.
//
// x + 1 of a row's last pixel and y + 1 of the last row are read at flat pos + 1
// and pos + s (solve3dMinimalArea.cu:65,76): padding, the row below the level, or,
// where rows have no padding, the next row's first pixel.  The first two are
// elements that no iteration changes, held by lanes of the region; for the third
// the lanes right of the level hold the first pixels of the next row and iterate
// them along.
//
// The arithmetic is that of the one-pixel half-steps (rf_pair.cuh): same bits.
// Bound by a block's instruction issue (about 1000 per pixel and iteration):
// 3 to 3.5 us per iteration, 5.2 to 6 by two launches.  Plain 640x480 pair 6.05 ->
// 4.79 ms, 1280x720 35.2 -> 31.3, 451x333 with a prior 4.55 -> 3.44.  With the next
// launch's blocks coming in while one runs (programmatic launches) 640x480 4.72 -> 4.58
// and the prior's 3.32 -> 3.22: there a launch has SMs to spare.
#pragma once

#include "rf_pair.cuh"
#include "rf_rules.h"

namespace rf {

// The state the iterations carry from launch to launch.
struct ReconState {
    float *duhat, *dvhat, *pu1, *pu2, *pv1, *pv2, *uproj, *vproj, *sku, *skv, *X, *Y, *Z;
};

namespace {

// what a block's threads show each other: p for part A, the points for A and
// (their triangulated form) for B, duhat for B; a ring around each
template <int ROWS>
struct TileShared {
    float pu2[ROWS][kTileW], pv2[ROWS][kTileW], du[ROWS][kTileW], dv[ROWS][kTileW];
    float X[3][ROWS + 2][kTileW + 2], X1[3][ROWS + 2][kTileW + 2];
    LevelConsts lc;
};

template <int ROWS>
__device__ __forceinline__ void tile_around(const float (&s)[ROWS + 2][kTileW + 2], int row,
                                            int lane, bool left, bool up, float own,
                                            float (&n)[5]) {
    n[0] = own;
    n[1] = s[row + 1][lane + 2];
    n[2] = s[row + 2][lane + 1];
    n[3] = left ? s[row + 1][lane] : 0.0f;
    n[4] = up ? s[row][lane + 1] : 0.0f;
}
// load_taps_one from a region
template <int ROWS>
__device__ __forceinline__ void tile_taps(const float (&s)[ROWS + 2][kTileW + 2], int row, int lane,
                                          PairEdges e, float (&t)[3][3]) {
#pragma unroll
    for (int j = 0; j < 3; j++) {
        const float* q = &s[row + j + (j == 0 && !e.up ? 1 : 0)][lane + 1];
        const bool in = j != 2 || e.down;
        t[j][0] = !in ? 0.0f : (e.left ? q[-1] : (j != 0 || e.up ? q[0] : 0.0f));
        t[j][1] = in ? q[0] : 0.0f;
        t[j][2] = in && e.both ? q[1] : 0.0f;
    }
}

template <int ROWS_, int K>
struct ReconTile {
    static constexpr int RING = 2 * K, W = kTileW - 2 * RING, H = ROWS_ - 2 * RING;
    static constexpr int THREADS = kTileW * ROWS_;
};

// A's arithmetic with IEEE division, out of line
template <int PRIOR>
__device__ __noinline__ void recon_a_point_slow(APoint& a, const LevelConsts& c, const Weights& wt,
                                                int x, int y, bool first, bool uc_from_buffer) {
    recon_a_point<PRIOR, true>(a, c, wt, x, y, first, uc_from_buffer);
}

// `n` <= K iterations; `first_launch`: duhat and p before them are zero;
// `last_launch`: the last of them makes the multiplier update and leaves the dual
// update out, as recon_b_one<true>.  in and out are f's state and another one;
// `uc_from_buffer` goes with the first launch.
template <int PRIOR, int ROWS, int K>
__global__ void __launch_bounds__(kTileW* ROWS)
    k_recon_tile(const __grid_constant__ ReconFields f, const __grid_constant__ ReconState in,
                 const __grid_constant__ ReconState out, const LevelConsts* __restrict__ lcp,
                 const __grid_constant__ Weights wt, LevelDims d, int n, int first_launch,
                 int last_launch, int uc_from_buffer) {
    __shared__ TileShared<ROWS> sm;
    const int lane = threadIdx.x & 31, row = threadIdx.x >> 5;
    using T = ReconTile<ROWS, K>;
    constexpr int RING = T::RING;
    const int tx = (int)blockIdx.x * T::W - RING + lane;
    const int ty = (int)blockIdx.y * T::H - RING + row;
    // the pixel of a lane right of the level, as x + 1 finds it in memory
    const bool wrapped = tx >= d.w && d.s == d.w;
    const int x = wrapped ? tx - d.w : tx, y = wrapped ? ty + 1 : ty;
    const bool near = !wrapped || x < RING;
    const bool pixel = near && x >= 0 && x < d.w && y >= 0 && y < d.h;
    // elements that only A's points read: the row below the level, the column
    // right of it where rows are padded
    const bool still = near && ((y == d.h && x >= 0 && x < d.w) || (x == d.w && y >= 0 && y < d.h));
    const int pos = x + y * d.s;
    const PairEdges e{x > 0, x + 1 < d.w, x + 1 < d.w, y > 0, y + 1 < d.h};

    if (threadIdx.x < sizeof(LevelConsts) / sizeof(float))
        reinterpret_cast<float*>(&sm.lc)[threadIdx.x] =
            reinterpret_cast<const float*>(lcp)[threadIdx.x];
    float u = 0.0f, v = 0.0f, dix = 0.0f, diy = 0.0f, dit = 0.0f, ufn = 0.0f, vfn = 0.0f, mk = 1.0f;
    float duhat = 0.0f, dvhat = 0.0f, uproj = 0.0f, vproj = 0.0f, sku = 0.0f, skv = 0.0f;
    float p[4] = {0.0f, 0.0f, 0.0f, 0.0f};  // pu1, pu2, pv1, pv2
    float X = 0.0f, Y = 0.0f, Z = 0.0f, uc = 0.0f, vc = 0.0f;
    if (pixel) {
        u = RF_AT(f, u, pos);
        v = RF_AT(f, v, pos);
        dix = RF_AT(f, Ix, pos);
        diy = RF_AT(f, Iy, pos);
        dit = RF_AT(f, Iz, pos);
        if (PRIOR != 0) {
            ufn = RF_AT(f, ufn, pos);
            vfn = RF_AT(f, vfn, pos);
            if (PRIOR == 2) mk = RF_AT(f, mask, pos);
        }
    }
    // what comes before this does not change between the launches of a warp, so it is
    // read while the launch before drains; then the next one may start likewise
    pdl_wait();
    pdl_release();
    if (pixel) {
        uproj = RF_PT(in.uproj, pos, f.extent);
        vproj = RF_PT(in.vproj, pos, f.extent);
        sku = RF_PT(in.sku, pos, f.extent);
        skv = RF_PT(in.skv, pos, f.extent);
        X = RF_PT(in.X, pos, f.extent);
        Y = RF_PT(in.Y, pos, f.extent);
        Z = RF_PT(in.Z, pos, f.extent);
        if (!first_launch) {
            duhat = RF_PT(in.duhat, pos, f.extent);
            dvhat = RF_PT(in.dvhat, pos, f.extent);
            p[0] = RF_PT(in.pu1, pos, f.extent);
            p[1] = RF_PT(in.pu2, pos, f.extent);
            p[2] = RF_PT(in.pv1, pos, f.extent);
            p[3] = RF_PT(in.pv2, pos, f.extent);
        }
        if (uc_from_buffer) {
            uc = RF_AT(f, uc, pos);
            vc = RF_AT(f, vc, pos);
        }
    } else if (still) {
        X = RF_AT(f, X, pos);
        Y = RF_AT(f, Y, pos);
        Z = RF_AT(f, Z, pos);
    }

    // the ring around the region: the nearest element's points, so that the outer
    // pixels, which are computed but not used, meet no odd values
    {
        const int r = row == 0 ? 0 : row == ROWS - 1 ? ROWS + 1 : row + 1;
        const int l = lane == 0 ? 0 : lane == kTileW - 1 ? kTileW + 1 : lane + 1;
        const float q[3] = {X, Y, Z};
        for (int c = 0; c < 3; c++) {
            sm.X[c][r][l] = sm.X[c][row + 1][l] = sm.X[c][r][lane + 1] = q[c];
            sm.X1[c][r][l] = sm.X1[c][row + 1][l] = sm.X1[c][r][lane + 1] = q[c];
        }
    }

#pragma unroll 1
    for (int it = 0; it < n; it++) {
        const bool first = first_launch && it == 0, last = last_launch && it + 1 == n;
        const bool ucb = uc_from_buffer && it == 0;
        sm.pu2[row][lane] = p[1];
        sm.pv2[row][lane] = p[3];
        sm.X[0][row + 1][lane + 1] = X;
        sm.X[1][row + 1][lane + 1] = Y;
        sm.X[2][row + 1][lane + 1] = Z;
        const float pu1l = __shfl_up_sync(0xFFFFFFFFu, p[0], 1);
        const float pv1l = __shfl_up_sync(0xFFFFFFFFu, p[2], 1);
        __syncthreads();
        // the rows that are right after this half-step
        const bool useful_a = row > 2 * it && row < ROWS - 1 - 2 * it;
        const bool useful_b = row > 2 * it + 1 && row < ROWS - 2 - 2 * it;
        if (pixel && useful_a) {
            const int above = row > 0 ? row - 1 : 0;
            auto load = [&](APoint& a) {
                a.u = u;
                a.v = v;
                a.dix = dix;
                a.diy = diy;
                a.dit = dit;
                a.uproj = uproj;
                a.vproj = vproj;
                a.sku = sku;
                a.skv = skv;
                a.duhat = duhat;
                a.dvhat = dvhat;
                a.pu1 = p[0];
                a.pu2 = p[1];
                a.pv1 = p[2];
                a.pv2 = p[3];
                a.pu1l = e.left ? pu1l : 0.0f;
                a.pv1l = e.left ? pv1l : 0.0f;
                a.pu2d = e.up ? sm.pu2[above][lane] : 0.0f;
                a.pv2d = e.up ? sm.pv2[above][lane] : 0.0f;
                tile_around<ROWS>(sm.X[0], row, lane, e.left, e.up, X, a.Xn);
                tile_around<ROWS>(sm.X[1], row, lane, e.left, e.up, Y, a.Yn);
                tile_around<ROWS>(sm.X[2], row, lane, e.left, e.up, Z, a.Zn);
                a.uc = uc;
                a.vc = vc;
                a.ufn = ufn;
                a.vfn = vfn;
                a.mk = mk;
            };
            APoint a;
            load(a);
            bool ok = recon_a_fast<PRIOR>(a, sm.lc, wt, x, y, first, ucb);
            if (!ok) {
                APoint b;
                load(b);
                recon_a_point_slow<PRIOR>(b, sm.lc, wt, x, y, first, ucb);
                a.sku = b.sku;
                a.skv = b.skv;
                a.duhat = b.duhat;
                a.dvhat = b.dvhat;
                a.uproj = b.uproj;
                a.vproj = b.vproj;
                a.Xo = b.Xo;
                a.Yo = b.Yo;
                a.Zo = b.Zo;
            }
            sku = a.sku;
            skv = a.skv;
            duhat = a.duhat;
            dvhat = a.dvhat;
            uproj = a.uproj;
            vproj = a.vproj;
            sm.X1[0][row + 1][lane + 1] = a.Xo;
            sm.X1[1][row + 1][lane + 1] = a.Yo;
            sm.X1[2][row + 1][lane + 1] = a.Zo;
            sm.du[row][lane] = duhat;
            sm.dv[row][lane] = dvhat;
        }
        __syncthreads();
        const float dur = __shfl_down_sync(0xFFFFFFFFu, duhat, 1);
        const float dvr = __shfl_down_sync(0xFFFFFFFFu, dvhat, 1);
        if (pixel && useful_b) {
            float t[3][3][3];
            tile_taps<ROWS>(sm.X1[0], row, lane, e, t[0]);
            tile_taps<ROWS>(sm.X1[1], row, lane, e, t[1]);
            tile_taps<ROWS>(sm.X1[2], row, lane, e, t[2]);
            point_one(t[0], t[1], t[2], X, Y, Z);
            if (last) {
                sku = sku + u + duhat - uproj;
                skv = skv + v + dvhat - vproj;
            } else {
                const int below = row < ROWS - 1 ? row + 1 : row;
                const float ux = e.both ? dur - duhat : 0.0f, vx = e.both ? dvr - dvhat : 0.0f;
                const float uy = e.down ? sm.du[below][lane] - duhat : 0.0f;
                const float vy = e.down ? sm.dv[below][lane] - dvhat : 0.0f;
                dual_one(ux, uy, vx, vy, wt.fac, p);
            }
        }
    }

    if (!pixel || wrapped || lane < RING || lane >= kTileW - RING || row < RING ||
        row >= ROWS - RING)
        return;
    RF_PT(out.duhat, pos, f.extent) = duhat;
    RF_PT(out.dvhat, pos, f.extent) = dvhat;
    RF_PT(out.uproj, pos, f.extent) = uproj;
    RF_PT(out.vproj, pos, f.extent) = vproj;
    RF_PT(out.sku, pos, f.extent) = sku;
    RF_PT(out.skv, pos, f.extent) = skv;
    RF_PT(out.X, pos, f.extent) = X;
    RF_PT(out.Y, pos, f.extent) = Y;
    RF_PT(out.Z, pos, f.extent) = Z;
    if (!last_launch) {
        RF_PT(out.pu1, pos, f.extent) = p[0];
        RF_PT(out.pu2, pos, f.extent) = p[1];
        RF_PT(out.pv1, pos, f.extent) = p[2];
        RF_PT(out.pv2, pos, f.extent) = p[3];
    }
}

}  // namespace
}  // namespace rf
