// Several inner iterations of plain TV-L1 in one launch (solveDataL1.cu:4-91 +
// solveSmoothDualTVGlobal.cu:4-65).
//
// An iteration of plain TV-L1 is about a hundred instructions per pixel, and as
// two launches the launches were what a solve waited for: 1500 of them at 2.3 us
// each for a 640x480 pair (5 levels, 3 warps, 50 iterations), as long at 40x30
// as at 160x120.  Here a block runs up to K iterations on a region in registers:
// 32 columns, one per lane, and R rows per warp.  The data step reads p to the
// left and above, the dual step duhat to the right and below, so each iteration
// uses up one ring of the region: after n <= K iterations all but the n outer
// pixels are right, and a block's tile is its region without K.  Neighbours in a
// row come by shuffles, rows of another warp through shared memory.  A tile's
// ring is other tiles' output, so the state goes from one set of planes to
// another.
//
// Every operation and its order are those of plain_data_px / plain_tv_px, with
// rf_packed.cuh's quotients, u and v as the halves of packed operands (the
// divisor |grad I|^2 of the data step does not change within a warp: its
// reciprocal is formed once per launch).  A guard per thread and half-step covers
// its pixels; where it fails they take IEEE division.  Every value has the same
// bits.
//
// Bound by instruction issue within a block: a launch of four iterations takes
// 5.4 us on small levels (eight launches before: 18) and 17 us at 640x480.  A
// 640x480 pair from 8-bit colour, 3.44 -> 1.49 ms; with 24 x 24 tiles throughout
// 1.72, then with a branch per pixel instead of a guard per thread 1.87, without
// packing 2.1 or more.
#pragma once

#include "rf_ops.cuh"
#include "rf_packed.cuh"

namespace rf {

// the state of the iterations: duhat and the dual field
struct PlainState {
    float *du, *dv, *pu1, *pu2, *pv1, *pv2;
};

namespace {

// one data step at a pixel with IEEE division, out of line
__device__ __noinline__ float2 plain_threshold_slow(f2 du, f2 di, float dit, float lambda,
                                                    float theta) {
    float a, b;
    l1_threshold_plain(du.x, du.y, di.x, di.y, dit, lambda, theta, a, b);
    return make_float2(a, b);
}
__device__ __noinline__ float2 plain_dual_slow(float dx, float dy, float fac, float p1, float p2) {
    dual_step(dx, dy, fac, p1, p2);
    return make_float2(p1, p2);
}

// What the data step of a pixel needs of its image derivatives; the operands
// of the packed instructions are the two components (u, v).
struct PlainPx {
    f2 di;          // (Ix, Iy)
    float dit, magi, nr;
};
// l1_threshold_plain (solveDataL1.cu:27-51): duhat after its step, if `g`
// holds.  The three branches are one addition: of -(rho grad I / |grad I|^2),
// lambda theta grad I, its negative, or -0 where there is no step.
__device__ __forceinline__ f2 plain_threshold(const PlainPx& c, f2 du, float lt, QuotientGuard& g) {
    const f2 m = c.di * du;
    const float rho = m.x + m.y + c.dit;
    const float upper = lt * c.magi;
    const bool in = rho <= upper && rho >= -upper;
    const f2 q = neg_quot<f2>(dup2(rho) * c.di, dup2(c.magi), dup2(c.nr));
    const f2 ld = dup2(rho < -upper ? lt : -lt) * c.di;
    f2 step = in ? q : ld;
    if (in && c.magi == 0.0f) step = dup2(-0.0f);
    g.at_most(f2{rho, upper});
    g.quot(step);
    g.at_most(step.x + step.y);  // a NaN in one of the two shows in their sum
    return du + step;
}

// dual_step of u's and v's fields (fac >= 0), if `g` holds; n1, n2 are their
// negatives (neg_quot's results; x - y for x + (-y) is the same operation)
__device__ __forceinline__ void plain_dual(f2 dx, f2 dy, float fac, f2& n1, f2& n2,
                                           QuotientGuard& g) {
    const f2 mag = sqrt_rn(dx * dx + dy * dy);
    const f2 den = dup2(1.0f) + dup2(fac) * mag;
    const f2 nr = neg_recip(den);
    n1 = neg_quot(dup2(fac) * dx - n1, den, nr);
    n2 = neg_quot(dup2(fac) * dy - n2, den, nr);
    g.quot(mag);
    g.at_most(den);
    g.quot(n1);
    g.quot(n2);
    g.at_most(n1 + n2);  // a NaN in one of them shows in the sum
}
__device__ __forceinline__ void plain_dual_slow2(f2 dx, f2 dy, float fac, f2& n1, f2& n2) {
    const float2 a = plain_dual_slow(dx.x, dy.x, fac, -n1.x, -n2.x);
    const float2 b = plain_dual_slow(dx.y, dy.y, fac, -n1.y, -n2.y);
    n1 = f2{-a.x, -b.x};
    n2 = f2{-a.y, -b.y};
}

__device__ __forceinline__ f2 shfl_up1(f2 a) {
    return f2{__shfl_up_sync(0xFFFFFFFFu, a.x, 1), __shfl_up_sync(0xFFFFFFFFu, a.y, 1)};
}
__device__ __forceinline__ f2 shfl_down1(f2 a) {
    return f2{__shfl_down_sync(0xFFFFFFFFu, a.x, 1), __shfl_down_sync(0xFFFFFFFFu, a.y, 1)};
}

// R rows per warp, WARPS warps, up to K iterations: tile of (32 - 2K) x
// (R WARPS - 2K) pixels
template <int R, int WARPS, int K>
struct PlainTile {
    static constexpr int ROWS = R * WARPS, W = 32 - 2 * K, H = ROWS - 2 * K, THREADS = 32 * WARPS;
};

// `n` iterations; `first`: the state before them is zero; `last`: only duhat is
// written (the next warp's dual field starts from zero).  SKIP: warps whose rows
// are used up or outside the level sit out (64x48 solve 0.90 -> 0.81 ms with 20
// warps of a row; with two rows per warp the branches cost registers and more
// time than they save: 1.49 -> 1.67 ms at 640x480).
template <int R, int WARPS, int K, bool SKIP>
__global__ void __launch_bounds__(32 * WARPS)
    k_plain_tile(PlainState in, PlainState out, const float* __restrict__ Ix,
                 const float* __restrict__ Iy, const float* __restrict__ Iz, PlainWeights wt,
                 LevelDims d, int n, int first, int last) {
    using T = PlainTile<R, WARPS, K>;
    __shared__ f2 s_n2[WARPS][32];  // a warp's last row of n2
    __shared__ f2 s_du[WARPS][32];  // its first row of duhat
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int x = (int)blockIdx.x * T::W - K + lane;
    const int y0 = (int)blockIdx.y * T::H - K + warp * R;
    const int first_row = warp * R;
    const bool any_y = y0 < d.h && y0 + R > 0;
    const bool in_x = x >= 0 && x < d.w;
    const long long end = (long long)d.s * d.h;  // of the level's planes
    const int above = warp > 0 ? warp - 1 : 0, below = warp < WARPS - 1 ? warp + 1 : warp;

    PlainPx c[R];
    f2 du[R], n1[R], n2[R];  // duhat, minus the dual field
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int y = y0 + r;
        c[r].di = dup2(0.0f);
        c[r].dit = 0.0f;
        if (in_x && y >= 0 && y < d.h) {
            const int pos = x + y * d.s;
            c[r].di = f2{RF_PT(Ix, pos, end), RF_PT(Iy, pos, end)};
            c[r].dit = RF_PT(Iz, pos, end);
        }
        const float m = c[r].di.x * c[r].di.x + c[r].di.y * c[r].di.y;
        c[r].magi = m;
        c[r].nr = m >= 0x1p-50f && m <= 0x1p120f ? neg_recip(m) : __uint_as_float(0x7FC00000u);
    }
    // the derivatives do not change between the launches of a warp: they are read while
    // the launch before drains; then the next one may start likewise
    pdl_wait();
    pdl_release();
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int y = y0 + r;
        du[r] = dup2(0.0f);
        n1[r] = n2[r] = dup2(-0.0f);
        if (!first && in_x && y >= 0 && y < d.h) {
            const int pos = x + y * d.s;
            du[r] = f2{RF_PT(in.du, pos, end), RF_PT(in.dv, pos, end)};
            n1[r] = f2{RF_PT(in.pu1, pos, end), RF_PT(in.pv1, pos, end)};
            n2[r] = f2{RF_PT(in.pu2, pos, end), RF_PT(in.pv2, pos, end)};
        }
    }
    s_n2[warp][lane] = n2[R - 1];
    __syncthreads();

    const float lt = wt.lambda * wt.theta;
#pragma unroll 1
    for (int it = 0; it < n; it++) {
        // warps with a row that is right after the half-step and in the level
        const bool data = !SKIP || (first_row + R > it + 1 && first_row < T::ROWS - it && any_y);
        const bool dual = !SKIP || (first_row + R > it + 1 && first_row < T::ROWS - 1 - it && any_y);
        if (data) {
            f2 up = s_n2[above][lane], t[R];
            QuotientGuard g;
#pragma unroll
            for (int r = 0; r < R; r++) t[r] = plain_threshold(c[r], du[r], lt, g);
            if (!g.ok()) {
#pragma unroll
                for (int r = 0; r < R; r++) {
                    const float2 e = plain_threshold_slow(du[r], c[r].di, c[r].dit, wt.lambda, wt.theta);
                    t[r] = f2{e.x, e.y};
                }
            }
#pragma unroll
            for (int r = 0; r < R; r++) {
                f2 left = shfl_up1(n1[r]);
                // (no neighbour: minus zero, which changes nothing)
                if (x == 0) left = dup2(-0.0f);
                if (y0 + r == 0) up = dup2(-0.0f);
                // divergence (solveDataL1.cu:54-85) of the negatives
                const f2 div = left - n1[r] - n2[r] + up;
                up = n2[r];
                du[r] = t[r] + dup2(wt.theta) * div;
            }
            s_du[warp][lane] = du[0];
        }
        __syncthreads();
        if (dual) {
            const f2 down = s_du[below][lane];
            f2 dx[R], dy[R], m1[R], m2[R];
            QuotientGuard gd;
#pragma unroll
            for (int r = 0; r < R; r++) {
                dx[r] = shfl_down1(du[r]) - du[r];
                dy[r] = (r < R - 1 ? du[r < R - 1 ? r + 1 : r] : down) - du[r];
                if (x + 1 >= d.w) dx[r] = dup2(0.0f);
                if (y0 + r + 1 >= d.h) dy[r] = dup2(0.0f);
                m1[r] = n1[r];
                m2[r] = n2[r];
                plain_dual(dx[r], dy[r], wt.fac, m1[r], m2[r], gd);
            }
            if (gd.ok()) {
#pragma unroll
                for (int r = 0; r < R; r++) {
                    n1[r] = m1[r];
                    n2[r] = m2[r];
                }
            } else {
#pragma unroll
                for (int r = 0; r < R; r++) plain_dual_slow2(dx[r], dy[r], wt.fac, n1[r], n2[r]);
            }
        }
        s_n2[warp][lane] = n2[R - 1];
        __syncthreads();
    }

    if (lane < K || lane >= 32 - K || !in_x) return;
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int row = warp * R + r, y = y0 + r;
        if (row < K || row >= R * WARPS - K || y >= d.h) continue;
        const int pos = x + y * d.s;
        RF_PT(out.du, pos, end) = du[r].x;
        RF_PT(out.dv, pos, end) = du[r].y;
        if (!last) {
            RF_PT(out.pu1, pos, end) = n1[r].x;
            RF_PT(out.pv1, pos, end) = n1[r].y;
            RF_PT(out.pu2, pos, end) = n2[r].x;
            RF_PT(out.pv2, pos, end) = n2[r].y;
        }
    }
}

}  // namespace
}  // namespace rf
