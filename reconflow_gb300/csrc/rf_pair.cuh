// The two half-steps of a ReconFlow inner iteration, one or two pixels per
// thread.
//
// A (data term, projection blend, point solve: recon_a_px) and B (dual
// update, 3x3 median and clean-up of the points, multiplier update:
// recon_b_px) were bound by instruction issue on large levels (732 and 451 warp
// instructions per 32 pixels) and by the length of a pixel's chain of
// instructions on small ones.
// * Quotients and roots are rf_packed.cuh's: IEEE division's own sequence,
//   with its check and branch, was a third of A's instructions.  A guard per
//   thread covers all of them; where it fails the thread takes IEEE division.
// * With camera 0 at the origin most products of the normal matrix are zeros
//   and are not formed.
// * The multiplier update moves from B to the next iteration's A, which reads
//   all its operands anyway (sk, u, duhat and uproj before A replaces them): B
//   then reads 9 planes and writes 7 instead of 15 and 9, and an iteration moves
//   172 bytes per pixel instead of 196.  The last B of a warp makes the update
//   itself, and leaves the dual update out: the next warp's dual field starts
//   from zero and nothing else reads it.
// * Large levels run two pixels (x, x + 1), x even, per thread, as the two
//   halves of packed FP32 instructions, loaded and stored as 64-bit vectors.
//
// Every operation and its order are those of recon_a_px / recon_b_px, so every
// value has the same bits.  Needs ordinary weights (pair_weights), pixel pairs
// a row stride that is a multiple of four (pair_stride); other weights run
// recon_a_px / recon_b_px.
#pragma once

#include <cstddef>

#include "rf_ops.cuh"
#include "rf_packed.cuh"
#include "rf_rules.h"

namespace rf {

namespace {

// elements i, i + 1 of a field (i even)
#ifdef RF_BOUNDS_CHECK
#define RF_LD2(f, name, i) mk2(RF_AT(f, name, i), RF_AT(f, name, (i) + 1))
__device__ __forceinline__ float2 ld2_at(const float* p, long long i, long long n) {
    return make_float2(rf_checked(p, i, n), rf_checked(p, i + 1, n));
}
#else
__device__ __forceinline__ f2 ld2(const float* p) {
    const float2 t = *reinterpret_cast<const float2*>(p);
    return f2{t.x, t.y};
}
#define RF_LD2(f, name, i) ld2((f).name + (i))
__device__ __forceinline__ float2 ld2_at(const float* p, int i, long long) {
    return *reinterpret_cast<const float2*>(p + i);
}
#endif
#ifdef RF_BOUNDS_CHECK
#define RF_ST2(f, name, i, v, both)                   \
    do {                                              \
        const f2 v__ = (v);                           \
        RF_AT(f, name, i) = v__.x;                    \
        if (both) RF_AT(f, name, (i) + 1) = v__.y;    \
    } while (0)
#else
#define RF_ST2(f, name, i, v, both)                                              \
    do {                                                                         \
        const f2 v__ = (v);                                                      \
        float* p__ = (f).name + (i);                                             \
        if (both) *reinterpret_cast<float2*>(p__) = make_float2(v__.x, v__.y);   \
        else *p__ = v__.x;                                                       \
    } while (0)
#endif

// ---- staging ---------------------------------------------------------------
// A block has a tile of kPairW x kPairRows pixels, a warp per row.  B copies
// all it reads to shared memory first, asynchronously and 16 bytes at a time
// (its taps would be 27 loads per pair and 36 registers: 64 registers and 42%
// occupancy with direct loads, 48 and 57% with copies, 0.95 -> 0.79 ms per 59
// million pixels).  Column 0 of the tile is at column 4 of a row in shared
// memory, so that every copy is aligned.
constexpr int kPitch = kPairW + 8;

// the fields A reads, as ReconFields has them in a row: u, v, duhat, dvhat,
// pu1, pu2, pv1, pv2, uproj, vproj, sku, skv, Ix, Iy, Iz, X, Y, Z
constexpr int kReconReads = 18;
__device__ __forceinline__ const float* recon_read(const ReconFields& f, int i) {
    return reinterpret_cast<const float* const*>(&f)[i];
}
static_assert(offsetof(ReconFields, X1) == kReconReads * sizeof(float*), "field order");

__device__ __forceinline__ void copy16(float* to, const float* from, int i, long long n) {
#ifdef RF_BOUNDS_CHECK
    for (int k = 0; k < 4; k++) to[k] = rf_checked(from, (long long)i + k, n);
#else
    (void)n;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(
                     (unsigned)__cvta_generic_to_shared(to)),
                 "l"(from + i)
                 : "memory");
#endif
}
__device__ __forceinline__ void copies_done() {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
}
__device__ __forceinline__ f2 lds2(const float* p) {
    const float2 t = *reinterpret_cast<const float2*>(p);
    return f2{t.x, t.y};
}

// minima and maxima that hand a NaN on (of two and of three values: one
// instruction each)
__device__ __forceinline__ float nmin(float a, float b) {
    float r;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float nmax(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float nmin3(float a, float b, float c) {
    float r;
    asm("min.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float nmax3(float a, float b, float c) {
    float r;
    asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
// the middle one of three
__device__ __forceinline__ float nmed3(float a, float b, float c) {
    return nmax(nmin(a, b), nmin(nmax(a, b), c));
}

// median9_finite of a window whose median is a zero (the exchange order
// decides its sign) or that holds a NaN; out of line, on the taps in registers
// (re-reading them lengthened the longest thread of a small level's launch)
__device__ __noinline__ float median9_slow(float a, float b, float c, float d, float e, float f,
                                           float g, float h, float i) {
    const float m[9] = {a, b, c, d, e, f, g, h, i};
    // zeros of one sign only (points set to the origin are +0): that zero
    bool nan = false, pos = false, neg = false;
#pragma unroll
    for (int k = 0; k < 9; k++) {
        const unsigned bits = __float_as_uint(m[k]);
        nan |= isnan(m[k]);
        pos |= bits == 0u;
        neg |= bits == 0x80000000u;
    }
    if (!nan && !(pos && neg)) return neg ? -0.0f : 0.0f;
    return median9_finite(m);
}
template <int N>
__device__ __forceinline__ float median9_slow(const float (&t)[3][N], int i) {
    return median9_slow(t[0][i], t[0][i + 1], t[0][i + 2], t[1][i], t[1][i + 1], t[1][i + 2],
                        t[2][i], t[2][i + 1], t[2][i + 2]);
}

// Where a pair's 3x3 windows lie in its level.
struct PairEdges {
    bool left, right, both, up, down;  // x > 0; x + 2 < w; x + 1 < w; y > 0; y + 1 < h
};
__device__ __forceinline__ PairEdges pair_edges(int x, int y, LevelDims d) {
    return PairEdges{x > 0, x + 2 < d.w, x + 1 < d.w, y > 0, y + 1 < d.h};
}

// The taps of the 3x3 windows of (x, y) and (x + 1, y) (`p`: their place in a
// staged plane), with the reference's border rules (median3_tap: left and top
// taps take the nearest pixel, right, bottom and corner taps are 0); columns
// 1 and 2 of row 1 are the pixels.
__device__ __forceinline__ void load_taps(const float* p, PairEdges e, float (&t)[3][4]) {
#pragma unroll
    for (int j = 0; j < 3; j++) {
        // the row above the level takes row 0's pixels (not at its corners)
        const float* q = j == 0 ? (e.up ? p - kPitch : p) : p + (j - 1) * kPitch;
        const f2 c = lds2(q);
        const float l = q[-1], r = q[2];
        const bool in = j != 2 || e.down;
        t[j][0] = e.left ? l : (j != 0 || e.up ? c.x : 0.0f);
        t[j][1] = c.x;
        t[j][2] = e.both ? c.y : 0.0f;
        t[j][3] = e.right ? r : 0.0f;
        if (!in) t[j][0] = t[j][1] = t[j][2] = t[j][3] = 0.0f;
    }
}

// The two windows' medians (median9_finite's values, except that a NaN is
// handed on and a zero may have the other sign).  A column of three taps
// belongs to up to three windows: its smallest, middle and largest tap are
// found once, and a window's median is the middle one of (largest of the
// smallest, middle of the middle, smallest of the largest).
__device__ __forceinline__ f2 median3_pair(const float (&t)[3][4]) {
    float lo[4], mid[4], hi[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float s = nmin(t[0][i], t[1][i]), g = nmax(t[0][i], t[1][i]);
        lo[i] = nmin(s, t[2][i]);
        hi[i] = nmax(g, t[2][i]);
        mid[i] = nmax(s, nmin(g, t[2][i]));
    }
    f2 m;
    m.x = nmed3(nmax3(lo[0], lo[1], lo[2]), nmed3(mid[0], mid[1], mid[2]),
                nmin3(hi[0], hi[1], hi[2]));
    m.y = nmed3(nmax3(lo[1], lo[2], lo[3]), nmed3(mid[1], mid[2], mid[3]),
                nmin3(hi[1], hi[2], hi[3]));
    return m;
}

// The points of B at (x, y), (x + 1, y): medians of X1, Y1, Z1 and clean-up.
struct PointTaps {
    float x[3][4], y[3][4], z[3][4];
};
__device__ __forceinline__ void points_pair(PairEdges e, const PointTaps& t, f2& X, f2& Y,
                                            f2& Z) {
    const float(&tx)[3][4] = t.x, (&ty)[3][4] = t.y, (&tz)[3][4] = t.z;
    f2 Xm = median3_pair(tx), Ym = median3_pair(ty), Zm = median3_pair(tz);
    auto sure = [](float m) { return fabsf(m) > 0.0f; };  // neither zero nor NaN
    if (!(sure(Xm.x) && sure(Ym.x) && sure(Zm.x) && sure(Xm.y) && sure(Ym.y) && sure(Zm.y))) {
        if (!sure(Xm.x)) Xm.x = median9_slow(tx, 0);
        if (!sure(Ym.x)) Ym.x = median9_slow(ty, 0);
        if (!sure(Zm.x)) Zm.x = median9_slow(tz, 0);
        if (e.both && !sure(Xm.y)) Xm.y = median9_slow(tx, 1);
        if (e.both && !sure(Ym.y)) Ym.y = median9_slow(ty, 1);
        if (e.both && !sure(Zm.y)) Zm.y = median9_slow(tz, 1);
    }
    cleanup_pixel(tx[1][1], ty[1][1], tz[1][1], Xm.x, Ym.x, Zm.x, X.x, Y.x, Z.x);
    cleanup_pixel(tx[1][2], ty[1][2], tz[1][2], Xm.y, Ym.y, Zm.y, X.y, Y.y, Z.y);
}

// dual_step (solveSmoothDualTVGlobal.cu:46-60; fac >= 0)
template <class V>
__device__ __forceinline__ void dual_step_v(V dx, V dy, float facs, V& p1, V& p2,
                                            QuotientGuard& g) {
    const V fac = splat<V>(facs);
    const V mag = sqrt_rn(dx * dx + dy * dy);
    const V den = splat<V>(1.0f) + fac * mag;
    const V nr = neg_recip(den);
    p1 = -neg_quot(p1 + fac * dx, den, nr);
    p2 = -neg_quot(p2 + fac * dy, den, nr);
    g.quot(mag);
    g.at_most(den);
    g.quot(p1);
    g.quot(p2);
}
// the same with IEEE operations, one pixel; out of line
__device__ __noinline__ float2 dual_step_slow(float dx, float dy, float fac, float p1, float p2) {
    dual_step(dx, dy, fac, p1, p2);
    return make_float2(p1, p2);
}
__device__ __forceinline__ void dual_step_slow2(f2 dx, f2 dy, float fac, f2& p1, f2& p2) {
    const float2 a = dual_step_slow(dx.x, dy.x, fac, p1.x, p2.x);
    const float2 b = dual_step_slow(dx.y, dy.y, fac, p1.y, p2.y);
    p1 = mk2(a.x, b.x);
    p2 = mk2(a.y, b.y);
}

// What the dual update of B at (x, y), (x + 1, y) reads.
struct DualIn {
    f2 u, v, ud, vd, pu1, pu2, pv1, pv2;  // duhat at the pixels and below them, p
    float ur, vr;                         // duhat at x + 2
};
// the dual field after it, in in.p*
__device__ __forceinline__ void dual_update(DualIn& in, float fac, PairEdges e) {
    const f2 zero = mk2(0.0f, 0.0f);
    f2 ux = mk2(in.u.y, in.ur) - in.u, vx = mk2(in.v.y, in.vr) - in.v;
    f2 uy = in.ud - in.u, vy = in.vd - in.v;
    if (!e.both) ux.x = vx.x = 0.0f;
    if (!e.right) ux.y = vx.y = 0.0f;
    if (!e.down) uy = vy = zero;
    QuotientGuard g;
    f2 pu1 = in.pu1, pu2 = in.pu2, pv1 = in.pv1, pv2 = in.pv2;
    dual_step_v(ux, uy, fac, pu1, pu2, g);
    dual_step_v(vx, vy, fac, pv1, pv2, g);
    // (a NaN in one of the four shows in their sum)
    const f2 sum = pu1 + pu2 + pv1 + pv2;
    if (g.ok() && isfinite(sum.x) && isfinite(sum.y)) {
        in.pu1 = pu1;
        in.pu2 = pu2;
        in.pv1 = pv1;
        in.pv2 = pv2;
    } else {
        dual_step_slow2(ux, uy, fac, in.pu1, in.pu2);
        dual_step_slow2(vx, vy, fac, in.pv1, in.pv2);
    }
}

// what a holds for the first pixel (the only one that can be in column 0)
// replaced by b's unless `keep`
__device__ __forceinline__ void first_or(float& a, float b, bool keep) { a = keep ? a : b; }
__device__ __forceinline__ void first_or(f2& a, f2 b, bool keep) { a.x = keep ? a.x : b.x; }

// divergence (solveReconDataL1.cu:66-97)
template <class V>
__device__ __forceinline__ V divergence_v(V p1, V p1l, V p2, V p2d, bool left, bool up) {
    V t = p1 - p1l;
    first_or(t, p1, left);
    t = t + p2;
    const V r = t - p2d;
    return up ? r : t;
}

// The level's constants and the weights by number, a value or an operand of
// two.  For pixel pairs a block has them in shared memory as pairs of equal
// floats, so that one 64-bit read gives a packed operand.
enum {
    kCP = 0, kCQ = 12, kCR = 24, kCt = 33, kCf = 36, kCcx = 37, kCcy = 38, kCtv = 39, kCproj = 40,
    kCA = 41, kCpden = 42, kClf = 43, kClms = 44, kCfn = 45, kCHalf = 46, kClam = 47, kCnrA = 48,
    kCnrP = 49,
    // camera 0 at the origin (P = [f 0 cx 0; 0 g cy 0; 0 0 1 0]): f^2, g^2, and
    // in kCorigin whether it is (LevelConsts::origin)
    kCff = 50, kCgg = 51, kCorigin = 52, kCount = 53
};

struct OneConsts {
    const LevelConsts& c;
    const Weights& wt;
    __device__ __forceinline__ float operator()(int i) const {
        if (i < kCQ) return c.P[i];
        if (i < kCR) return c.Q[i - kCQ];
        if (i < kCt) return c.R1[i - kCR];
        if (i < kCf) return c.t1[i - kCt];
        switch (i) {
            case kCf: return c.focal;
            case kCcx: return c.cx;
            case kCcy: return c.cy;
            case kCtv: return wt.alpha_tv;
            case kCproj: return wt.alpha_proj;
            case kCA: return wt.A;
            case kCpden: return wt.proj_den;
            case kClf: return wt.lambdaf;
            case kClms: return wt.lambdams;
            case kCfn: return wt.alpha_fn;
            case kClam: return wt.lambda;
            case kCnrA: return wt.nrA;
            case kCnrP: return wt.nrP;
            case kCff: return c.P[0] * c.P[0];
            case kCgg: return c.P[5] * c.P[5];
            case kCorigin: return c.origin;
            default: return 0.5f;
        }
    }
    __device__ __forceinline__ bool origin() const { return c.origin != 0.0f; }
};

struct PairConsts {
    const float2* sc;
    __device__ __forceinline__ f2 operator()(int i) const {
        const float2 t = sc[i];
        return f2{t.x, t.y};
    }
    __device__ __forceinline__ bool origin() const { return sc[kCorigin].x != 0.0f; }
};

__device__ __forceinline__ void pair_consts(const LevelConsts* __restrict__ lc, const Weights& wt,
                                            float2* sc, int tid, int nthr) {
    const OneConsts c{*lc, wt};
    for (int i = tid; i < kCount; i += nthr) {
        const float v = i < kCtv ? reinterpret_cast<const float*>(lc)[i] : c(i);
        sc[i] = make_float2(v, v);
    }
}

// project_uc (solveUcSk.cu:21-33)
template <class V, class C>
__device__ __forceinline__ void project_uc_v(const C& c, V X, V Y, V Z, V fx, V fy, V& uc, V& vc,
                                             QuotientGuard& g) {
    const V X2 = c(kCR + 0) * X + c(kCR + 1) * Y + c(kCR + 2) * Z + c(kCt + 0);
    const V Y2 = c(kCR + 3) * X + c(kCR + 4) * Y + c(kCR + 5) * Z + c(kCt + 1);
    const V Z2 = c(kCR + 6) * X + c(kCR + 7) * Y + c(kCR + 8) * Z + c(kCt + 2);
    const V nr = neg_recip(Z2);
    const V nu = neg_quot<V>(c(kCf) * X2, Z2, nr), nv = neg_quot<V>(c(kCf) * Y2, Z2, nr);
    g.div(Z2);
    g.quot_nonzero(nu);
    g.quot_nonzero(nv);
    uc = c(kCcx) - nu - fx;
    vc = c(kCcy) - nv - fy;
}

// l1_threshold (solveReconDataL1.cu:36-63): the branch's factor, with the sign
// of its step, and its divisor; whether it steps at all (a NaN rho does not)
__device__ __forceinline__ bool l1_branch(float rho, float nupper, float magi, float A, float lambda,
                                          float& fac, float& den) {
    const bool inside = rho <= -nupper && rho >= nupper;
    const bool step = inside ? magi != 0.0f : (rho < nupper || rho > -nupper);
    fac = inside ? rho : (rho < nupper ? -lambda : lambda);
    den = step ? (inside ? magi : A) : 1.0f;
    return step;
}
struct Steps {
    bool x, y;
};
__device__ __forceinline__ bool l1_branches(float rho, float nupper, float magi, float A,
                                            float lambda, float& fac, float& den) {
    return l1_branch(rho, nupper, magi, A, lambda, fac, den);
}
__device__ __forceinline__ Steps l1_branches(f2 rho, f2 nupper, f2 magi, f2 A, f2 lambda, f2& fac,
                                             f2& den) {
    return Steps{l1_branch(rho.x, nupper.x, magi.x, A.x, lambda.x, fac.x, den.x),
                 l1_branch(rho.y, nupper.y, magi.y, A.y, lambda.y, fac.y, den.y)};
}
__device__ __forceinline__ float choose(bool s, float a, float b) { return s ? a : b; }
__device__ __forceinline__ f2 choose(Steps s, f2 a, f2 b) {
    return f2{s.x ? a.x : b.x, s.y ? a.y : b.y};
}
template <class V>
__device__ __forceinline__ void l1_threshold_v(V dusub, V dvsub, V dix, V diy, V dit, V lambda,
                                               V A, V nrA, V& du, V& dv, QuotientGuard& g) {
    const V rho = dix * dusub + diy * dvsub + dit;
    const V magi = dix * dix + diy * diy;
    const V nupper = neg_quot<V>(lambda * magi, A, nrA);  // = lower
    g.quot(nupper);
    g.at_most(nupper);
    V fac, den;
    const auto step = l1_branches(rho, nupper, magi, A, lambda, fac, den);
    const V nr = neg_recip(den);
    const V nu = neg_quot<V>(fac * dix, den, nr), nv = neg_quot<V>(fac * diy, den, nr);
    g.div(den);
    g.quot(nu);
    g.quot(nv);
    du = choose(step, dusub + nu, dusub);
    dv = choose(step, dvsub + nv, dvsub);
}

// solve3d_pixel (solve3dMinimalArea.cu:23-184; its operations in its order, the
// symmetric entries of the normal matrix, whose products commute bit for bit,
// formed once)
template <class V, class C>
__device__ __forceinline__ void solve3d_v(const C& c, V uproj, V vproj, V x1, V y1, bool left,
                                          bool up, const V (&Xn)[5], const V (&Yn)[5],
                                          const V (&Zn)[5], V& Xo, V& Yo, V& Zo,
                                          QuotientGuard& g) {
    const V x2 = x1 + uproj, y2 = y1 + vproj;
    V ax, bx, cx, dx, by, cy, dy, cz, dz;
    {
        V c8 = c(kCQ + 8), c9 = c(kCQ + 9), c10 = c(kCQ + 10),
           c11 = c(kCQ + 11);
        const V r1 = x2 * c8 - c(kCQ + 0), r2 = x2 * c9 - c(kCQ + 1),
                 r3 = x2 * c10 - c(kCQ + 2), r4 = x2 * c11 - c(kCQ + 3);
        const V s1 = y2 * c8 - c(kCQ + 4), s2 = y2 * c9 - c(kCQ + 5),
                 s3 = y2 * c10 - c(kCQ + 6), s4 = y2 * c11 - c(kCQ + 7);
        const V lf = c(kClf);
        if (c.origin()) {
            // camera 0 at the origin: p = (-f, 0, x - cx, 0), q = (0, -g, y - cy, 0)
            // and most of their products are zeros, which leave the sums as they
            // are (but for the sign of a zero, which no point that is not zero
            // itself depends on; a zero point takes the slow path)
            const V p3 = x1 - c(kCP + 2), q3 = y1 - c(kCP + 6);
            const V nf = c(kCP + 0), ng = c(kCP + 5);
            ax = lf * (c(kCff) + r1 * r1 + s1 * s1);
            bx = lf * (r1 * r2 + s1 * s2);
            cx = lf * (r1 * r3 - nf * p3 + s1 * s3);
            dx = lf * (r1 * r4 + s1 * s4);
            by = lf * (c(kCgg) + r2 * r2 + s2 * s2);
            cy = lf * (r2 * r3 - ng * q3 + s2 * s3);
            dy = lf * (r2 * r4 + s2 * s4);
            cz = lf * (p3 * p3 + q3 * q3 + r3 * r3 + s3 * s3);
            dz = lf * (r3 * r4 + s3 * s4);
        } else {
            c8 = c(kCP + 8);
            c9 = c(kCP + 9);
            c10 = c(kCP + 10);
            c11 = c(kCP + 11);
            const V p1 = x1 * c8 - c(kCP + 0), p2 = x1 * c9 - c(kCP + 1),
                     p3 = x1 * c10 - c(kCP + 2), p4 = x1 * c11 - c(kCP + 3);
            const V q1 = y1 * c8 - c(kCP + 4), q2 = y1 * c9 - c(kCP + 5),
                     q3 = y1 * c10 - c(kCP + 6), q4 = y1 * c11 - c(kCP + 7);
            ax = lf * (p1 * p1 + q1 * q1 + r1 * r1 + s1 * s1);
            bx = lf * (p1 * p2 + q1 * q2 + r1 * r2 + s1 * s2);
            cx = lf * (p1 * p3 + q1 * q3 + r1 * r3 + s1 * s3);
            dx = lf * (p1 * p4 + q1 * q4 + r1 * r4 + s1 * s4);
            by = lf * (p2 * p2 + q2 * q2 + r2 * r2 + s2 * s2);
            cy = lf * (p2 * p3 + q2 * q3 + r2 * r3 + s2 * s3);
            dy = lf * (p2 * p4 + q2 * q4 + r2 * r4 + s2 * s4);
            cz = lf * (p3 * p3 + q3 * q3 + r3 * r3 + s3 * s3);
            dz = lf * (p3 * p4 + q3 * q4 + r3 * r4 + s3 * s4);
        }
    }

    const V Xx = Xn[1] - Xn[0], Yx = Yn[1] - Yn[0], Zx = Zn[1] - Zn[0];
    const V Xy = Xn[2] - Xn[0], Yy = Yn[2] - Yn[0], Zy = Zn[2] - Zn[0];

    const V na = Yx * Zy - Zx * Yy, nb = Zx * Xy - Xx * Zy, nc = Xx * Yy - Yx * Xy;
    const V area = na * na + nb * nb + nc * nc + splat<V>(0.001f);
    const V root = sqrt_rn(area);  // at least sqrt(0.001)
    // -lambdams / sqrt(area), and below everything it enters with the sign
    // turned: the quotients at the end turn it back
    const V nlms = neg_quot<V>(c(kClms), root, neg_recip(root));
    g.quot_nonzero(nlms);

    const V half = c(kCHalf);
    V Xi = half * Xn[3] + half * Xn[1], Yi = half * Yn[3] + half * Yn[1],
       Zi = half * Zn[3] + half * Zn[1];
    first_or(Xi, Xn[1], left);
    first_or(Yi, Yn[1], left);
    first_or(Zi, Zn[1], left);
    V Xj = half * Xn[4] + half * Xn[2], Yj = half * Yn[4] + half * Yn[2],
       Zj = half * Zn[4] + half * Zn[2];
    if (!up) {
        Xj = Xn[2];
        Yj = Yn[2];
        Zj = Zn[2];
    }

    const V Xxx = Xx * Xx, Yxx = Yx * Yx, Zxx = Zx * Zx;
    const V Xyy = Xy * Xy, Yyy = Yy * Yy, Zyy = Zy * Zy;
    const V XYx = Xx * Yx, XYy = Xy * Yy, XZx = Xx * Zx, XZy = Xy * Zy, YZx = Yx * Zx,
             YZy = Yy * Zy;

    const V a11 = ax - nlms * (Yxx + Zxx + Yyy + Zyy);
    const V a12 = bx + nlms * (XYx + XYy);
    const V a13 = cx + nlms * (XZx + XZy);
    const V a22 = by - nlms * (Xxx + Zxx + Xyy + Zyy);
    const V a23 = cy + nlms * (YZx + YZy);
    const V a33 = cz - nlms * (Xxx + Yxx + Xyy + Yyy);

    // cofactors; with a21 = a12, a31 = a13, a32 = a23 the reference's E12, E13
    // and E23 are the same expressions as E21, E31 and E32
    const V m2233 = a22 * a33, m2323 = a23 * a23, m1233 = a12 * a33, m2313 = a23 * a13,
             m1223 = a12 * a23, m2213 = a22 * a13;
    const V E11 = m2233 - m2323;
    const V E12 = m2313 - m1233;
    const V E13 = m1223 - m2213;
    const V E22 = a11 * a33 - a13 * a13;
    const V E23 = a13 * a12 - a11 * a23;
    const V E33 = a11 * a22 - a12 * a12;
    const V detA = a11 * E11 - a12 * (m1233 - m2313) + a13 * (m1223 - m2213);

    const V nXYy = -XYy, nXZy = -XZy;
    const V nb1 = nlms * ((Zyy + Yyy) * Xi + (Zxx + Yxx) * Xj - XYy * Yi - XYx * Yj - XZy * Zi -
                         XZx * Zj) + dx;
    const V nb2 = nlms * (nXYy * Xi - XYx * Xj + (Xyy + Zyy) * Yi + (Xxx + Zxx) * Yj - YZy * Zi -
                         YZx * Zj) + dy;
    const V nb3 = nlms * (nXZy * Xi - XZx * Xj - YZy * Yi - YZx * Yj + (Xyy + Yyy) * Zi +
                         (Xxx + Yxx) * Zj) + dz;

    const V nr = neg_recip(detA);
    Xo = neg_quot<V>(E11 * nb1 + E12 * nb2 + E13 * nb3, detA, nr);
    Yo = neg_quot<V>(E12 * nb1 + E22 * nb2 + E23 * nb3, detA, nr);
    Zo = neg_quot<V>(E13 * nb1 + E23 * nb2 + E33 * nb3, detA, nr);
    g.div(detA);
    g.quot_nonzero(Xo);
    g.quot_nonzero(Yo);
    g.quot_nonzero(Zo);
}

// One pixel of A with IEEE divisions (recon_a_px), for pairs whose quotients
// are not sure; out of line.
template <int PRIOR>
__device__ __noinline__ void recon_a_slow(const ReconFields& f, const LevelConsts* lc,
                                          const Weights& wt, LevelDims d, int base, int x, int y,
                                          int first, int uc_from_buffer) {
    recon_a_px<PRIOR, true>(f, *lc, wt, d, x, y, first, uc_from_buffer, base);
}

// A at (x, y), (x + 1, y).  `sc`: pair_consts, filled by the block; every
// thread of the block must call it (it synchronises the block once the loads
// are on their way).
template <int PRIOR>
__device__ __forceinline__ void recon_a_pair(const ReconFields& f, const LevelConsts* lc,
                                             const float2* sc, const Weights& wt, LevelDims d,
                                             int base, int x, int y, bool inside, bool first,
                                             bool uc_from_buffer) {
    const int s = d.s, pos = base + x + y * s;
    const bool both = x + 1 < d.w, left = x > 0, up = y > 0;
    const f2 zero = mk2(0.0f, 0.0f);
    f2 u = zero, v = zero, uproj = zero, vproj = zero, sku = zero, skv = zero;
    f2 dix = zero, diy = zero, dit = zero, duhat = zero, dvhat = zero;
    f2 pu1 = zero, pu2 = zero, pv1 = zero, pv2 = zero, pu2d = zero, pv2d = zero;
    float pu1l = 0.0f, pv1l = 0.0f;
    f2 Xn[5], Yn[5], Zn[5];
#pragma unroll
    for (int i = 0; i < 5; i++) Xn[i] = Yn[i] = Zn[i] = zero;
    if (inside) {
        u = RF_LD2(f, u, pos);
        v = RF_LD2(f, v, pos);
        dix = RF_LD2(f, Ix, pos);
        diy = RF_LD2(f, Iy, pos);
        dit = RF_LD2(f, Iz, pos);
        uproj = RF_LD2(f, uproj, pos);
        vproj = RF_LD2(f, vproj, pos);
        sku = RF_LD2(f, sku, pos);
        skv = RF_LD2(f, skv, pos);
        if (!first) {
            duhat = RF_LD2(f, duhat, pos);
            dvhat = RF_LD2(f, dvhat, pos);
            pu1 = RF_LD2(f, pu1, pos);
            pu2 = RF_LD2(f, pu2, pos);
            pv1 = RF_LD2(f, pv1, pos);
            pv2 = RF_LD2(f, pv2, pos);
            if (left) {
                pu1l = RF_AT(f, pu1, pos - 1);
                pv1l = RF_AT(f, pv1, pos - 1);
            }
            if (up) {
                pu2d = RF_LD2(f, pu2, pos - s);
                pv2d = RF_LD2(f, pv2, pos - s);
            }
        }
        // the points at: 0 = the pixel, 1 = x + 1 (flat pos + 1), 2 = y + 1
        // (flat pos + s), also on the last column and row; 3 = x - 1, 4 = y - 1
        auto around = [&](const float* a, f2 (&n)[5]) {
            const float2 c = ld2_at(a, pos, f.extent), dn = ld2_at(a, pos + s, f.extent);
            n[0] = mk2(c.x, c.y);
            n[1] = mk2(c.y, both ? RF_PT(a, pos + 2, f.extent) : 0.0f);
            n[2] = mk2(dn.x, dn.y);
            n[3] = mk2(left ? RF_PT(a, pos - 1, f.extent) : 0.0f, c.x);
            if (up) {
                const float2 un = ld2_at(a, pos - s, f.extent);
                n[4] = mk2(un.x, un.y);
            }
        };
        around(f.X, Xn);
        around(f.Y, Yn);
        around(f.Z, Zn);
    }
    __syncthreads();
    if (!inside) return;
    const PairConsts c{sc};
    f2 divu = zero, divv = zero;  // of a zero dual field: +0
    if (!first) {
        // multiplier update of the previous B (solveUcSk.cu:94-95)
        sku = sku + u + duhat - uproj;
        skv = skv + v + dvhat - vproj;
        divu = divergence_v(pu1, mk2(pu1l, pu1.x), pu2, pu2d, left, up);
        divv = divergence_v(pv1, mk2(pv1l, pv1.x), pv2, pv2d, left, up);
    }

    // --- data step (solveReconDataL1.cu:24-100) ---
    const f2 atv = c(kCtv), aproj = c(kCproj);
    QuotientGuard g;
    f2 A, nrA, nu, nv;
    const f2 ru = uproj - u - sku, rv = vproj - v - skv;
    if (PRIOR == 0) {
        A = c(kCA);
        nrA = c(kCnrA);
        nu = neg_quot<f2>(atv * duhat + aproj * ru, A, nrA);
        nv = neg_quot<f2>(atv * dvhat + aproj * rv, A, nrA);
    } else {
        f2 afn = c(kCfn);
        if (PRIOR == 2) afn = afn * RF_LD2(f, mask, pos);
        A = atv + aproj + afn;
        nrA = neg_recip(A);
        g.div(A);
        const f2 ufn = RF_LD2(f, ufn, pos), vfn = RF_LD2(f, vfn, pos);
        nu = neg_quot<f2>(afn * (ufn - u) + atv * duhat + aproj * ru, A, nrA);
        nv = neg_quot<f2>(afn * (vfn - v) + atv * dvhat + aproj * rv, A, nrA);
    }
    g.quot(nu);
    g.quot(nv);
    f2 du, dv;
    l1_threshold_v(-nu, -nv, dix, diy, dit, c(kClam), A, nrA, du, dv, g);
    const f2 ndu = neg_quot<f2>(divu, A, nrA), ndv = neg_quot<f2>(divv, A, nrA);
    g.quot(ndu);
    g.quot(ndv);
    const f2 duhat1 = du - ndu, dvhat1 = dv - ndv;

    // --- projection blend (solveUVProj.cu:13-21) ---
    const f2 fx = mk2((float)x, (float)(x + 1)), fy = dup2((float)y);
    f2 uc, vc;
    if (uc_from_buffer) {
        uc = RF_LD2(f, uc, pos);
        vc = RF_LD2(f, vc, pos);
    } else {
        project_uc_v(c, Xn[0], Yn[0], Zn[0], fx, fy, uc, vc, g);
    }
    const f2 lf = c(kClf), pden = c(kCpden), nrP = c(kCnrP);
    uproj = -neg_quot<f2>(lf * uc + aproj * (u + duhat1 + sku), pden, nrP);
    vproj = -neg_quot<f2>(lf * vc + aproj * (v + dvhat1 + skv), pden, nrP);
    g.quot_nonzero(uproj);
    g.quot_nonzero(vproj);

    // --- triangulation with minimal-area smoothing ---
    f2 Xo, Yo, Zo;
    solve3d_v(c, uproj, vproj, fx, fy, left, up, Xn, Yn, Zn, Xo, Yo, Zo, g);
    // any quotient that is not sure, or anything that is not finite (it
    // reaches the points): the pixels with IEEE divisions
    if (!(g.ok() && finite3(Xo.x, Yo.x, Zo.x) && finite3(Xo.y, Yo.y, Zo.y))) {
        recon_a_slow<PRIOR>(f, lc, wt, d, base, x, y, first, uc_from_buffer);
        if (both) recon_a_slow<PRIOR>(f, lc, wt, d, base, x + 1, y, first, uc_from_buffer);
        return;
    }
    if (!first) {
        RF_ST2(f, sku, pos, sku, both);
        RF_ST2(f, skv, pos, skv, both);
    }
    RF_ST2(f, duhat, pos, duhat1, both);
    RF_ST2(f, dvhat, pos, dvhat1, both);
    RF_ST2(f, uproj, pos, uproj, both);
    RF_ST2(f, vproj, pos, vproj, both);
    RF_ST2(f, X1, pos, Xo, both);
    RF_ST2(f, Y1, pos, Yo, both);
    RF_ST2(f, Z1, pos, Zo, both);
}

// What B stages: planes 0 .. 2 are X1, Y1, Z1 (with the ring of eight
// neighbours), 3, 4 are duhat (with the row below and the column to the
// right), 5 .. 8 are pu1, pu2, pv1, pv2 (the tile's rows).
struct StageB {
    static constexpr int ROWS = kPairRows;
    static __device__ constexpr int off(int i) {
        return i < 3 ? (i * (ROWS + 2) + 1) * kPitch
                     : (i < 5 ? (3 * (ROWS + 2) + (i - 3) * (ROWS + 1)) * kPitch
                              : (3 * (ROWS + 2) + 2 * (ROWS + 1) + (i - 5) * ROWS) * kPitch);
    }
    static constexpr int FLOATS = (3 * (ROWS + 2) + 2 * (ROWS + 1) + 4 * ROWS) * kPitch;
};

template <bool LAST>
__device__ __forceinline__ void stage_b(const ReconFields& f, float* sm, LevelDims d, int base,
                                        int x0, int y0, bool first) {
    using S = StageB;
    constexpr int ROWS = kPairRows;
    const int lane = threadIdx.x & 31, row = threadIdx.x >> 5, half = lane >> 4;
    const int c = 4 * (lane & 15), x = x0 + c, y = y0 + row, s = d.s;
    const int src = base + x + y * s, dst = row * kPitch + 4 + c;
    const bool in = y < d.h && x < s;
    auto two = [&](const float* a, int ia, const float* b, int ib, bool ok) {
        if (ok) copy16(sm + dst + (half ? S::off(ib) : S::off(ia)), half ? b : a, src, f.extent);
    };
    two(f.X1, 0, f.Y1, 1, in);
    two(f.Z1, 2, f.duhat, 3, in);
    if (LAST) {
        two(f.dvhat, 4, f.dvhat, 4, in && half == 0);
    } else if (first) {
        two(f.dvhat, 4, f.dvhat, 4, in && half == 0);
    } else {
        two(f.dvhat, 4, f.pu1, 5, in);
        two(f.pu2, 6, f.pv1, 7, in);
        two(f.pv2, 8, f.pv2, 8, in && half == 0);
    }
    // the rows above and below: X1, Y1, Z1 above, X1, Y1, Z1 and duhat below
    for (int k = 2 * row + half; k < (LAST ? 6 : 8); k += 2 * ROWS) {
        const int i = k < 3 ? k : k - 3;
        const float* a = i == 0 ? f.X1 : (i == 1 ? f.Y1 : (i == 2 ? f.Z1 : (i == 3 ? f.duhat : f.dvhat)));
        const int r = k < 3 ? -1 : ROWS, yr = y0 + r;
        if (yr >= 0 && yr < d.h && x < s)
            copy16(sm + S::off(i) + r * kPitch + 4 + c, a, base + x + yr * s, f.extent);
    }
    // the columns: X1, Y1, Z1 left and right, duhat right
    constexpr int kR = ROWS + 2;
    for (int k = threadIdx.x; k < (LAST ? 6 : 8) * kR; k += 32 * ROWS) {
        const int t = k / kR, r = k % kR - 1, yr = y0 + r;
        const int i = t < 3 ? t : t - 3;
        const float* a = i == 0 ? f.X1 : (i == 1 ? f.Y1 : (i == 2 ? f.Z1 : (i == 3 ? f.duhat : f.dvhat)));
        const bool right = t >= 3;
        const int xr = right ? x0 + kPairW : x0 - 4;
        if (yr >= 0 && yr < d.h && (right ? xr < d.w : x0 > 0) && !(t >= 6 && (r < 0 || r >= ROWS)))
            copy16(sm + S::off(i) + r * kPitch + (right ? kPairW + 4 : 0), a, base + xr + yr * s,
                   f.extent);
    }
}

// B for the tile at (x0, y0); `first`: the dual field before it is zero.
// LAST: a warp's last B (the multiplier update instead of the dual update).
// `sm`: StageB::FLOATS; synchronises the block.
template <bool LAST>
__device__ __forceinline__ void recon_b_tile(const ReconFields& f, const Weights& wt, float* sm,
                                             LevelDims d, int base, int x0, int y0, bool first) {
    using S = StageB;
    stage_b<LAST>(f, sm, d, base, x0, y0, first);
    const int lane = threadIdx.x & 31, row = threadIdx.x >> 5;
    const int x = x0 + 2 * lane, y = y0 + row, pos = base + x + y * d.s;
    const PairEdges e = pair_edges(x, y, d);
    copies_done();
    if (x >= d.w || y >= d.h) return;
    const float* my = sm + row * kPitch + 4 + 2 * lane;
    PointTaps t;
    load_taps(my + S::off(0), e, t.x);
    load_taps(my + S::off(1), e, t.y);
    load_taps(my + S::off(2), e, t.z);
    f2 X, Y, Z;
    points_pair(e, t, X, Y, Z);
    if (LAST) {
        const f2 u = RF_LD2(f, u, pos), v = RF_LD2(f, v, pos);
        const f2 uproj = RF_LD2(f, uproj, pos), vproj = RF_LD2(f, vproj, pos);
        const f2 sku = RF_LD2(f, sku, pos), skv = RF_LD2(f, skv, pos);
        RF_ST2(f, sku, pos, sku + u + lds2(my + S::off(3)) - uproj, e.both);
        RF_ST2(f, skv, pos, skv + v + lds2(my + S::off(4)) - vproj, e.both);
    } else {
        const f2 zero = mk2(0.0f, 0.0f);
        DualIn in;
        in.u = lds2(my + S::off(3));
        in.v = lds2(my + S::off(4));
        in.ur = my[S::off(3) + 2];
        in.vr = my[S::off(4) + 2];
        in.ud = lds2(my + S::off(3) + kPitch);
        in.vd = lds2(my + S::off(4) + kPitch);
        in.pu1 = first ? zero : lds2(my + S::off(5));
        in.pu2 = first ? zero : lds2(my + S::off(6));
        in.pv1 = first ? zero : lds2(my + S::off(7));
        in.pv2 = first ? zero : lds2(my + S::off(8));
        dual_update(in, wt.fac, e);
        RF_ST2(f, pu1, pos, in.pu1, e.both);
        RF_ST2(f, pu2, pos, in.pu2, e.both);
        RF_ST2(f, pv1, pos, in.pv1, e.both);
        RF_ST2(f, pv2, pos, in.pv2, e.both);
    }
    RF_ST2(f, X, pos, X, e.both);
    RF_ST2(f, Y, pos, Y, e.both);
    RF_ST2(f, Z, pos, Z, e.both);
}

// ---- one pixel per thread ---------------------------------------------------
// Part A's arithmetic at (x, y), the multiplier update first (recon_a_point
// with the quotients above); false where they are not sure: `a` is then spoilt.
template <int PRIOR>
__device__ __forceinline__ bool recon_a_fast(APoint& a, const LevelConsts& lc, const Weights& wt,
                                             int x, int y, bool first, bool uc_from_buffer) {
    const bool left = x > 0, up = y > 0;
    const OneConsts c{lc, wt};
    float divu = 0.0f, divv = 0.0f;
    if (!first) {
        a.sku = a.sku + a.u + a.duhat - a.uproj;
        a.skv = a.skv + a.v + a.dvhat - a.vproj;
        divu = divergence_v(a.pu1, a.pu1l, a.pu2, a.pu2d, left, up);
        divv = divergence_v(a.pv1, a.pv1l, a.pv2, a.pv2d, left, up);
    }
    QuotientGuard g;
    float A, nrA, nu, nv;
    const float ru = a.uproj - a.u - a.sku, rv = a.vproj - a.v - a.skv;
    if (PRIOR == 0) {
        A = wt.A;
        nrA = wt.nrA;
        nu = neg_quot(wt.alpha_tv * a.duhat + wt.alpha_proj * ru, A, nrA);
        nv = neg_quot(wt.alpha_tv * a.dvhat + wt.alpha_proj * rv, A, nrA);
    } else {
        const float afn = PRIOR == 2 ? wt.alpha_fn * a.mk : wt.alpha_fn;
        A = wt.alpha_tv + wt.alpha_proj + afn;
        nrA = neg_recip(A);
        g.div(A);
        nu = neg_quot(afn * (a.ufn - a.u) + wt.alpha_tv * a.duhat + wt.alpha_proj * ru, A, nrA);
        nv = neg_quot(afn * (a.vfn - a.v) + wt.alpha_tv * a.dvhat + wt.alpha_proj * rv, A, nrA);
    }
    g.quot(nu);
    g.quot(nv);
    float du, dv;
    l1_threshold_v(-nu, -nv, a.dix, a.diy, a.dit, wt.lambda, A, nrA, du, dv, g);
    const float ndu = neg_quot(divu, A, nrA), ndv = neg_quot(divv, A, nrA);
    g.quot(ndu);
    g.quot(ndv);
    a.duhat = du - ndu;
    a.dvhat = dv - ndv;
    const float fx = (float)x, fy = (float)y;
    if (!uc_from_buffer) project_uc_v(c, a.Xn[0], a.Yn[0], a.Zn[0], fx, fy, a.uc, a.vc, g);
    a.uproj = -neg_quot(wt.lambdaf * a.uc + wt.alpha_proj * (a.u + a.duhat + a.sku), wt.proj_den, wt.nrP);
    a.vproj = -neg_quot(wt.lambdaf * a.vc + wt.alpha_proj * (a.v + a.dvhat + a.skv), wt.proj_den, wt.nrP);
    g.quot_nonzero(a.uproj);
    g.quot_nonzero(a.vproj);
    solve3d_v(c, a.uproj, a.vproj, fx, fy, left, up, a.Xn, a.Yn, a.Zn, a.Xo, a.Yo, a.Zo, g);
    return g.ok() && finite3(a.Xo, a.Yo, a.Zo);
}

// A at a pixel (recon_a_px with the multiplier update first and the quotients
// above).
template <int PRIOR>
__device__ __forceinline__ void recon_a_one(const ReconFields& f, const LevelConsts& lc,
                                            const Weights& wt, LevelDims d, int base, int x, int y,
                                            bool first, bool uc_from_buffer) {
    const int pos = base + x + y * d.s;
    APoint a;
    load_a<PRIOR>(f, d, pos, x, y, first, uc_from_buffer, a);
    if (recon_a_fast<PRIOR>(a, lc, wt, x, y, first, uc_from_buffer)) store_a<true>(f, pos, first, a);
    else recon_a_slow<PRIOR>(f, &lc, wt, d, base, x, y, first, uc_from_buffer);
}

// the 3x3 taps of a pixel, border rules as load_taps
__device__ __forceinline__ void load_taps_one(const float* a, int p, int s, long long n,
                                              PairEdges e, float (&t)[3][3]) {
#pragma unroll
    for (int j = 0; j < 3; j++) {
        const int q = j == 0 ? (e.up ? p - s : p) : (j == 1 ? p : p + s);
        const bool in = j != 2 || e.down;
        const float c = in ? RF_PT(a, q, n) : 0.0f;
        t[j][0] = !in ? 0.0f : (e.left ? RF_PT(a, q - 1, n) : (j != 0 || e.up ? c : 0.0f));
        t[j][1] = c;
        t[j][2] = in && e.both ? RF_PT(a, q + 1, n) : 0.0f;
    }
}
__device__ __forceinline__ float median3_one(const float (&t)[3][3]) {
    float lo[3], mid[3], hi[3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const float s = nmin(t[0][i], t[1][i]), g = nmax(t[0][i], t[1][i]);
        lo[i] = nmin(s, t[2][i]);
        hi[i] = nmax(g, t[2][i]);
        mid[i] = nmax(s, nmin(g, t[2][i]));
    }
    return nmed3(nmax3(lo[0], lo[1], lo[2]), nmed3(mid[0], mid[1], mid[2]),
                 nmin3(hi[0], hi[1], hi[2]));
}

// the point of B from the taps: medians and clean-up
__device__ __forceinline__ void point_one(const float (&tx)[3][3], const float (&ty)[3][3],
                                          const float (&tz)[3][3], float& X, float& Y, float& Z) {
    float Xm = median3_one(tx), Ym = median3_one(ty), Zm = median3_one(tz);
    auto sure = [](float m) { return fabsf(m) > 0.0f; };
    if (!(sure(Xm) && sure(Ym) && sure(Zm))) {
        if (!sure(Xm)) Xm = median9_slow(tx, 0);
        if (!sure(Ym)) Ym = median9_slow(ty, 0);
        if (!sure(Zm)) Zm = median9_slow(tz, 0);
    }
    cleanup_pixel(tx[1][1], ty[1][1], tz[1][1], Xm, Ym, Zm, X, Y, Z);
}
// the dual update of B from the differences of duhat; p = pu1, pu2, pv1, pv2
__device__ __forceinline__ void dual_one(float ux, float uy, float vx, float vy, float fac,
                                         float* p) {
    QuotientGuard g;
    float pu1 = p[0], pu2 = p[1], pv1 = p[2], pv2 = p[3];
    dual_step_v(ux, uy, fac, pu1, pu2, g);
    dual_step_v(vx, vy, fac, pv1, pv2, g);
    if (g.ok() && isfinite(pu1 + pu2 + pv1 + pv2)) {
        p[0] = pu1;
        p[1] = pu2;
        p[2] = pv1;
        p[3] = pv2;
    } else {
        const float2 pu = dual_step_slow(ux, uy, fac, p[0], p[1]);
        const float2 pv = dual_step_slow(vx, vy, fac, p[2], p[3]);
        p[0] = pu.x;
        p[1] = pu.y;
        p[2] = pv.x;
        p[3] = pv.y;
    }
}

// B at a pixel (recon_b_px without the multiplier update); LAST as
// recon_b_tile.
template <bool LAST>
__device__ __forceinline__ void recon_b_one(const ReconFields& f, const Weights& wt, LevelDims d,
                                            int base, int x, int y, bool first) {
    const int s = d.s, pos = base + x + y * s;
    // `both`, `right`: x + 1 < w
    const PairEdges e{x > 0, x + 1 < d.w, x + 1 < d.w, y > 0, y + 1 < d.h};
    float tx[3][3], ty[3][3], tz[3][3];
    load_taps_one(f.X1, pos, s, f.extent, e, tx);
    load_taps_one(f.Y1, pos, s, f.extent, e, ty);
    load_taps_one(f.Z1, pos, s, f.extent, e, tz);
    const float duhat = RF_AT(f, duhat, pos), dvhat = RF_AT(f, dvhat, pos);
    float a[6] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    float ux = 0.0f, uy = 0.0f, vx = 0.0f, vy = 0.0f;
    if (LAST) {
        a[0] = RF_AT(f, u, pos);
        a[1] = RF_AT(f, v, pos);
        a[2] = RF_AT(f, uproj, pos);
        a[3] = RF_AT(f, vproj, pos);
        a[4] = RF_AT(f, sku, pos);
        a[5] = RF_AT(f, skv, pos);
    } else {
        if (!first) {
            a[0] = RF_AT(f, pu1, pos);
            a[1] = RF_AT(f, pu2, pos);
            a[2] = RF_AT(f, pv1, pos);
            a[3] = RF_AT(f, pv2, pos);
        }
        if (e.both) {
            ux = RF_AT(f, duhat, pos + 1) - duhat;
            vx = RF_AT(f, dvhat, pos + 1) - dvhat;
        }
        if (e.down) {
            uy = RF_AT(f, duhat, pos + s) - duhat;
            vy = RF_AT(f, dvhat, pos + s) - dvhat;
        }
    }
    float X, Y, Z;
    point_one(tx, ty, tz, X, Y, Z);
    if (LAST) {
        RF_AT(f, sku, pos) = a[4] + a[0] + duhat - a[2];
        RF_AT(f, skv, pos) = a[5] + a[1] + dvhat - a[3];
    } else {
        dual_one(ux, uy, vx, vy, wt.fac, a);
        RF_AT(f, pu1, pos) = a[0];
        RF_AT(f, pu2, pos) = a[1];
        RF_AT(f, pv1, pos) = a[2];
        RF_AT(f, pv2, pos) = a[3];
    }
    RF_AT(f, X, pos) = X;
    RF_AT(f, Y, pos) = Y;
    RF_AT(f, Z, pos) = Z;
}

}  // namespace
}  // namespace rf
