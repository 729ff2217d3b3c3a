// Learned warm start: a small convolutional encoder-decoder that maps a
// coarse image pair (+ pixel coordinates and camera pose) to flow and inverse
// depth at two scales, trained on the GPU with hand-written forward and
// backward kernels.  No counterpart in the reference.
//
// Network (NHWC, 3x3 convolutions, padding 1):
//   in  (16 ch: the features of rf_ws_features: coarse frames, plane-sweep
//        costs, epipolar derivative)
//   c1  16 -> 32, ReLU                      (input resolution, "1/8")
//   c2  32 -> 96, stride 2, ReLU            (half resolution, "1/16")
//   c3  96 -> 96, ReLU
//   h16 96 -> 8 (u, v, inverse depth, 5 unused), linear   -> output at 1/16
//   cat [nearest-upsampled c3 (96), c1 (32)] = 128 channels
//   c4  128 -> 64, ReLU
//   h8  64 -> 8, linear                                    -> output at 1/8
// Weights and activations are BF16, accumulation FP32; the master weights
// and Adam moments are FP32.
//
// Every convolution (forward, gradient of its input, gradient of its
// weights) is one implicit GEMM on the Blackwell tensor cores (rf_tc.cuh:
// tcgen05.mma, BF16 operands gathered into shared memory, FP32 accumulator
// in tensor memory).  The weight gradient splits the pixel (reduction)
// dimension into chunks whose partial sums are added in a fixed order, so
// training is deterministic.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "../../include/reconflow_gb300.h"
#include "rf_alloc.h"
#include "rf_nvtx.h"
#include "rf_kernels.cuh"
#include "rf_rules.h"
#include "rf_tc.cuh"

namespace rf_cnn_impl {

typedef __nv_bfloat16 bf16;

__device__ __forceinline__ uint32_t pack2(bf16 lo, bf16 hi) {
    return (uint32_t)__bfloat16_as_ushort(lo) | ((uint32_t)__bfloat16_as_ushort(hi) << 16);
}

struct Shape {
    int B, H, W, C;  // NHWC
};

// ---- tcgen05 GEMM operands: 8 consecutive K elements of one row (rf_tc.cuh) ----
__device__ __forceinline__ uint4 pack8(const bf16 (&v)[8]) {
    return make_uint4(pack2(v[0], v[1]), pack2(v[2], v[3]), pack2(v[4], v[5]), pack2(v[6], v[7]));
}

using rf_tc::TcPos;
using rf_tc::TcRow;
// (a buffer has at most 2^26 pixels of 128 channels, 2^30 units of 16 bytes)
__device__ __forceinline__ const uint4* units(const bf16* p) {
    return reinterpret_cast<const uint4*>(p);
}

// forward A: im2col row of output pixel m, k = (ky*3 + kx)*C + ci (C % 8 == 0)
struct TcConvIn {
    const bf16* x;
    int H, W, C, Ho, Wo, stride;
    __device__ const uint4* base() const { return units(x); }
    __device__ TcRow row(int m, int M) const {
        const int xo = m % Wo, r = m / Wo, yo = r % Ho, b = r / Ho;
        const int y = yo * stride - 1, xx = xo * stride - 1;
        return TcRow{((b * H + y) * W + xx) * (C / 8), m < M ? rf_tc::conv_taps(y, xx, H, W) : 0u};
    }
    __device__ TcPos kpos(int k) const {
        const int ci = k % C, t = k / C;
        return TcPos{(t / 3 * W + t % 3) * (C / 8) + ci / 8, t};
    }
};

// K-major matrix rows: w[n][k], K % 8 == 0
struct TcRows {
    const bf16* w;
    int K;
    __device__ const uint4* base() const { return units(w); }
    __device__ TcRow row(int n, int N) const { return TcRow{n * (K / 8), n < N ? 1u : 0u}; }
    __device__ TcPos kpos(int k) const { return TcPos{k / 8, 0}; }
};

// input-gradient A (stride 1): input pixel m, k = (ky*3 + kx)*Cout + co -> dy at
// the output pixel that tap (ky, kx) of m feeds (Cout % 8 == 0)
struct TcDataGradA {
    const bf16* dy;
    int H, W, Cout;
    __device__ const uint4* base() const { return units(dy); }
    __device__ TcRow row(int m, int M) const {
        const int x = m % W, r = m / W, y = r % H, b = r / H;
        unsigned taps = 0, cols = 0;
#pragma unroll
        for (int i = 0; i < 3; i++) cols |= (unsigned)(x + 1 - i) < (unsigned)W ? 1u << i : 0u;
#pragma unroll
        for (int i = 0; i < 3; i++) taps |= (unsigned)(y + 1 - i) < (unsigned)H ? cols << 3 * i : 0u;
        return TcRow{((b * H + y + 1) * W + x + 1) * (Cout / 8), m < M ? taps : 0u};
    }
    __device__ TcPos kpos(int k) const {
        const int co = k % Cout, t = k / Cout;
        return TcPos{co / 8 - (t / 3 * W + t % 3) * (Cout / 8), t};
    }
};

// the same for a stride of 2 and the input pixels (2 yc + py, 2 xc + px): 1, 2 or
// 4 of the nine taps reach them, k = (index among those)*Cout + co.  All pixels at
// once spent three quarters of the K loop on zeros (0.49 ms for 64 images of
// 160 x 120; 0.19 by parity, four launches).
struct Parity2 {
    int py, px;
    __device__ int taps_x() const { return px + 1; }
    __device__ int tap(int i) const {  // ky * 3 + kx
        const int iy = i / taps_x(), ix = i % taps_x();
        return (py ? 2 * iy : 1) * 3 + (px ? 2 * ix : 1);
    }
};
struct TcDataGrad2A {
    const bf16* dy;
    int Hc, Wc, Ho, Wo, Cout;
    Parity2 q;
    __device__ const uint4* base() const { return units(dy); }
    __device__ TcRow row(int m, int M) const {
        // tap (iy, ix) of those reads output pixel (y - iy, x - ix)
        const int xc = m % Wc, r = m / Wc, yc = r % Hc, b = r / Hc;
        const int y = yc + q.py, x = xc + q.px;
        unsigned taps = 0;
        for (int iy = 0; iy <= q.py; iy++)
            for (int ix = 0; ix <= q.px; ix++)
                if ((unsigned)(y - iy) < (unsigned)Ho && (unsigned)(x - ix) < (unsigned)Wo)
                    taps |= 1u << (iy * q.taps_x() + ix);
        return TcRow{((b * Ho + y) * Wo + x) * (Cout / 8), m < M ? taps : 0u};
    }
    __device__ TcPos kpos(int k) const {
        const int i = k / Cout, iy = i / q.taps_x(), ix = i % q.taps_x();
        return TcPos{k % Cout / 8 - (iy * Wo + ix) * (Cout / 8), i};
    }
};
struct TcTapRows {
    const bf16* w;  // [n][tap][Cout]
    int Cout;
    Parity2 q;
    __device__ const uint4* base() const { return units(w); }
    __device__ TcRow row(int n, int N) const { return TcRow{n * 9 * (Cout / 8), n < N ? 1u : 0u}; }
    __device__ TcPos kpos(int k) const {
        return TcPos{(q.tap(k / Cout) * Cout + k % Cout) / 8, 0};
    }
};

// weight-gradient partial of split z: part[z][co = n][row m]
struct TcStoreWGrad {
    float* part;
    int M, N;
    __device__ void operator()(int z, int m, int n, float v) const {
        part[((size_t)z * N + n) * M + m] = v;
    }
};

// [co][tap][ci] -> [ci][tap][co] (the input gradient's K-major B operand)
__global__ void k_transpose_w(const bf16* w, int cin, int cout, bf16* wt) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int n = cout * 9 * cin;
    if (i >= n) return;
    int ci = i % cin, t = (i / cin) % 9, co = i / (9 * cin);
    wt[((size_t)ci * 9 + t) * cout + co] = w[i];
}

__device__ __forceinline__ void store8(float* p, const float (&v)[8]) {
    reinterpret_cast<float4*>(p)[0] = make_float4(v[0], v[1], v[2], v[3]);
    reinterpret_cast<float4*>(p)[1] = make_float4(v[4], v[5], v[6], v[7]);
}
__device__ __forceinline__ uint4 pack8(const float (&v)[8]) {
    bf16 h[8];
#pragma unroll
    for (int e = 0; e < 8; e++) h[e] = __float2bfloat16(v[e]);
    return pack8(h);
}
// + bias, optional ReLU
__device__ __forceinline__ void bias_relu(const float* bias, int relu, const float (&v)[8],
                                          float (&o)[8]) {
#pragma unroll
    for (int e = 0; e < 8; e++) {
        const float t = v[e] + bias[e];
        o[e] = relu ? fmaxf(t, 0.f) : t;
    }
}

// forward epilogue: + bias, optional ReLU; BF16 activation and/or FP32 copy
struct ConvOut {
    const float* bias;
    bf16* y;
    float* yf;
    int Cout, relu;
    __device__ void operator()(int m, int n, const float (&v)[8]) const {
        float o[8];
        bias_relu(bias + n, relu, v, o);
        if (y) *(uint4*)(y + (size_t)m * Cout + n) = pack8(o);
        if (yf) store8(yf + (size_t)m * Cout + n, o);
    }
};

struct StoreF32 {
    float* out;
    int N;
    __device__ void operator()(int m, int n, const float (&v)[8]) const {
        store8(out + (size_t)m * N + n, v);
    }
};

struct StoreF32Parity {
    float* out;
    int N, H, W, Hc, Wc;
    Parity2 q;
    __device__ void operator()(int m, int n, const float (&v)[8]) const {
        const int xc = m % Wc, r = m / Wc, yc = r % Hc, b = r / Hc;
        store8(out + (((size_t)b * H + 2 * yc + q.py) * W + 2 * xc + q.px) * N + n, v);
    }
};

__global__ void k_reduce_partials(const float* part, int chunks, int n, float* out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float s = 0.f;
    for (int c = 0; c < chunks; c++) s += part[(size_t)c * n + i];
    out[i] = s;
}

// The elementwise passes take 4 (FP32) or 8 (BF16 copies) channels per thread:
// every channel count is a multiple of 8, and one element per thread, with its
// index divisions, ran at 0.3 - 0.4 of the HBM rate.
__device__ __forceinline__ uint2 bf16x4(float4 v) {
    return make_uint2(pack2(__float2bfloat16(v.x), __float2bfloat16(v.y)),
                      pack2(__float2bfloat16(v.z), __float2bfloat16(v.w)));
}
// n a multiple of 4; `a` may be the caller's, aligned as a float only
__global__ void k_f32_to_bf16(const float* a, bf16* b, size_t n) {
    const size_t i = 4 * ((size_t)blockIdx.x * blockDim.x + threadIdx.x);
    if (i >= n) return;
    const float4 v = (uintptr_t)a % 16 == 0 ? *(const float4*)(a + i)
                                            : make_float4(a[i], a[i + 1], a[i + 2], a[i + 3]);
    *(uint2*)(b + i) = bf16x4(v);
}
__device__ __forceinline__ bool bf16_positive(unsigned bits) {  // > 0 (not NaN)
    bits &= 0xFFFFu;
    return bits != 0 && bits <= 0x7F80u;
}

// A layer's output gradient dy = (g + add) * [act > 0] (`add` null: none; `act`
// null: a linear layer) as BF16, and the partial sums of its bias gradient: block b
// takes pixels [b kGradSpan, (b + 1) kGradSpan), thread t the four channels
// 4 (t % (C / 4)) of every R-th pixel; the R sums of a channel are added in order,
// k_reduce_bias adds the blocks' (deterministic).  One pass and no FP32 copy of dy:
// as two passes (masked gradient in place and BF16 copy, then the sums) the
// 64-channel layer of 64 images of 160 x 120 took 0.26 ms, now 0.09 (6.9 TB/s).
constexpr int kGradThreads = 256, kGradSpan = 512;

__global__ void __launch_bounds__(kGradThreads) k_grad_in(const float* g, const float* add,
                                                          const bf16* act, bf16* gb, int P, int C,
                                                          float* part) {
    __shared__ float4 red[kGradThreads];
    const int t = threadIdx.x, Q = C / 4, R = kGradThreads / Q;
    const int q = t % Q, r = t / Q;
    const int p0 = blockIdx.x * kGradSpan, p1 = min(P, p0 + kGradSpan);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < R)
#pragma unroll 4
        for (int p = p0 + r; p < p1; p += R) {
            const size_t i = (size_t)p * C + 4 * q;
            float4 v = *(const float4*)(g + i);
            if (add) {
                const float4 a = *(const float4*)(add + i);
                v.x += a.x;
                v.y += a.y;
                v.z += a.z;
                v.w += a.w;
            }
            if (act) {
                const uint2 a = *(const uint2*)(act + i);
                if (!bf16_positive(a.x)) v.x = 0.f;
                if (!bf16_positive(a.x >> 16)) v.y = 0.f;
                if (!bf16_positive(a.y)) v.z = 0.f;
                if (!bf16_positive(a.y >> 16)) v.w = 0.f;
            }
            *(uint2*)(gb + i) = bf16x4(v);
            acc.x += v.x;
            acc.y += v.y;
            acc.z += v.z;
            acc.w += v.w;
        }
    red[t] = acc;
    __syncthreads();
    if (t < Q) {
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int k = 0; k < R; k++) {
            const float4 v = red[t + k * Q];
            s.x += v.x;
            s.y += v.y;
            s.z += v.z;
            s.w += v.w;
        }
        *(float4*)(part + (size_t)blockIdx.x * C + 4 * t) = s;
    }
}

// channel blockIdx.x of `n` blocks' partial sums
__global__ void __launch_bounds__(kGradThreads) k_reduce_bias(const float* part, int n, int C,
                                                              float* out) {
    __shared__ float red[kGradThreads];
    float s = 0.f;
    for (int i = threadIdx.x; i < n; i += kGradThreads) s += part[(size_t)i * C + blockIdx.x];
    red[threadIdx.x] = s;
    for (int k = kGradThreads / 2; k > 0; k /= 2) {
        __syncthreads();
        if (threadIdx.x < k) red[threadIdx.x] += red[threadIdx.x + k];
    }
    if (threadIdx.x == 0) out[blockIdx.x] = red[0];
}

// cat = [nearest 2x upsample of a (Ha x Wa x Ca), b (H x W x Cb)], 8 channels
// per thread
__global__ void k_concat_up(const bf16* a, int Ha, int Wa, int Ca, const bf16* b, int Cb,
                            int Bn, int H, int W, bf16* cat) {
    const int C = Ca + Cb, G = C / 8;
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)Bn * H * W * G) return;
    const int c = (int)(i % G) * 8;
    const size_t p = i / G;
    const int x = (int)(p % W), r = (int)(p / W), y = r % H, bb = r / H;
    *(uint4*)(cat + p * C + c) =
        c < Ca ? *(const uint4*)(a + (((size_t)bb * Ha + y / 2) * Wa + x / 2) * Ca + c)
               : *(const uint4*)(b + p * Cb + (c - Ca));
}

// split the concat gradient: d_a (half resolution) = sum of its 2x2 children
// (in row order), d_b = the rest; 4 channels per thread
__global__ void k_concat_up_grad(const float* dcat, int Ha, int Wa, int Ca, int Cb, int Bn,
                                 int H, int W, float* da, float* db) {
    const size_t i = 4 * ((size_t)blockIdx.x * blockDim.x + threadIdx.x);
    const size_t na = (size_t)Bn * Ha * Wa * Ca;
    const size_t nb = (size_t)Bn * H * W * Cb;
    const int C = Ca + Cb;
    if (i < na) {
        const int c = (int)(i % Ca);
        const size_t p = i / Ca;
        const int x = (int)(p % Wa), r = (int)(p / Wa), y = r % Ha, bb = r / Ha;
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int dy = 0; dy < 2; dy++)
            for (int dx = 0; dx < 2; dx++) {
                const int yy = 2 * y + dy, xx = 2 * x + dx;
                if (yy < H && xx < W) {
                    const float4 t = *(const float4*)(dcat + (((size_t)bb * H + yy) * W + xx) * C + c);
                    s.x += t.x;
                    s.y += t.y;
                    s.z += t.z;
                    s.w += t.w;
                }
            }
        *(float4*)(da + i) = s;
    }
    if (i < nb) {
        const int c = (int)(i % Cb);
        *(float4*)(db + i) = *(const float4*)(dcat + i / Cb * C + Ca + c);
    }
}

// L1 loss on channels 0..2 of 8 with per-channel weights, masked; writes dL/dpred
// (already divided by the number of valid pixels) and accumulates the loss.
__global__ void k_l1_loss(const float4* pred, const float* tgt, const float* mask, int P,
                          float w0, float w1, float w2, float inv_count, float4* grad,
                          double* loss) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    double l = 0.0;
    if (p < P) {
        const float m = mask[p];
        float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
        if (m > 0.f) {
            const float4 a = pred[2 * (size_t)p];
            const float* t = tgt + 8 * (size_t)p;  // the caller's, aligned as a float only
            auto term = [&](float wc, float d) {
                l += (double)(wc * fabsf(d)) * inv_count;
                return (d > 0.f ? wc : (d < 0.f ? -wc : 0.f)) * inv_count;
            };
            g.x = term(w0, a.x - t[0]);
            g.y = term(w1, a.y - t[1]);
            g.z = term(w2, a.z - t[2]);
        }
        grad[2 * (size_t)p] = g;
        grad[2 * (size_t)p + 1] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    for (int o = 16; o > 0; o >>= 1) l += __shfl_down_sync(0xffffffffu, l, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(loss, l);
}

__global__ void k_adam(float* w, const float* g, float* m, float* v, size_t n, float lr, float b1,
                       float b2, float eps, float c1, float c2) {
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float gi = g[i];
    float mi = b1 * m[i] + (1.f - b1) * gi;
    float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    float mh = mi / c1, vh = vi / c2;
    w[i] -= lr * mh / (sqrtf(vh) + eps);
}

inline unsigned blocks_for(size_t n, int t = 256) { return (unsigned)((n + t - 1) / t); }

// ---- inference path on padded activations (rf_tc::k_tc_conv3) -------------
// A padded buffer holds [C / 8] planes of [B][H + 2][W + 2] positions of 8 BF16
// channels with a zero one-pixel border; interior pixel (b, y, x) is at position
// (b (H + 2) + y + 1)(W + 2) + x + 1.  Borders are zeroed when a frame size is
// first used and never written; planes are max_batch images apart.
__device__ __forceinline__ size_t pad_pos(int b, int y, int x, int H, int W) {
    return ((size_t)b * (H + 2) + y + 1) * (W + 2) + x + 1;
}

// FP32 input [B][H][W][16] -> padded BF16 interior, 8 channels per thread
__global__ void k_pad_input(const float* in, int B, int H, int W, size_t plane, bf16* xp) {
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    size_t n = (size_t)B * H * W * 2;
    if (i >= n) return;
    const int g = (int)(i % 2);
    const size_t p = i / 2;
    const int x = (int)(p % W), r = (int)(p / W), y = r % H, b = r / H;
    const float* s = in + p * 16 + g * 8;
    bf16 v[8];
#pragma unroll
    for (int e = 0; e < 8; e++) v[e] = __float2bfloat16(s[e]);
    *(uint4*)(xp + (g * plane + pad_pos(b, y, x, H, W)) * 8) = pack8(v);
}

// nearest 2x upsample of the padded a (Ha x Wa), plane blockIdx.y, a pixel per
// thread.  (What follows those planes in the concatenation, the convolution reads
// where it is: ConvGeom::x2.)
__global__ void k_up_pad(const bf16* a, int Ha, int Wa, size_t plane_a, int Bn, int H, int W,
                         size_t plane, bf16* out) {
    const size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= (size_t)Bn * H * W) return;
    const int x = (int)(p % W), r = (int)(p / W), y = r % H, b = r / H;
    const uint4 v = *(const uint4*)(a + (blockIdx.y * plane_a + pad_pos(b, y / 2, x / 2, Ha, Wa)) * 8);
    *(uint4*)(out + (blockIdx.y * plane + pad_pos(b, y, x, H, W)) * 8) = v;
}

// weights [co][tap][ci] -> the direct kernel's [stage][tap][NT / 8][2][8][8]
// (co = 8 group + row, ci = 16 stage + 8 half + e; rows co >= cout are zero)
__global__ void k_conv_wc(const bf16* w, int cin, int cout, int NT, bf16* wc) {
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int ng = NT / 8;
    size_t n = (size_t)(cin / 16) * 9 * NT * 16;
    if (i >= n) return;
    const int e = (int)(i % 8), r = (int)(i / 8 % 8), kh = (int)(i / 64 % 2);
    const int gi = (int)(i / 128 % ng), t = (int)(i / (128 * (size_t)ng) % 9);
    const int j = (int)(i / (128 * (size_t)ng * 9));
    const int co = gi * 8 + r, ci = 16 * j + 8 * kh + e;
    wc[i] = co < cout ? w[((size_t)co * 9 + t) * cin + ci] : __float2bfloat16(0.f);
}

// epilogue of the direct kernel: + bias, optional ReLU; BF16 into the padded
// output (same geometry as the input) and / or FP32 into an unpadded
// [B][H][W][cout_f] buffer
struct ConvOutPadded {
    const float* bias;
    int nbias;
    bf16* y;  // padded or null
    size_t plane;
    float* yf;  // unpadded FP32 or null
    int relu, H, W, npos;
    __device__ int pos(int q) const {
        if (q >= npos) return -1;
        const int Wp = W + 2, Hp = H + 2;
        const int x = q % Wp, r = q / Wp, yy = r % Hp, b = r / Hp;
        if (x < 1 || x > W || yy < 1 || yy > H) return -1;
        return (b * H + yy - 1) * W + (x - 1);
    }
    __device__ void store(int q, int p, int c0, const float (&v)[16]) const {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int c = c0 + 8 * h;
            if (c >= nbias) return;  // a multiple of 8
            const float4 b0 = *(const float4*)(bias + c), b1 = *(const float4*)(bias + c + 4);
            const float b[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
            float o[8];
#pragma unroll
            for (int e = 0; e < 8; e++) {
                const float t = v[8 * h + e] + b[e];
                o[e] = relu ? fmaxf(t, 0.f) : t;
            }
            if (y) {
                bf16 t[8];
#pragma unroll
                for (int e = 0; e < 8; e++) t[e] = __float2bfloat16(o[e]);
                *(uint4*)(y + (c / 8 * plane + q) * 8) = pack8(t);
            }
            if (yf) store8(yf + (size_t)p * nbias + c, o);
        }
    }
};

// the stride-2 layer keeps the im2col GEMM: its input and output padded (the
// border supplies the zeros of the padding)
struct TcConvInPadded {
    const bf16* x;
    int H, W, C, Ho, Wo, stride, plane;
    __device__ const uint4* base() const { return units(x); }
    __device__ TcRow row(int m, int M) const {
        const int xo = m % Wo, r = m / Wo, yo = r % Ho, b = r / Ho;
        return TcRow{(b * (H + 2) + yo * stride) * (W + 2) + xo * stride, m < M ? 1u : 0u};
    }
    __device__ TcPos kpos(int k) const {
        const int ci = k % C, t = k / C;
        return TcPos{t / 3 * (W + 2) + t % 3 + ci / 8 * plane, 0};
    }
};

struct ConvOutToPadded {
    const float* bias;
    bf16* y;
    int relu, Ho, Wo;
    size_t plane;
    __device__ void operator()(int m, int n, const float (&v)[8]) const {
        float o[8];
        bias_relu(bias + n, relu, v, o);
        const int xo = m % Wo, r = m / Wo, yo = r % Ho, b = r / Ho;
        *(uint4*)(y + (n / 8 * plane + pad_pos(b, yo, xo, Ho, Wo)) * 8) = pack8(o);
    }
};

struct Layer {
    int cin, cout, stride, relu;
    size_t woff, boff;  // offsets into the parameter vector
};

}  // namespace rf_cnn_impl

using namespace rf_cnn_impl;

struct rf_cnn {
    int max_batch = 0, H = 0, W = 0;  // input resolution
    std::vector<Layer> layers;        // c1, c2, c3, h16, c4, h8
    size_t n_params = 0;
    float *w = nullptr, *g = nullptr, *m = nullptr, *v = nullptr;  // FP32 master, grad, Adam
    bf16* wb = nullptr;               // BF16 copy used by the kernels
    bf16* wt = nullptr;               // BF16 weights per layer as [ci][tap][co]
    int* d_status = nullptr;          // set by a tensor-core launch whose wait gave up
    int test_first_wait_polls = -1;   // rf_cnn_set_test_wait_limit (-1: the normal limit)
    int step = 0;
    // activations (BF16) and gradients (FP32 / BF16)
    bf16 *x = nullptr, *a1 = nullptr, *a2 = nullptr, *a3 = nullptr, *cat = nullptr, *a4 = nullptr;
    float *o16 = nullptr, *o8 = nullptr;
    float *g_o16 = nullptr, *g_o8 = nullptr, *g_a4 = nullptr, *g_cat = nullptr, *g_a3 = nullptr,
          *g_a2 = nullptr, *g_a1 = nullptr;
    bf16* gb = nullptr;   // BF16 staging of the gradient being propagated
    float* part = nullptr;
    size_t part_floats = 0;
    double* d_loss = nullptr;
    cudaStream_t stream = nullptr;
    uint64_t launches = 0;
    // inference on padded activations (rf_cnn_forward; training keeps the GEMMs)
    bool direct = false;
    bf16* pad[6] = {};  // the allocations: kConvMargin positions, the planes, the margin
    bf16 *xp = nullptr, *a1p = nullptr, *a2p = nullptr, *a3p = nullptr, *upp = nullptr,
         *a4p = nullptr;  // their first planes
    int pad_h = -1, pad_w = -1;  // the frame size whose borders the padded buffers hold zero
    size_t pad_elems[6] = {};    // BF16 elements allocated per padded buffer
    bf16* wc[6] = {};  // per layer, the direct kernel's weight layout (null: c2)
    int nt[6] = {};    // per layer, the direct kernel's N tile
};

namespace rf_cnn_impl {

rf_status cfail(rf_status st, const std::string& msg) {
    return static_cast<rf_status>(rf::set_last_error(st, msg.c_str()));
}

#define CN(call)                                                                      \
    do {                                                                              \
        cudaError_t e__ = (call);                                                     \
        if (e__ != cudaSuccess)                                                       \
            return cfail(e__ == cudaErrorMemoryAllocation ? RF_ERR_OOM : RF_ERR_CUDA,         \
                        std::string(#call ": ") + cudaGetErrorString(e__));            \
    } while (0)

int Ho_of(int H, int s) { return s == 1 ? H : (H + 1) / 2; }

template <int NT, class LA, class LB, class EP>
rf_status tc_launch(rf_cnn* c, int M, int N, int K, LA la, LB lb, EP ep) {
    using S = rf_tc::TcSmem<NT>;
    static bool attr_set = false;
    if (!attr_set) {
        CN(cudaFuncSetAttribute(rf_tc::k_tc_gemm<NT, LA, LB, EP>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, S::kBytes));
        attr_set = true;
    }
    dim3 grid((M + rf_tc::kTM - 1) / rf_tc::kTM, (N + NT - 1) / NT);
    rf_tc::k_tc_gemm<NT, LA, LB, EP><<<grid, rf_tc::kThreads, S::kBytes, c->stream>>>(
        M, N, K, la, lb, ep, c->d_status, c->test_first_wait_polls);
    c->launches++;
    CN(cudaGetLastError());
    return RF_OK;
}

// D[M x N] = A[M x K] B[N x K]^T on the tensor cores
template <class LA, class LB, class EP>
rf_status tc_gemm(rf_cnn* c, int M, int N, int K, LA la, LB lb, EP ep) {
    if (N <= 16) return tc_launch<16>(c, M, N, K, la, lb, ep);
    if (N <= 32) return tc_launch<32>(c, M, N, K, la, lb, ep);
    if (N <= 64) return tc_launch<64>(c, M, N, K, la, lb, ep);
    if (N <= 96) return tc_launch<96>(c, M, N, K, la, lb, ep);
    return tc_launch<128>(c, M, N, K, la, lb, ep);
}

template <int NT>
rf_status wgrad_launch(rf_cnn* c, int M, int N, int K, int kspan, int splits,
                       const rf_tc::WgradGeom& w, TcStoreWGrad ep) {
    using S = rf_tc::WgSmem<NT>;
    static bool attr_set = false;
    if (!attr_set) {
        CN(cudaFuncSetAttribute(rf_tc::k_tc_wgrad<NT, TcStoreWGrad>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, S::kBytes));
        attr_set = true;
    }
    const dim3 grid((M + rf_tc::kTM - 1) / rf_tc::kTM, 1, splits);
    rf_tc::k_tc_wgrad<NT, TcStoreWGrad><<<grid, rf_tc::kThreads, S::kBytes, c->stream>>>(
        M, N, K, kspan, w, ep, c->d_status, c->test_first_wait_polls);
    c->launches++;
    CN(cudaGetLastError());
    return RF_OK;
}

// weight gradient of layer L over K pixels in `splits` parts; returns the
// number of parts actually used through *used
rf_status conv_wgrad(rf_cnn* c, const Layer& L, const rf_tc::WgradGeom& w, int K, int splits,
                     int* used) {
    const int M = 9 * L.cin, N = L.cout;
    const int kspan = ((K + splits - 1) / splits + rf_tc::kTK - 1) / rf_tc::kTK * rf_tc::kTK;
    splits = *used = (K + kspan - 1) / kspan;
    const TcStoreWGrad ep{c->part, M, N};
    if (N <= 16) return wgrad_launch<16>(c, M, N, K, kspan, splits, w, ep);
    if (N <= 32) return wgrad_launch<32>(c, M, N, K, kspan, splits, w, ep);
    if (N <= 64) return wgrad_launch<64>(c, M, N, K, kspan, splits, w, ep);
    return wgrad_launch<96>(c, M, N, K, kspan, splits, w, ep);
}

// forward conv of layer L: x (B x H x W x cin) -> y (BF16) and/or yf (FP32)
rf_status conv_fwd(rf_cnn* c, const Layer& L, const bf16* x, int B, int H, int W, bf16* y,
                   float* yf) {
    int Ho = Ho_of(H, L.stride), Wo = Ho_of(W, L.stride);
    int M = B * Ho * Wo, K = 9 * L.cin;
    TcConvIn la{x, H, W, L.cin, Ho, Wo, L.stride};
    TcRows lb{c->wb + L.woff, K};
    ConvOut ep{c->w + L.boff, y, yf, L.cout, L.relu};
    return tc_gemm(c, M, L.cout, K, la, lb, ep);
}

// the output gradient of layer L (k_grad_in) into c->gb, and its bias gradient
rf_status grad_in(rf_cnn* c, const Layer& L, const float* g, const float* add, const bf16* act,
                  int P) {
    const int nblk = (P + kGradSpan - 1) / kGradSpan;
    if ((size_t)nblk * L.cout > c->part_floats || L.cout > kGradThreads)
        return cfail(RF_ERR_STATE, "cnn: partial buffer too small for the bias gradient");
    k_grad_in<<<nblk, kGradThreads, 0, c->stream>>>(g, add, act, c->gb, P, L.cout, c->part);
    k_reduce_bias<<<L.cout, kGradThreads, 0, c->stream>>>(c->part, nblk, L.cout, c->g + L.boff);
    c->launches += 2;
    CN(cudaGetLastError());
    return RF_OK;
}

// backward of layer L given its output gradient in c->gb (through the ReLU mask):
// the weight gradient, and the input gradient if dx != null
rf_status conv_bwd(rf_cnn* c, const Layer& L, const bf16* x, int B, int H, int W, float* dx) {
    const bf16* dyb = c->gb;
    int Ho = Ho_of(H, L.stride), Wo = Ho_of(W, L.stride);
    int P = B * Ho * Wo, Mw = 9 * L.cin;
    // weight gradient: [tap*cin + ci] x [co] over the pixels, split over K
    int splits = std::max(1, std::min(128, P / 4096));
    int used = 1;
    size_t need = (size_t)splits * L.cout * Mw;
    if (need > c->part_floats) return cfail(RF_ERR_STATE, "cnn: partial buffer too small");
    rf_status rs = conv_wgrad(c, L, rf_tc::WgradGeom{x, dyb, H, W, L.cin, Ho, Wo, L.cout, L.stride},
                              P, splits, &used);
    if (rs != RF_OK) return rs;
    k_reduce_partials<<<blocks_for((size_t)L.cout * Mw), 256, 0, c->stream>>>(
        c->part, used, L.cout * Mw, c->g + L.woff);
    c->launches++;
    if (dx && L.stride == 1) {
        int M = B * H * W, K = 9 * L.cout;
        rs = tc_gemm(c, M, L.cin, K, TcDataGradA{dyb, H, W, L.cout},
                     TcRows{c->wt + L.woff, K}, StoreF32{dx, L.cin});
    } else if (dx) {
        for (int i = 0; i < 4 && rs == RF_OK; i++) {
            const Parity2 q{i >> 1, i & 1};
            const int Hc = (H - q.py + 1) / 2, Wc = (W - q.px + 1) / 2;
            const int K = (q.py + 1) * (q.px + 1) * L.cout;
            if (Hc > 0 && Wc > 0)
                rs = tc_gemm(c, B * Hc * Wc, L.cin, K, TcDataGrad2A{dyb, Hc, Wc, Ho, Wo, L.cout, q},
                             TcTapRows{c->wt + L.woff, L.cout, q},
                             StoreF32Parity{dx, L.cin, H, W, Hc, Wc, q});
        }
    }
    if (rs != RF_OK) return rs;
    CN(cudaGetLastError());
    return RF_OK;
}

rf_status sync_bf16_weights(rf_cnn* c) {
    k_f32_to_bf16<<<blocks_for(c->n_params / 4), 256, 0, c->stream>>>(c->w, c->wb, c->n_params);
    c->launches++;
    for (size_t li = 0; li < c->layers.size(); li++) {
        const Layer& L = c->layers[li];
        k_transpose_w<<<blocks_for((size_t)L.cout * 9 * L.cin), 256, 0, c->stream>>>(
            c->wb + L.woff, L.cin, L.cout, c->wt + L.woff);
        c->launches++;
        if (c->wc[li]) {
            const size_t n = (size_t)(L.cin / 16) * 9 * c->nt[li] * 16;
            k_conv_wc<<<blocks_for(n), 256, 0, c->stream>>>(c->wb + L.woff, L.cin, L.cout,
                                                           c->nt[li], c->wc[li]);
            c->launches++;
        }
    }
    CN(cudaGetLastError());
    return RF_OK;
}

// the input planes of a layer: `split` of them at x, the rest at x2
struct ConvInput {
    const bf16 *x, *x2;
    int split;
};
size_t pad_plane(const rf_cnn* c, int H, int W) {
    return (size_t)c->max_batch * (H + 2) * (W + 2);
}

// one stride-1 layer on the direct kernel
template <int NT, int MT>
rf_status conv3_launch(rf_cnn* c, int li, ConvInput in, int B, int H, int W, bf16* y, float* yf) {
    const Layer& L = c->layers[li];
    using S = rf_tc::ConvSmem<NT, MT>;
    const rf_tc::ConvGeom g{W + 2, B * (H + 2) * (W + 2), L.cin / 16, in.x, in.x2, in.split,
                            pad_plane(c, H, W)};
    const size_t smem = S::bytes(g.Wp);
    static bool attr_set = false;
    if (!attr_set) {
        CN(cudaFuncSetAttribute(rf_tc::k_tc_conv3<NT, MT, ConvOutPadded>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
        attr_set = true;
    }
    if (smem > 227 * 1024) return cfail(RF_ERR_UNSUPPORTED, "cnn: row too long for the direct kernel");
    ConvOutPadded ep{c->w + L.boff, L.cout, y, g.plane, yf, L.relu, H, W, g.npos};
    const int tile = rf_tc::kTM * MT;
    rf_tc::k_tc_conv3<NT, MT, ConvOutPadded>
        <<<(unsigned)((g.npos + tile - 1) / tile), rf_tc::kThreads, smem, c->stream>>>(
            c->wc[li], g, ep, c->d_status, c->test_first_wait_polls);
    c->launches++;
    CN(cudaGetLastError());
    return RF_OK;
}
template <int NT>
rf_status conv3_direct(rf_cnn* c, int li, ConvInput in, int B, int H, int W, bf16* y, float* yf) {
    const long long npos = (long long)B * (H + 2) * (W + 2);
    if (rf::conv_wide_tile(npos, rf_tc::ConvSmem<NT, 2>::bytes(W + 2), rf::sm_count()))
        return conv3_launch<NT, 2>(c, li, in, B, H, W, y, yf);
    return conv3_launch<NT, 1>(c, li, in, B, H, W, y, yf);
}

// inference: padded activations (laid out for this call's frame size, up to
// the allocated one), the stride-1 layers on the direct kernel, the stride-2
// layer on the im2col GEMM
rf_status forward_direct(rf_cnn* c, const float* input, int B, int H, int W) {
    const int H2 = Ho_of(H, 2), W2 = Ho_of(W, 2);
    const Layer &c1 = c->layers[0], &c2 = c->layers[1], &c3 = c->layers[2];
    if (H != c->pad_h || W != c->pad_w) {
        // a new frame size moves the borders: clear the buffers once (the
        // kernels never write a border position of the size they run at)
        for (int k = 0; k < 6; k++)
            CN(cudaMemsetAsync(c->pad[k], 0, c->pad_elems[k] * 2, c->stream));
        c->pad_h = H;
        c->pad_w = W;
    }
    const size_t plane = pad_plane(c, H, W), plane2 = pad_plane(c, H2, W2);
    auto all = [](const bf16* x, const Layer& L) { return ConvInput{x, x, L.cin / 8}; };
    k_pad_input<<<blocks_for((size_t)B * H * W * 2), 256, 0, c->stream>>>(input, B, H, W, plane,
                                                                        c->xp);
    c->launches++;
    rf_status rs = conv3_direct<32>(c, 0, all(c->xp, c1), B, H, W, c->a1p, nullptr);
    if (rs == RF_OK) {
        const int M = B * H2 * W2, K = 9 * c2.cin;
        rs = tc_gemm(c, M, c2.cout, K,
                     TcConvInPadded{c->a1p, H, W, c2.cin, H2, W2, c2.stride, (int)plane},
                     TcRows{c->wb + c2.woff, K},
                     ConvOutToPadded{c->w + c2.boff, c->a2p, c2.relu, H2, W2, plane2});
    }
    if (rs == RF_OK) rs = conv3_direct<96>(c, 2, all(c->a2p, c3), B, H2, W2, c->a3p, nullptr);
    if (rs == RF_OK)
        rs = conv3_direct<16>(c, 3, all(c->a3p, c->layers[3]), B, H2, W2, nullptr, c->o16);
    if (rs != RF_OK) return rs;
    const dim3 up(blocks_for((size_t)B * H * W), c3.cout / 8);
    k_up_pad<<<up, 256, 0, c->stream>>>(c->a3p, H2, W2, plane2, B, H, W, plane, c->upp);
    c->launches++;
    rs = conv3_direct<64>(c, 4, ConvInput{c->upp, c->a1p, c3.cout / 8}, B, H, W, c->a4p, nullptr);
    if (rs == RF_OK) rs = conv3_direct<16>(c, 5, all(c->a4p, c->layers[5]), B, H, W, nullptr, c->o8);
    if (rs != RF_OK) return rs;
    CN(cudaGetLastError());
    return RF_OK;
}

rf_status forward(rf_cnn* c, const float* input, int B, int H, int W) {
    const Layer &c1 = c->layers[0], &c2 = c->layers[1], &c3 = c->layers[2], &h16 = c->layers[3],
                &c4 = c->layers[4], &h8 = c->layers[5];
    size_t nin = (size_t)B * H * W * 16;
    k_f32_to_bf16<<<blocks_for(nin / 4), 256, 0, c->stream>>>(input, c->x, nin);
    c->launches++;
    int H2 = Ho_of(H, 2), W2 = Ho_of(W, 2);
    rf_status rs = conv_fwd(c, c1, c->x, B, H, W, c->a1, nullptr);
    if (rs == RF_OK) rs = conv_fwd(c, c2, c->a1, B, H, W, c->a2, nullptr);
    if (rs == RF_OK) rs = conv_fwd(c, c3, c->a2, B, H2, W2, c->a3, nullptr);
    if (rs == RF_OK) rs = conv_fwd(c, h16, c->a3, B, H2, W2, nullptr, c->o16);
    if (rs != RF_OK) return rs;
    size_t ncat = (size_t)B * H * W * (c3.cout + c1.cout);
    k_concat_up<<<blocks_for(ncat / 8), 256, 0, c->stream>>>(c->a3, H2, W2, c3.cout, c->a1, c1.cout,
                                                         B, H, W, c->cat);
    c->launches++;
    rs = conv_fwd(c, c4, c->cat, B, H, W, c->a4, nullptr);
    if (rs == RF_OK) rs = conv_fwd(c, h8, c->a4, B, H, W, nullptr, c->o8);
    return rs;
}

rf_status backward(rf_cnn* c, int B, int H, int W) {
    const Layer &c1 = c->layers[0], &c2 = c->layers[1], &c3 = c->layers[2], &h16 = c->layers[3],
                &c4 = c->layers[4], &h8 = c->layers[5];
    const int H2 = Ho_of(H, 2), W2 = Ho_of(W, 2), P = B * H * W, P2 = B * H2 * W2;
    const size_t n3 = (size_t)P2 * c3.cout, n1 = (size_t)P * c1.cout;
    // heads (linear)
    rf_status rs = grad_in(c, h8, c->g_o8, nullptr, nullptr, P);
    if (rs == RF_OK) rs = conv_bwd(c, h8, c->a4, B, H, W, c->g_a4);
    if (rs == RF_OK) rs = grad_in(c, c4, c->g_a4, nullptr, c->a4, P);
    if (rs == RF_OK) rs = conv_bwd(c, c4, c->cat, B, H, W, c->g_cat);
    if (rs != RF_OK) return rs;
    // split the concat gradient: g_a3 = up^T(g_cat[:96]), g_a1 = g_cat[96:]
    k_concat_up_grad<<<blocks_for(std::max(n3, n1) / 4), 256, 0, c->stream>>>(
        c->g_cat, H2, W2, c3.cout, c1.cout, B, H, W, c->g_a3, c->g_a1);
    c->launches++;
    // 1/16 head adds into g_a3
    float* tmp = c->g_a2;  // scratch for the head's input gradient (same size as g_a3)
    rs = grad_in(c, h16, c->g_o16, nullptr, nullptr, P2);
    if (rs == RF_OK) rs = conv_bwd(c, h16, c->a3, B, H2, W2, tmp);
    if (rs == RF_OK) rs = grad_in(c, c3, c->g_a3, tmp, c->a3, P2);
    if (rs == RF_OK) rs = conv_bwd(c, c3, c->a2, B, H2, W2, c->g_a2);
    if (rs == RF_OK) rs = grad_in(c, c2, c->g_a2, nullptr, c->a2, P2);
    // c2's input gradient adds into g_a1 (which holds the skip part): use tmp2
    float* tmp2 = c->g_a4;  // free now, large enough (B*H*W*64 >= B*H*W*32)
    if (rs == RF_OK) rs = conv_bwd(c, c2, c->a1, B, H, W, tmp2);
    if (rs == RF_OK) rs = grad_in(c, c1, c->g_a1, tmp2, c->a1, P);
    if (rs == RF_OK) rs = conv_bwd(c, c1, c->x, B, H, W, nullptr);
    if (rs != RF_OK) return rs;
    CN(cudaGetLastError());
    return RF_OK;
}

// whether the direct kernel's shared memory fits rows of width W
bool direct_fits(int W) {
    const size_t lim = 227 * 1024;
    return W + 2 < rf_tc::kConvMargin / 2 && rf_tc::ConvSmem<32, 1>::bytes(W + 2) <= lim &&
           rf_tc::ConvSmem<64, 1>::bytes(W + 2) <= lim &&
           rf_tc::ConvSmem<96, 1>::bytes(W + 2) <= lim;
}

}  // namespace rf_cnn_impl

extern "C" {

rf_status rf_cnn_create(int max_batch, int height, int width, unsigned long long seed,
                        rf_cnn** out) {
    if (!out || max_batch < 1 || height < 2 || width < 2 || (long long)max_batch * height * width > (1LL << 26))
        return cfail(RF_ERR_INVALID_ARG, "rf_cnn_create: bad size");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev < 1)
        return cfail(RF_ERR_NO_DEVICE, "rf_cnn_create: no CUDA device");
    rf_cnn* c = new rf_cnn();
    c->max_batch = max_batch;
    c->H = height;
    c->W = width;
    const int spec[6][4] = {{16, 32, 1, 1}, {32, 96, 2, 1}, {96, 96, 1, 1},
                            {96, 8, 1, 0},  {128, 64, 1, 1}, {64, 8, 1, 0}};
    size_t off = 0;
    for (auto& s : spec) {
        Layer L{s[0], s[1], s[2], s[3], 0, 0};
        L.woff = off;
        off += (size_t)L.cout * 9 * L.cin;
        L.boff = off;
        off += L.cout;
        c->layers.push_back(L);
    }
    c->n_params = off;
    // He-normal initialization from a seeded generator (Box-Muller on a
    // 64-bit LCG), biases zero
    std::vector<float> hw(off, 0.0f);
    uint64_t st = seed * 6364136223846793005ULL + 1442695040888963407ULL;
    auto uni = [&]() {
        st = st * 6364136223846793005ULL + 1442695040888963407ULL;
        return ((st >> 11) + 0.5) / 9007199254740992.0;
    };
    for (const Layer& L : c->layers) {
        double sd = std::sqrt(2.0 / (9.0 * L.cin)) * (L.relu ? 1.0 : 0.1);
        for (size_t i = 0; i < (size_t)L.cout * 9 * L.cin; i++) {
            double u1 = uni(), u2 = uni();
            hw[L.woff + i] = (float)(sd * std::sqrt(-2.0 * std::log(u1)) * std::cos(6.283185307179586 * u2));
        }
    }
    const size_t B = max_batch, P = (size_t)height * width;
    const size_t P2 = (size_t)((height + 1) / 2) * ((width + 1) / 2);
    cudaError_t e = cudaSuccess;
    auto alloc = [&](auto** p, size_t bytes) {
        if (e == cudaSuccess) e = rf::dev_malloc((void**)p, bytes);
    };
    alloc(&c->w, off * 4); alloc(&c->g, off * 4); alloc(&c->m, off * 4); alloc(&c->v, off * 4);
    alloc(&c->wb, off * 2);
    alloc(&c->wt, off * 2);
    alloc(&c->d_status, sizeof(int));
    alloc(&c->x, B * P * 16 * 2); alloc(&c->a1, B * P * 32 * 2); alloc(&c->a2, B * P2 * 96 * 2);
    alloc(&c->a3, B * P2 * 96 * 2); alloc(&c->cat, B * P * 128 * 2); alloc(&c->a4, B * P * 64 * 2);
    alloc(&c->o16, B * P2 * 8 * 4); alloc(&c->o8, B * P * 8 * 4);
    alloc(&c->g_o16, B * P2 * 8 * 4); alloc(&c->g_o8, B * P * 8 * 4);
    alloc(&c->g_a4, B * P * 64 * 4); alloc(&c->g_cat, B * P * 128 * 4);
    alloc(&c->g_a3, B * P2 * 96 * 4); alloc(&c->g_a2, B * P2 * 96 * 4);
    alloc(&c->g_a1, B * P * 32 * 4); alloc(&c->gb, B * P * 128 * 2);
    c->part_floats = (size_t)256 * 96 * 9 * 96;  // chunks x largest cout x 9 cin
    alloc(&c->part, c->part_floats * 4);
    alloc(&c->d_loss, sizeof(double));
    // inference on padded activations: on unless RF_CNN_DIRECT=0 (or rows too long)
    const char* de = std::getenv("RF_CNN_DIRECT");
    c->direct = !(de && de[0] == '0') && direct_fits(width);
    const size_t PP = (size_t)(height + 2) * (width + 2);
    const size_t PP2 = (size_t)((height + 1) / 2 + 2) * ((width + 1) / 2 + 2);
    if (c->direct) {
        const size_t elems[6] = {B * PP * 16, B * PP * 32, B * PP2 * 96,
                                 B * PP2 * 96, B * PP * 96, B * PP * 64};
        bf16** first[6] = {&c->xp, &c->a1p, &c->a2p, &c->a3p, &c->upp, &c->a4p};
        for (int k = 0; k < 6; k++) {
            // cleared before the first call (forward_direct, per frame size)
            c->pad_elems[k] = elems[k] + 2 * rf_tc::kConvMargin * 8;
            alloc(&c->pad[k], c->pad_elems[k] * 2);
            *first[k] = c->pad[k] + rf_tc::kConvMargin * 8;
        }
        const int nts[6] = {32, 0, 96, 16, 64, 16};  // c2 (stride 2) keeps the GEMM
        for (int li = 0; li < 6; li++)
            if (nts[li]) {
                c->nt[li] = nts[li];
                alloc(&c->wc[li], (size_t)(c->layers[li].cin / 16) * 9 * nts[li] * 16 * 2);
            }
    }
    if (e == cudaSuccess) e = cudaMemcpy(c->w, hw.data(), off * 4, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemset(c->m, 0, off * 4);
    if (e == cudaSuccess) e = cudaMemset(c->v, 0, off * 4);
    if (e == cudaSuccess) e = cudaMemset(c->g, 0, off * 4);
    if (e != cudaSuccess) {
        rf_cnn_destroy(c);
        return cfail(RF_ERR_OOM, std::string("rf_cnn_create: ") + cudaGetErrorString(e));
    }
    if (cudaMemset(c->d_status, 0, sizeof(int)) != cudaSuccess) {
        rf_cnn_destroy(c);
        return cfail(RF_ERR_CUDA, "rf_cnn_create: status init");
    }
    rf_status rs = sync_bf16_weights(c);
    // the initialisation above ran on the legacy default stream; a stream
    // set later (rf_cnn_set_stream) may be non-blocking: finish it now
    if (rs == RF_OK && cudaDeviceSynchronize() != cudaSuccess)
        rs = cfail(RF_ERR_CUDA, "rf_cnn_create: initialisation");
    if (rs != RF_OK) {
        rf_cnn_destroy(c);
        return rs;
    }
    *out = c;
    return RF_OK;
}

rf_status rf_cnn_destroy(rf_cnn* c) {
    if (!c) return RF_OK;
    cudaDeviceSynchronize();
    for (void* p : {(void*)c->wt, (void*)c->d_status}) if (p) cudaFree(p);
    for (void* p : {(void*)c->w, (void*)c->g, (void*)c->m, (void*)c->v, (void*)c->wb, (void*)c->x,
                    (void*)c->a1, (void*)c->a2, (void*)c->a3, (void*)c->cat, (void*)c->a4,
                    (void*)c->o16, (void*)c->o8, (void*)c->g_o16, (void*)c->g_o8, (void*)c->g_a4,
                    (void*)c->g_cat, (void*)c->g_a3, (void*)c->g_a2, (void*)c->g_a1, (void*)c->gb,
                    (void*)c->part, (void*)c->d_loss, (void*)c->pad[0], (void*)c->pad[1],
                    (void*)c->pad[2], (void*)c->pad[3], (void*)c->pad[4], (void*)c->pad[5]})
        if (p) cudaFree(p);
    for (bf16* p : c->wc)
        if (p) cudaFree(p);
    delete c;
    return RF_OK;
}

int rf_cnn_num_params(const rf_cnn* c) { return c ? (int)c->n_params : -1; }

rf_status rf_cnn_set_stream(rf_cnn* c, void* stream) {
    if (!c) return cfail(RF_ERR_INVALID_ARG, "rf_cnn_set_stream: null");
    c->stream = static_cast<cudaStream_t>(stream);
    return RF_OK;
}

rf_status rf_cnn_get_params(rf_cnn* c, float* host) {
    if (!c || !host) return cfail(RF_ERR_INVALID_ARG, "rf_cnn_get_params: null");
    CN(cudaStreamSynchronize(c->stream));
    CN(cudaMemcpy(host, c->w, c->n_params * 4, cudaMemcpyDeviceToHost));
    return RF_OK;
}

rf_status rf_cnn_set_params(rf_cnn* c, const float* host) {
    if (!c || !host) return cfail(RF_ERR_INVALID_ARG, "rf_cnn_set_params: null");
    // on the network's stream, ahead of the conversion kernels that read it
    CN(cudaMemcpyAsync(c->w, host, c->n_params * 4, cudaMemcpyHostToDevice, c->stream));
    return sync_bf16_weights(c);
}

rf_status rf_cnn_get_grads(rf_cnn* c, float* host) {
    if (!c || !host) return cfail(RF_ERR_INVALID_ARG, "rf_cnn_get_grads: null");
    CN(cudaStreamSynchronize(c->stream));
    CN(cudaMemcpy(host, c->g, c->n_params * 4, cudaMemcpyDeviceToHost));
    return RF_OK;
}

static rf_status check_batch(rf_cnn* c, int B, int H, int W) {
    if (B < 1 || B > c->max_batch || H > c->H || W > c->W || H < 2 || W < 2)
        return cfail(RF_ERR_INVALID_ARG, "rf_cnn: batch or size beyond the allocation");
    return RF_OK;
}

rf_status rf_cnn_forward(rf_cnn* c, const float* input, int B, int H, int W, float* out16,
                         float* out8) {
    rf::NvtxRange range("rf_cnn_forward");
    if (!c || !input) return cfail(RF_ERR_INVALID_ARG, "rf_cnn_forward: null");
    rf_status rs = check_batch(c, B, H, W);
    if (rs == RF_OK)
        rs = c->direct ? forward_direct(c, input, B, H, W) : forward(c, input, B, H, W);
    if (rs != RF_OK) return rs;
    int H2 = (H + 1) / 2, W2 = (W + 1) / 2;
    if (out16)
        CN(cudaMemcpyAsync(out16, c->o16, (size_t)B * H2 * W2 * 8 * 4, cudaMemcpyDeviceToDevice,
                           c->stream));
    if (out8)
        CN(cudaMemcpyAsync(out8, c->o8, (size_t)B * H * W * 8 * 4, cudaMemcpyDeviceToDevice,
                           c->stream));
    return RF_OK;
}

rf_status rf_cnn_backward(rf_cnn* c, const float* input, const float* tgt16, const float* mask16,
                          const float* tgt8, const float* mask8, int B, int H, int W,
                          const float* weights, double* loss) {
    rf::NvtxRange range("rf_cnn_backward");
    if (!c || !input || !tgt16 || !mask16 || !tgt8 || !mask8 || !weights)
        return cfail(RF_ERR_INVALID_ARG, "rf_cnn_backward: null");
    rf_status rs = check_batch(c, B, H, W);
    if (rs == RF_OK) rs = forward(c, input, B, H, W);
    if (rs != RF_OK) return rs;
    int H2 = (H + 1) / 2, W2 = (W + 1) / 2;
    int P8 = B * H * W, P16 = B * H2 * W2;
    CN(cudaMemsetAsync(c->d_loss, 0, sizeof(double), c->stream));
    k_l1_loss<<<blocks_for(P16), 256, 0, c->stream>>>((const float4*)c->o16, tgt16, mask16, P16,
                                                      weights[0], weights[1], weights[2],
                                                      1.0f / P16, (float4*)c->g_o16, c->d_loss);
    k_l1_loss<<<blocks_for(P8), 256, 0, c->stream>>>((const float4*)c->o8, tgt8, mask8, P8,
                                                     weights[0], weights[1], weights[2], 1.0f / P8,
                                                     (float4*)c->g_o8, c->d_loss);
    c->launches += 2;
    rs = backward(c, B, H, W);
    if (rs != RF_OK) return rs;
    if (loss) {
        CN(cudaMemcpyAsync(loss, c->d_loss, sizeof(double), cudaMemcpyDeviceToHost, c->stream));
        CN(cudaStreamSynchronize(c->stream));
    }
    return RF_OK;
}

rf_status rf_cnn_adam_step(rf_cnn* c, float lr, float beta1, float beta2, float eps) {
    rf::NvtxRange range("rf_cnn_adam_step");
    if (!c) return cfail(RF_ERR_INVALID_ARG, "rf_cnn_adam_step: null");
    c->step++;
    float c1 = 1.0f - std::pow(beta1, (float)c->step);
    float c2 = 1.0f - std::pow(beta2, (float)c->step);
    k_adam<<<blocks_for(c->n_params), 256, 0, c->stream>>>(c->w, c->g, c->m, c->v, c->n_params, lr,
                                                           beta1, beta2, eps, c1, c2);
    c->launches++;
    CN(cudaGetLastError());
    return sync_bf16_weights(c);
}

uint64_t rf_cnn_kernel_launches(const rf_cnn* c) { return c ? c->launches : 0; }

rf_status rf_cnn_status(rf_cnn* c, int* gave_up) {
    if (!c || !gave_up) return cfail(RF_ERR_INVALID_ARG, "rf_cnn_status: null");
    int v = 0;
    CN(cudaMemcpyAsync(&v, c->d_status, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    CN(cudaStreamSynchronize(c->stream));
    if (v) CN(cudaMemsetAsync(c->d_status, 0, sizeof(int), c->stream));
    *gave_up = v;
    return RF_OK;
}

rf_status rf_cnn_set_test_wait_limit(rf_cnn* c, int polls) {
    if (!c) return cfail(RF_ERR_INVALID_ARG, "rf_cnn_set_test_wait_limit: null");
    c->test_first_wait_polls = polls < 0 ? -1 : polls;
    return RF_OK;
}

}  // extern "C"
