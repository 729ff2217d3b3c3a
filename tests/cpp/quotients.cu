// Compares the quotients and roots of rf_packed.cuh, one value and the halves of two,
// with IEEE division and square root.  Prints "<what> <compared> <differing>" per
// comparison.
#include <cstdio>

#include "rf_packed.cuh"

using namespace rf;

namespace quotients {

__device__ __forceinline__ bool same(float a, float b) {
    return __float_as_uint(a) == __float_as_uint(b);
}
__device__ __forceinline__ unsigned long long mix(unsigned long long z) {  // splitmix64
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

struct Tally {
    unsigned long long n = 0, bad = 0;
    __device__ void check(bool ok) {
        n++;
        bad += !ok;
    }
    __device__ void done(unsigned long long* out) const {
        atomicAdd(out, n);
        atomicAdd(out + 1, bad);
    }
};

// -(n / d) and -(d / n), alone and as the halves of two
__device__ void compare(float n, float d, Tally& t) {
    const float q0 = neg_quot(n, d, neg_recip(d)), q1 = neg_quot(d, n, neg_recip(n));
    const f2 den = mk2(d, n), q = neg_quot(mk2(n, d), den, neg_recip(den));
    const float e0 = -__fdiv_rn(n, d), e1 = -__fdiv_rn(d, n);
    t.check(same(q0, e0) && same(q1, e1) && same(q.x, e0) && same(q.y, e1));
}

// the reciprocals of every significand, at three exponents
__global__ void k_reciprocals(unsigned long long* out) {
    Tally t;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < 1u << 23; i += gridDim.x * blockDim.x)
        for (unsigned e : {127u, 127u - 49u, 127u + 119u}) {
            const float d = __uint_as_float(e << 23 | i);
            const f2 r = neg_recip(mk2(d, -d));
            const float want = -__fdiv_rn(1.0f, d);
            t.check(same(neg_recip(d), want) && same(r.x, want) && same(r.y, -want));
        }
    t.done(out);
}

// every pair of significands whose quotient is nearest a tie: n 2^s = d x + r with x odd
// in [2^24, 2^25) (x / 2 between two significands), |r| <= 3; s = 24: n >= d, 25: n < d
__global__ void k_near_ties(unsigned long long* out) {
    Tally t;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < 1u << 23; i += gridDim.x * blockDim.x) {
        const unsigned D = 1u << 23 | i;
        const int z = D & 1 ? 0 : D & 2 ? 1 : 2;  // factors of two; from 2 on no such r
        if (z == 2) continue;
        const unsigned odd = D >> z;
        unsigned inv = odd;  // 1 / odd modulo 2^32 (Newton)
        for (int k = 0; k < 4; k++) inv *= 2u - odd * inv;
        for (int s = 24; s <= 25; s++)
            for (int r = -3; r <= 3; r++) {
                if (r == 0 || (z == 0 ? r % 2 == 0 : r != 2 && r != -2)) continue;
                const unsigned period = 1u << (s - z);
                const unsigned x0 = ((unsigned)-(r >> z) * inv) & (period - 1u);
                for (unsigned x = x0; x < 1u << 25; x += period) {
                    if (x < 1u << 24) continue;
                    const unsigned long long p = (unsigned long long)((long long)D * x + r);
                    const unsigned long long n = p >> s;
                    if ((n << s) != p || n < 1u << 23 || n >= 1u << 24) continue;
                    const unsigned h = (unsigned)mix(D * 64ull + s * 8 + r);
                    // at exponents of their own, within the quotients' range
                    const float a = ldexpf((float)n, (int)(h % 41) - 20);
                    const float b = ldexpf((float)D, (int)(h / 64 % 41) - 20);
                    compare(h >> 31 ? -a : a, h >> 30 & 1 ? -b : b, t);
                }
            }
    }
    t.done(out);
}

// any bits: whatever the guard lets pass, and is finite, is IEEE's
__global__ void k_guarded(unsigned long long* out, int rounds) {
    Tally t;
    const unsigned id = blockIdx.x * blockDim.x + threadIdx.x;
    for (int k = 0; k < rounds; k++) {
        const unsigned long long b = mix((unsigned long long)id * rounds + k);
        float n = __uint_as_float((unsigned)b), d = __uint_as_float((unsigned)(b >> 32));
        if (k % 8 == 0) n = __uint_as_float((unsigned)b & 0x80000000u);  // a zero
        if (k % 2) {  // most within the range
            n = __uint_as_float((unsigned)b & 0x9FFFFFFFu | 0x20000000u);
            d = __uint_as_float((unsigned)(b >> 32) & 0x9FFFFFFFu | 0x20000000u);
        }
        const float q = neg_quot(n, d, neg_recip(d)), want = -__fdiv_rn(n, d);
        const f2 den = mk2(d, d), q2 = neg_quot(mk2(n, n), den, neg_recip(den));
        QuotientGuard g;
        g.div(d);
        if (d > 0.0f) g.quot(q);
        else g.quot_nonzero(q);
        if (g.ok() && isfinite(q)) t.check(same(q, want) && same(q2.x, want) && same(q2.y, want));
        const float a = fabsf(n), root = sqrt_rn(a);
        const f2 root2 = sqrt_rn(mk2(a, a));
        QuotientGuard h;
        h.quot(root);
        if (h.ok() && isfinite(root))
            t.check(same(root, __fsqrt_rn(a)) && same(root2.x, root) && same(root2.y, root));
    }
    t.done(out);
}

// the roots of every significand, at both parities and the ends of the range
__global__ void k_roots(unsigned long long* out) {
    Tally t;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < 1u << 23; i += gridDim.x * blockDim.x)
        for (unsigned e : {127u, 128u, 27u, 28u, 253u, 254u}) {
            const float a = __uint_as_float(e << 23 | i), want = __fsqrt_rn(a);
            const f2 r = sqrt_rn(mk2(a, a));
            t.check(same(sqrt_rn(a), want) && same(r.x, want) && same(r.y, want));
        }
    t.done(out);
}

// a packed product and the sum it goes into are rounded one after the other
__global__ void k_products(unsigned long long* out, int rounds) {
    Tally t;
    const unsigned id = blockIdx.x * blockDim.x + threadIdx.x;
    for (int k = 0; k < rounds; k++) {
        const unsigned long long b = mix((unsigned long long)id * rounds + k);
        auto one = [&](int s) { return __uint_as_float(0x3F800000u | (unsigned)(b >> s) & 0x7FFFFFu); };
        const float x = one(0), y = one(23), z = -one(40) * 1.5f;
        const f2 v = mk2(x, y) * mk2(y, y) + mk2(z, z), w = mk2(x, y) * mk2(y, x) - mk2(z, y);
        t.check(same(v.x, __fadd_rn(__fmul_rn(x, y), z)) && same(v.y, __fadd_rn(__fmul_rn(y, y), z)) &&
                same(w.x, __fsub_rn(__fmul_rn(x, y), z)) && same(w.y, __fsub_rn(__fmul_rn(y, x), y)));
    }
    t.done(out);
}

}  // namespace quotients

using namespace quotients;

int main() {
    unsigned long long* out;
    if (cudaMallocManaged(&out, 2 * sizeof *out) != cudaSuccess) return 2;
    auto report = [&](const char* what, auto&& launch) {
        out[0] = out[1] = 0;
        launch();
        if (cudaDeviceSynchronize() != cudaSuccess) return false;
        std::printf("%s %llu %llu\n", what, out[0], out[1]);
        return true;
    };
    bool ok = report("reciprocals", [&] { k_reciprocals<<<1024, 256>>>(out); });
    ok = ok && report("near_ties", [&] { k_near_ties<<<1024, 256>>>(out); });
    ok = ok && report("guarded", [&] { k_guarded<<<1024, 256>>>(out, 256); });
    ok = ok && report("roots", [&] { k_roots<<<1024, 256>>>(out); });
    ok = ok && report("products", [&] { k_products<<<1024, 256>>>(out, 64); });
    cudaFree(out);
    return ok ? 0 : 3;
}
