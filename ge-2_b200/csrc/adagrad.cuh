// The Adagrad step of one element or of a few, shared by the kernels that update rows.
#pragma once
#include "common.cuh"

namespace ge2 {

constexpr float kAdagradEps = 1e-10f;  // literal in cpp/src/data/batch.cpp:266 of the reference project

// state += g*g ; delta = -lr * g / (sqrt(state) + eps), one IEEE operation at a time
__device__ __forceinline__ void adagrad_elem(float g, float& state, float& delta, float& upd, float neg_lr) {
    upd = __fmul_rn(g, g);
    state = __fadd_rn(state, upd);
    const float den = __fadd_rn(__fsqrt_rn(state), kAdagradEps);
    delta = __fmul_rn(neg_lr, __fdiv_rn(g, den));
}

// -g / (sqrt(s) + eps) with both operations rounded correctly, for s in [2^-40, 2^60], g zero or at least 2^-94 in size, and a denominator d
// (an output) whose significand is not all ones.
// Square root and quotient by the iterations of P. Markstein (IA-64 and Elementary Functions, 2000): from y ~ 1 / sqrt(s), the pair
// (r, h) = (s y, y / 2) is refined once together, and the last correction r + (s - r r) h, whose remainder is exact, rounds correctly.  2 h then
// is 1 / (r + eps) to 2^-13 or better (that is what the lower bound on s is for); two Newton steps round the reciprocal correctly, unless
// the significand is all ones, and q + (g - q d) / d does the quotient, provided that it is a normal number: the last sum would break a tie
// between two subnormal ones the wrong way.  That is what the bound on g is for (d is at most 2^30); the remainder is a multiple of 2^-141 then.
// Compared with the IEEE operations on 64 quotients for every significand of s at both parities of the exponent and on 2^34 random pairs.
__device__ __forceinline__ float2 neg_step2(float2 g, float2 s, float2& d) {
    float2 y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y.x) : "f"(s.x));
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y.y) : "f"(s.y));
    float2 r = mul2(s, y), nh = mul2(y, both(-0.5f));  // (the negative of h, and of everything that is made from it)
    const float2 u = fma2(r, nh, both(0.5f));
    r = fma2(r, u, r), nh = fma2(nh, u, nh);
    r = fma2(fma2(r, r, mul2(s, both(-1.f))), nh, r);
    d = add2(r, both(kAdagradEps));
    float2 ny = add2(nh, nh);
    ny = fma2(ny, fma2(d, ny, both(1.f)), ny);
    ny = fma2(ny, fma2(d, ny, both(1.f)), ny);
    const float2 nq = mul2(g, ny);
    return fma2(fma2(d, nq, g), ny, nq);
}

// (called: what the other does not cover is rare, and this code long)
static __device__ __noinline__ float2 adagrad_one(float g, float state, float neg_lr) {
    float2 r = make_float2(state, 0.f);
    float upd;
    adagrad_elem(g, r.x, r.y, upd, neg_lr);
    return r;
}

// adagrad_elem on N elements (one, or an even number), the same results: an element takes 11 instructions of the FMA pipe in straight-line code,
// where the IEEE functions test and branch for every one, one behind the other.  The finish kernel at 10 000 edges, 2 x 10 000 negatives, ComplEx
// 100: 18.9 to 17.7 us; 50 000 and 50 000, Dot 100: 81.4 to 77.2; 100 000 and 2 x 200 000, DistMult 128: 211 to 203.
template <int N>
__device__ __forceinline__ void adagrad_elems(const float (&g)[N], float (&state)[N], float (&delta)[N], float (&upd)[N], float neg_lr) {
    if constexpr (N == 1) {
        adagrad_elem(g[0], state[0], delta[0], upd[0], neg_lr);
    } else {
        bool fine = true;
        uint32_t least = 0xFFFFFFFFu, most = 0u;  // of twice the bits of |g|, less one (the largest value for a zero); of the denominators' significands
        float2 s[N / 2];
#pragma unroll
        for (int k = 0; k < N / 2; k++) {
            // (scalar where a product is added to something: a packed product and a packed sum were seen to come out as one fused operation)
            const float2 x = make_float2(g[2 * k], g[2 * k + 1]), up = make_float2(__fmul_rn(x.x, x.x), __fmul_rn(x.y, x.y));
            s[k] = make_float2(__fadd_rn(state[2 * k], up.x), __fadd_rn(state[2 * k + 1], up.y));
            fine = fine && s[k].x >= 0x1p-40f && s[k].x <= 0x1p60f && s[k].y >= 0x1p-40f && s[k].y <= 0x1p60f;
            least = min(least, min(2u * __float_as_uint(x.x) - 1u, 2u * __float_as_uint(x.y) - 1u));
            float2 d;
            const float2 nq = neg_step2(x, s[k], d);
            most = max(most, max(__float_as_uint(d.x) << 9, __float_as_uint(d.y) << 9));
            upd[2 * k] = up.x, upd[2 * k + 1] = up.y, delta[2 * k] = __fmul_rn(-neg_lr, nq.x), delta[2 * k + 1] = __fmul_rn(-neg_lr, nq.y);
        }
        fine = fine && least >= 2u * 0x10800000u - 1u && most < 0xFFFFFE00u;  // 2^-94; all ones
        if (__builtin_expect(!fine, 0)) {
#pragma unroll
            for (int k = 0; k < N; k++) {
                const float2 r = adagrad_one(g[k], state[k], neg_lr);
                state[k] = r.x, delta[k] = r.y;
            }
        } else {
#pragma unroll
            for (int k = 0; k < N / 2; k++) state[2 * k] = s[k].x, state[2 * k + 1] = s[k].y;
        }
    }
}

}  // namespace ge2
