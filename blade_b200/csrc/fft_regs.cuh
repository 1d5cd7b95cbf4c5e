// Register-blocked DFTs on pairs of complex values: two polarisations of a sample,
// or two spectra of a single-polarisation block, transformed together.
//
// A pair keeps its real parts in one FP32x2 register pair and its imaginary parts in
// another, so every add, subtract and product with a shared twiddle is one packed
// instruction for both members, a product with -i is a renaming, and one twiddle
// (one recurrence) serves two transforms.
#pragma once

#include "common.cuh"

namespace bb {
namespace fft {

struct c2 {
    float2 re, im;  // .x: first member of the pair, .y: second
};

__device__ __forceinline__ c2 add(const c2& a, const c2& b) {
    return {__fadd2_rn(a.re, b.re), __fadd2_rn(a.im, b.im)};
}
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
__device__ __forceinline__ c2 sub(const c2& a, const c2& b) { return {sub2(a.re, b.re), sub2(a.im, b.im)}; }
// a + (-i) b and a - (-i) b
__device__ __forceinline__ c2 add_mi(const c2& a, const c2& b) { return {__fadd2_rn(a.re, b.im), sub2(a.im, b.re)}; }
__device__ __forceinline__ c2 sub_mi(const c2& a, const c2& b) { return {sub2(a.re, b.im), __fadd2_rn(a.im, b.re)}; }
__device__ __forceinline__ float2 dup(float v) { return make_float2(v, v); }
// a * w for one twiddle w shared by the pair: each member rounds as
// (fma(a.re, w.re, -(a.im w.im)), fma(a.re, w.im, a.im w.re))
__device__ __forceinline__ c2 mul(const c2& a, float wr, float wi) {
    return {__ffma2_rn(a.re, dup(wr), __fmul2_rn(a.im, dup(-wi))), __ffma2_rn(a.re, dup(wi), __fmul2_rn(a.im, dup(wr)))};
}
__device__ __forceinline__ c2 mul(const c2& a, float2 w) { return mul(a, w.x, w.y); }
// a * (w + l) for a constant w rounded to FP32 and what the rounding left out, l
__device__ __forceinline__ c2 mul_fine(const c2& a, float wr, float wi, float lr, float li) {
    const float2 re = __ffma2_rn(a.re, dup(lr), __fmul2_rn(a.im, dup(-li)));
    const float2 im = __ffma2_rn(a.re, dup(li), __fmul2_rn(a.im, dup(lr)));
    return {__ffma2_rn(a.re, dup(wr), __ffma2_rn(a.im, dup(-wi), re)),
            __ffma2_rn(a.re, dup(wi), __ffma2_rn(a.im, dup(wr), im))};
}

__device__ __forceinline__ void dft4(c2& a, c2& b, c2& c, c2& d) {
    const c2 e0 = add(a, c), e1 = sub(a, c), o0 = add(b, d), o1 = sub(b, d);
    a = add(e0, o0);
    b = add_mi(e1, o1);
    c = sub(e0, o0);
    d = sub_mi(e1, o1);
}

// In-place R-point DFT, natural order in and out.  FINE (R = 16): with twice the precision
// in its constants.  Rounded ones are short by 2.8e-8 (cos pi / 8) and 1.7e-8 (sqrt 1 / 2), which
// every output of a stage shares: two stages of radix 16 put 1.3e-8 on the mean power of a
// spectrum, which sums over windows and antennas do not average out.
template <int R, bool FINE = false>
__device__ __forceinline__ void dft(c2 (&v)[R]) {
    constexpr float h = 0.70710678118654752f;
    if constexpr (R == 2) {
        const c2 a = v[0], b = v[1];
        v[0] = add(a, b);
        v[1] = sub(a, b);
    } else if constexpr (R == 4) {
        dft4(v[0], v[1], v[2], v[3]);
    } else if constexpr (R == 8) {
        // X[k] = E[k mod 4] + w8^k O[k mod 4]
        dft4(v[0], v[2], v[4], v[6]);
        dft4(v[1], v[3], v[5], v[7]);
        const c2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1], o2 = v[5];
        const c2 o1 = mul(v[3], h, -h), o3 = mul(v[7], -h, -h);
        v[0] = add(e0, o0);
        v[4] = sub(e0, o0);
        v[1] = add(e1, o1);
        v[5] = sub(e1, o1);
        v[2] = add_mi(e2, o2);
        v[6] = sub_mi(e2, o2);
        v[3] = add(e3, o3);
        v[7] = sub(e3, o3);
    } else {
        static_assert(R == 16, "radix 2, 4, 8 or 16");
        constexpr float c1 = 0.92387953251128676f, s1 = 0.38268343236508977f;
        constexpr float hl = (float)(0.70710678118654752 - (double)h);
        constexpr float cl = (float)(0.92387953251128676 - (double)c1), sl = (float)(0.38268343236508977 - (double)s1);
        // v[i] * (wr, wi), the constants' remainders beside them
        auto turn = [&](int i, float wr, float wi, float lr, float li) {
            v[i] = FINE ? mul_fine(v[i], wr, wi, lr, li) : mul(v[i], wr, wi);
        };
        // n = 4 a + b, k = c + 4 d: DFT-4 over a, w16^(b c), DFT-4 over b
#pragma unroll
        for (int b = 0; b < 4; b++) dft4(v[b], v[4 + b], v[8 + b], v[12 + b]);
        turn(5, c1, -s1, cl, -sl);
        turn(9, h, -h, hl, -hl);
        turn(13, s1, -c1, sl, -cl);
        turn(6, h, -h, hl, -hl);
        const c2 t = v[10];  // w16^4 = -i
        v[10] = {t.im, make_float2(-t.re.x, -t.re.y)};
        turn(14, -h, -h, -hl, -hl);
        turn(7, s1, -c1, sl, -cl);
        turn(11, -h, -h, -hl, -hl);
        turn(15, -c1, s1, -cl, sl);
#pragma unroll
        for (int c = 0; c < 4; c++) dft4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
        // position 4 c + d holds X[c + 4 d]
#pragma unroll
        for (int c = 0; c < 4; c++)
#pragma unroll
            for (int d = c + 1; d < 4; d++) {
                const c2 x = v[4 * c + d];
                v[4 * c + d] = v[4 * d + c];
                v[4 * d + c] = x;
            }
    }
}

// v[k] *= tw[(k - 1) ld], 0 < k < R: a column of a twiddle table in shared memory, each
// entry rounded once.  (Powers of one rounded root would carry k times its error:
// 1.3e-7 instead of 0.8e-7 relative L2 at 64 points.)
template <int R>
__device__ __forceinline__ void twiddle_column(c2 (&v)[R], const float2* tw, uint32_t ld) {
#pragma unroll
    for (int k = 1; k < R; k++) v[k] = mul(v[k], tw[(k - 1) * ld]);
}

// exp(-2 pi i m / N), m < N <= 2^23 (the quotient is exact for N a power of two)
__device__ __forceinline__ float2 root(uint32_t m, uint32_t N) {
    float s, c;
    sincospif(-2.0f * (float)m / (float)N, &s, &c);
    return make_float2(c, s);
}

__device__ __forceinline__ c2 pair(float4 q) { return {make_float2(q.x, q.z), make_float2(q.y, q.w)}; }

// One dual-polarisation CI8 sample [p0 re, p0 im, p1 re, p1 im], exact
__device__ __forceinline__ c2 pair_ci8(uint32_t w) {
    return pair(ci8_f4(w));
}

// The pair as consecutive complex values; circular != 0: (X + iY, X - iY)
__device__ __forceinline__ float4 unpair(const c2& v, int circular) {
    if (circular)
        return make_float4(v.re.x - v.im.y, v.im.x + v.re.y, v.re.x + v.im.y, v.im.x - v.re.y);
    return make_float4(v.re.x, v.im.x, v.re.y, v.im.y);
}

}  // namespace fft
}  // namespace bb
