// exp(-x) of the parity kernels' samples, correctly rounded without double precision for nearly all of them.
#pragma once

#include "rg_common.cuh"

namespace rg {

constexpr int kPairs = kBuf / 2;        // a slab's samples in pairs (2p and 2p + 1)

// exp of the eight exponents, correctly rounded (out of line: rare)
__device__ __noinline__ float exp_exact(float x) { return (float)exp((double)x); }

// exp(-sig dt) of a slab's samples, correctly rounded (parity arithmetic: one ulp of the exponential is
// ~1e-5 of the opacity, enough to move T > 0.003).  For x = sig dt <= 1/4 the sum 1 - x + x^2 / 2 -
// x^3 / 6 + ... (the Taylor series to x^8) is carried as t + tail with |tail| under half an ulp of t
// or so: 1 - x and its rounding error, x^2 / 2 and the error of the square are exact, and the rest is
// x^3 P(x), whose rounding stays under d = 5e-8 x^3 + 2^-43.  Rounding t + tail gives the correctly
// rounded value unless the remainder comes within d of half an ulp, 2^-25 (results are in [1/2, 1)):
// then, and above 1/4, double precision decides.  Checked against it for every float in [2e-4, 1/4]:
// the largest error is 0.73 d, one argument in a thousand is handed on.  14 packed FP32 issue slots
// per sample instead of a double-precision exp().
__device__ __forceinline__ void exp_neg_slab(const f2* sig, f2* ex, f2 nz) {
    float worst = 0.f, top = 0.f;
#pragma unroll
    for (int p = 0; p < kPairs; ++p) {
        const f2 x = mul2_rn(sig[p], dup2(kDt), nz), m1 = dup2(-1.f), one = dup2(1.f);
        const f2 s = fma2(x, m1, one), nx = mul2_rn(x, m1, nz);
        const f2 sl = add2(fma2(s, m1, one), nx);
        const f2 x2 = mul2_rn(x, x, nz), x2l = fma2(x, x, mul2_rn(x2, m1, nz)), h = mul2_rn(x2, dup2(0.5f), nz);
        f2 P = fma2(x, dup2(1.f / 40320.f), dup2(-1.f / 5040.f));
        P = fma2(x, P, dup2(1.f / 720.f));
        P = fma2(x, P, dup2(-1.f / 120.f));
        P = fma2(x, P, dup2(1.f / 24.f));
        P = fma2(x, P, dup2(-1.f / 6.f));
        const f2 x3 = mul2_rn(x2, x, nz), t = add2(s, h);
        const f2 e = add2(fma2(t, m1, s), h);
        const f2 tail = fma2(x3, P, add2(fma2(x2l, dup2(0.5f), sl), e));
        const f2 r = add2(t, tail);
        const f2 rest = add2(tail, fma2(r, m1, t));   // tail - (r - t)
        const f2 d = fma2(x3, dup2(5e-8f), dup2(0x1p-43f));
        worst = max3f(worst, fabsf(lo2(rest)) + lo2(d), fabsf(hi2(rest)) + hi2(d));
        top = max3f(top, lo2(x), hi2(x));
        ex[p] = r;
    }
    if (worst > 0x1p-25f || top > 0.25f) {
#pragma unroll
        for (int p = 0; p < kPairs; ++p)
            ex[p] = pk(exp_exact(-__fmul_rn(lo2(sig[p]), kDt)), exp_exact(-__fmul_rn(hi2(sig[p]), kDt)));
    }
}

}  // namespace rg
