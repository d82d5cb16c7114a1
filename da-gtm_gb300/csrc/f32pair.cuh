// f32pair.cuh -- FP32 arguments of the exponentials that equal the FP64 expression's
// rounding, without FP64 (the FP32 form's passes, estep_f32.cu); and the widening of an
// FP32 value by integer operations.
//
// Host/device code, so that it can be compared with the FP64 expressions on the CPU.
#pragma once

#include <math.h>
#include <stdint.h>
#include <string.h>

#if defined(__CUDACC__)
#define F32_HD __host__ __device__ __forceinline__
#else
#define F32_HD static inline
#endif

namespace dgtm {

#if defined(__CUDA_ARCH__)
F32_HD float rn_add(float a, float b) { return __fadd_rn(a, b); }
F32_HD float rn_sub(float a, float b) { return __fsub_rn(a, b); }
F32_HD float rn_mul(float a, float b) { return __fmul_rn(a, b); }
F32_HD float rn_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
F32_HD uint32_t float_bits(float f) { return __float_as_uint(f); }
F32_HD double double_of(uint32_t hi, uint32_t lo) { return __hiloint2double((int) hi, (int) lo); }
#else
// compiled without contraction
F32_HD float rn_add(float a, float b) { return a + b; }
F32_HD float rn_sub(float a, float b) { return a - b; }
F32_HD float rn_mul(float a, float b) { return a * b; }
F32_HD float rn_fma(float a, float b, float c) { return fmaf(a, b, c); }
F32_HD uint32_t float_bits(float f)
{
    uint32_t b;
    memcpy(&b, &f, sizeof b);
    return b;
}
F32_HD double double_of(uint32_t hi, uint32_t lo)
{
    const uint64_t b = ((uint64_t) hi << 32) | lo;
    double v;
    memcpy(&v, &b, sizeof v);
    return v;
}
#endif

// a double as an unevaluated sum of two FP32 (48 bits)
struct Pair {
    float h, l;
};

F32_HD Pair split(double v)
{
    Pair r;
    r.h = (float) v;
    r.l = (float) (v - (double) r.h);
    return r;
}

// s + e = a + b exactly
F32_HD void two_sum(float a, float b, float &s, float &e)
{
    s = rn_add(a, b);
    const float t = rn_sub(s, a);
    e = rn_add(rn_sub(a, rn_sub(s, t)), rn_sub(b, t));
}

// h + l rounded to FP32; ok is cleared when it is not safely away from a rounding
// boundary (or not finite).  The remainder e may be off by 2^-42 |r|, at most 2^-17 of
// the distance to the nearest boundary from r, so r is safe if e grown by 2^-16 still
// rounds to it.
F32_HD float settle(float h, float l, bool &ok)
{
    const float r = rn_add(h, l);
    const float e = rn_sub(l, rn_sub(r, h));
    ok = ok && rn_add(r, rn_mul(e, 1.f + 0x1p-16f)) == r;
    return r;
}

// Whether c x is exactly h + l with h = c.h xh: then its rounding is that of the
// FP64 product too, even half way between two FP32 numbers (a beta / 2 of a few
// bits, such as 3, puts a quarter of the products there)
F32_HD bool exact_product(Pair c, float xh, float xl)
{
    const float h = rn_mul(c.h, xh), l = rn_fma(c.h, xh, -h), p = rn_mul(c.h, xl);
    float s, e;
    two_sum(l, p, s, e);
    return c.l == 0.f && rn_fma(c.h, xl, -p) == 0.f && e == 0.f;
}

// c x as a pair, x = xh + xl
F32_HD void times(Pair c, float xh, float xl, float &h, float &l)
{
    h = rn_mul(c.h, xh);
    l = rn_fma(c.h, xh, -h);
    l = rn_fma(c.h, xl, l);
    l = rn_fma(c.l, xh, l);
}

// (float) (-c x), x = xh + xl; not to be used where ok comes back false and c x is not an
// exact_product
F32_HD float pass1_argument(Pair c, float xh, float xl, bool &ok)
{
    float h, l;
    times(c, xh, xl, h, l);
    return -settle(h, l, ok);
}

// (float) (-c (d - dref) - ln s) with ln s = sh + sl, d >= dref and s >= 1 (its best centre
// adds 1), so that nothing cancels; not to be used where ok comes back false
F32_HD float pass2_argument(Pair c, float d, float dref, float sh, float sl, bool &ok)
{
    float xh, xl, h, l, t, u;
    two_sum(d, -dref, xh, xl);
    times(c, xh, xl, h, l);
    two_sum(h, sh, t, u);
    u = rn_add(u, rn_add(l, sl));
    return -settle(t, u, ok);
}

// An FP32 value as FP64 by integer operations (a conversion takes the FP64 pipe's 16
// clocks of the SM per warp); a subnormal is first scaled by 2^24, exactly, and
// non-finite values are converted.
F32_HD double widen(float f)
{
    const bool small = fabsf(f) < 1.17549435e-38f;
    const uint32_t b = float_bits(small ? rn_mul(f, 16777216.f) : f), m = b & 0x7FFFFFFFu;
    if (m >= 0x7F800000u) {
#if defined(__CUDA_ARCH__)
        asm volatile("");  // keeps the conversion behind the branch
#endif
        return (double) f;
    }
    const uint32_t hi = (m >> 3) + (small ? 0x38000000u - (24u << 20) : 0x38000000u);
    return double_of((b & 0x80000000u) | (m ? hi : 0u), b << 29);
}

}  // namespace dgtm
