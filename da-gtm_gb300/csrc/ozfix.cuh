// ozfix.cuh -- fixed-point pieces of the digit-slice products (oz.cu): FP64
// values as 56-bit integers in eight balanced base-128 digits, and powers of
// two of a fixed-point exponent in 64-bit integer arithmetic.
//
// GB300 issues FP64 at 2 operations per clock per SM, 1/64 of its FP32 rate and
// 1/32 of its integer rate.  A library exp(double) is about 20 such operations;
// exp2_neg below is about 50 integer ones, and more exact: its argument is a
// fixed-point number with an absolute error of 2^-53, where an FP64 argument of
// 10 already carries 2^-50.
//
// Everything here is host/device code so that it can be checked on the CPU.
#pragma once

#include <math.h>
#include <stdint.h>
#include <string.h>

#if defined(__CUDACC__)
#define OZ_HD __host__ __device__ __forceinline__
#else
#define OZ_HD static inline
#endif

namespace dgtm {
namespace oz {

constexpr int DIGITS = 8;        // balanced base-128 digits, each |d| <= 64
constexpr int FIX = 55;          // |v| < 2^e is held as rint(v 2^(FIX - e)), |q| <= 2^55
constexpr int TAB_BITS = 12;     // exp2_neg: 2^-(i / 4096), i = 0 .. 4095
constexpr int TAB = 1 << TAB_BITS;
constexpr int WFRAC = 53;        // exponents in units of 2^-53
constexpr int WBIAS = 4;         // exponents carry + 4, so a slightly negative one fits

OZ_HD uint64_t mulhi(uint64_t a, uint64_t b)
{
#if defined(__CUDA_ARCH__)
    return __umul64hi(a, b);
#else
    return (uint64_t) (((unsigned __int128) a * b) >> 64);
#endif
}

// mulhi(a, b) or up to two less (without the low halves' product): three 32-bit
// multiplies instead of four and their carries
OZ_HD uint64_t mulhi_low(uint64_t a, uint64_t b)
{
    const uint32_t ah = (uint32_t) (a >> 32), al = (uint32_t) a, bh = (uint32_t) (b >> 32), bl = (uint32_t) b;
    return (uint64_t) ah * bh + (((uint64_t) ah * bl) >> 32) + (((uint64_t) al * bh) >> 32);
}

OZ_HD uint32_t mulhi32(uint32_t a, uint32_t b) { return (uint32_t) (((uint64_t) a * b) >> 32); }

OZ_HD uint64_t double_bits(double v)
{
#if defined(__CUDA_ARCH__)
    return (uint64_t) __double_as_longlong(v);
#else
    uint64_t b;
    memcpy(&b, &v, sizeof b);
    return b;
#endif
}

OZ_HD double bits_double(uint64_t b)
{
#if defined(__CUDA_ARCH__)
    return __longlong_as_double((long long) b);
#else
    double v;
    memcpy(&v, &b, sizeof v);
    return v;
#endif
}

// the bits of |v| order like |v| (with infinities and NaN on top)
constexpr uint64_t ABS_MASK = 0x7FFFFFFFFFFFFFFFull;
constexpr uint64_t INF_BITS = 0x7FF0000000000000ull;

// e with |v| < 2^e for every |v| up to the one with these bits
OZ_HD int exponent_of(uint64_t absbits)
{
    const int E = (int) (absbits >> 52);
    return (E ? E : 1) - 1022;
}

// rint(v 2^(FIX - e)) (ties away from zero), for |v| < 2^e; integer operations only
OZ_HD int64_t to_fixed(double v, int e)
{
    const uint64_t b = double_bits(v);
    const int E = (int) ((b >> 52) & 0x7FF);
    const uint64_t m = (b & 0xFFFFFFFFFFFFFull) | (E ? (1ull << 52) : 0ull);
    const int sh = (E ? E : 1) - 1020 - e;  // at most 2
    uint64_t q;
    if (sh >= 0)
        q = m << (sh & 3);
    else if (sh > -60)
        q = (m + (1ull << (-sh - 1))) >> (-sh);
    else
        q = 0;
    return (b >> 63) ? -(int64_t) q : (int64_t) q;
}

// Whether v is below 2^(e - BULK) and not a whole number of the grid 2^(e - FIX): then
// to_fixed keeps fewer than 50 bits of it.
constexpr int BULK = 6;

OZ_HD bool short_of_bits(double v, int e)
{
    const uint64_t b = double_bits(v);
    const int E = (int) ((b >> 52) & 0x7FF), drop = e + 1020 - (E ? E : 1);
    const uint64_t m = (b & 0xFFFFFFFFFFFFFull) | (E ? (1ull << 52) : 0ull);
    return drop >= BULK - 2 && (m & ((1ull << (drop < 63 ? drop : 63)) - 1)) != 0;
}

// q 2^k as an int64 from a double q, rounded to nearest, saturated
OZ_HD int64_t scaled_int(double v, int k)
{
    const uint64_t b = double_bits(v);
    const int E = (int) ((b >> 52) & 0x7FF);
    const uint64_t m = (b & 0xFFFFFFFFFFFFFull) | (E ? (1ull << 52) : 0ull);
    const int sh = (E ? E : 1) - 1075 + k;
    uint64_t q;
    if (sh >= 10)
        q = m ? 0x7FFFFFFFFFFFFFFFull : 0ull;
    else if (sh >= 0)
        q = m << sh;
    else if (sh > -63)
        q = (m + (1ull << (-sh - 1))) >> (-sh);
    else
        q = 0;
    return (b >> 63) ? -(int64_t) q : (int64_t) q;
}

// digit i (0 the top one) of q: with 64 added to every digit the digits are the
// 7-bit fields of an unsigned number (the top one 8 bits), so none waits for another
OZ_HD uint64_t digit_bias()
{
    // 64 (1 + 2^7 + ... + 2^49)
    return (64ull << 0) + (64ull << 7) + (64ull << 14) + (64ull << 21) + (64ull << 28) + (64ull << 35) +
           (64ull << 42) + (64ull << 49);
}

OZ_HD uint32_t digit_field(uint64_t biased, int i)
{
    return (uint32_t) (biased >> (7 * (DIGITS - 1 - i))) & (i == 0 ? 255u : 127u);
}

// x 2^s for s of 0 and more, zeros from 64 on; and x 2^-s towards minus infinity
OZ_HD uint64_t shl(uint64_t x, int s)
{
#if defined(__CUDA_ARCH__)
    uint64_t r;
    asm("shl.b64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(s));
    return r;
#else
    return s < 64 ? x << s : 0ull;
#endif
}

OZ_HD int64_t sar(int64_t x, int s)
{
#if defined(__CUDA_ARCH__)
    int64_t r;
    asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(s));
    return r;
#else
    return x >> (s < 63 ? s : 63);
#endif
}

OZ_HD uint64_t shr(uint64_t x, int s)
{
#if defined(__CUDA_ARCH__)
    uint64_t r;
    asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(s));
    return r;
#else
    return s < 64 ? x >> s : 0ull;
#endif
}

// w = x kappa in units of 2^-53, for 0 <= x <= lim: (mulhi(x << a, m)) >> b.  lim leaves
// out the last 32nd of what x << a has room for, so that w is below 1984 there; beyond it
// w is 992 or more.
struct Mul {
    uint64_t m;
    uint64_t lim;
    int a, b;
};

constexpr uint64_t W_END = 2000ull << WFRAC;  // a power from here on is 0

// kappa = k0 2^u with k0 known on the host and u (the unit of x) on the device
struct MulBase {
    uint64_t m;  // k0 = m 2^(ex - 64), m's top bit set
    int ex;
};

static inline MulBase make_mul(double k0)
{
    MulBase r;
    int ex = 0;
    const double f = frexp(k0, &ex);  // k0 = f 2^ex, f in [0.5, 1)
    r.m = (uint64_t) ldexp(f, 64);
    r.ex = r.m ? ex : -4096;  // beta / 2 = 0: every exponent 0
    return r;
}

OZ_HD Mul mul_at(const MulBase &k, int u)
{
    Mul r;
    // x kappa 2^53 = x m 2^(ex + u + 53 - 64) = mulhi(x << a, m) >> b
    const int sh = k.ex + u + WFRAC;  // a - b
    r.m = k.m;
    r.a = sh > 0 ? sh : 0;  // from 64 on only x = 0 is within lim
    r.b = sh < 0 ? -sh : 0;
    const uint64_t cap = shr(~0ull, r.a);
    r.lim = cap - (cap >> 5);
    return r;
}

OZ_HD uint64_t mul_w(const Mul &k, uint64_t x) { return shr(mulhi(shl(x, k.a), k.m), k.b); }

// w of x > lim: ~0 from 2000 on.  What x << a has no room for below that has one bit
// too many (m >= 2^63), so it is 2 mulhi(x << (a - 1), m): every power that FP64 can
// hold, 2^-1074 the last, is kept whatever kappa's mantissa.
OZ_HD uint64_t mul_far(const Mul &k, uint64_t x)
{
    if (k.a < 1 || k.a > 64 || x > ~0ull >> (k.a - 1))
        return ~0ull;
    const uint64_t h = mulhi(x << (k.a - 1), k.m);
    return h < W_END / 2 ? 2 * h : ~0ull;
}

// 2^-(W 2^-53) = E 2^-63 2^-n with n = W >> 53: returns E in (2^62, 2^63].
// 2^-f = T[f's top 12 bits] (1 - x), x = y - y^2/2 + y^3/6 - y^4/24 for
// y = rho ln 2 below 2^-12.5; x within 2^-57, T within 2^-63.
OZ_HD uint64_t exp2_neg(uint64_t W, const uint64_t *tab)
{
    const uint32_t i = (uint32_t) (W >> (WFRAC - TAB_BITS)) & (TAB - 1);
    const uint64_t T = tab[i];
    const uint64_t rho = W << (64 - (WFRAC - TAB_BITS));      // the low 41 bits on top
    const uint64_t y = mulhi_low(rho, 0xB17217F7D1CF79ACull) >> TAB_BITS;  // ln 2; y in 2^-64
    const uint32_t yh = (uint32_t) ((y + (1ull << 19)) >> 20);         // y in 2^-44
    const uint64_t yy = (uint64_t) yh * yh;                            // y^2 in 2^-88
    const uint32_t s = (uint32_t) (yy >> 32);                          // y^2 in 2^-56
    const uint32_t s6 = mulhi32(s, 715827883u);                        // y^2 / 6
    const uint64_t y3 = ((uint64_t) s6 * yh) >> 36;                    // y^3 / 6 in 2^-64
    const uint32_t y4 = mulhi32(mulhi32(s, s), 178956971u) >> 16;      // y^4 / 24 in 2^-64
    const uint64_t x = y - (yy >> 25) + y3 - y4;
    return T - mulhi_low(T, x);
}

// E 2^-63 2^(-n) as a double, E in (2^62, 2^63]
OZ_HD double to_double(uint64_t E, int n)
{
    // round to 53 bits: E + half an ulp, carried into the exponent by the add
    const bool one = (E >> 63) != 0;
    const uint64_t m = one ? 0ull : ((E << 2) + (1ull << 11)) >> 12;  // 52 fraction bits (may carry)
    const int e = (one ? 0 : -1) - n;
    if (e < -1021)
        return e < -1100 ? 0.0 : scalbn((double) (int64_t) (E >> 1), -62 - n);
    return bits_double(((uint64_t) (e + 1023) << 52) + m);
}

// Units of the distances.  v = t.y - |y|^2 / 2 = (|t|^2 - d) / 2 of a point and a centre
// is a 64-bit integer in units 2^u of the point's own, because only one point's distances
// are compared with each other; a value elsewhere in the data or on a far centre changes
// nothing for it.  With |t|^2 < 2^x, and 2^ymin next above the least |y|^2 of the centres,
//     u = max(max(x, ymin) - 59, ucap):
// |t|^2 and the smallest centre's |y|^2 are at most 2^59 units, so v of the best
// centre is above -2^60.  A centre with |y|^2 / 2 >= 2^62 has |y| >= 2^31.5 against
// |t| <= 2^29.5, so v <= -|y|^2 / 4 <= -2^61: it gets FAR instead.  Any other has
// |t.y| <= 2^61: nothing overflows.  ucap (unit_cap) bounds the unit from below by what
// the exponentials can tell apart, so that FAR is beyond every distance with an R.
constexpr int64_t FAR = -(1ll << 61);

OZ_HD int point_unit(int x, int ymin, int ucap)
{
    const int u = (x > ymin ? x : ymin) - 59;
    return u > ucap ? u : ucap;
}

// ucap for exponents c1 d and c2 d: 2^60 units are past the reference's cut c1 d = 746 and
// past c2 (d - d_min) = 64, whose R adds nothing to a sum in FP64.  c1 u is then at most
// 2^-50.3, or c2 u at most 2^-54.
static inline int unit_cap(double c1, double c2)
{
    int ex = 0;
    const double range = c1 / 400.0 < c2 / 32.0 ? 400.0 / c1 : 32.0 / c2;
    frexp(range < 0x1p1000 ? range : 0x1p1000, &ex);  // < 2^ex (a c below 1e-298 tells nothing apart)
    return ex - 60;
}

// x 2^s, towards minus infinity, for a result within 63 bits
OZ_HD int64_t shifted(int64_t x, int s)
{
    return sar((int64_t) shl((uint64_t) x, s > 0 ? s : 0), s < 0 ? -s : 0);
}

// a centre of a product: |y|^2 = yy 2^yx, yy in [2^52, 2^53) or 0; |y_d| < 2^f
struct alignas(16) Centre {
    int64_t yy;
    int f, yx;
};

OZ_HD Centre make_centre(uint64_t ymax_bits, double yy)
{
    const uint64_t b = double_bits(yy) & ABS_MASK;
    uint64_t m = b & 0xFFFFFFFFFFFFFull;
    int E = (int) (b >> 52);
    Centre c;
    c.f = exponent_of(ymax_bits);
    if (E) {
        m |= 1ull << 52;  // an infinity (the square of a finite y) becomes 2^1024
    } else if (m) {
        for (E = 1; !(m >> 52); E--)
            m <<= 1;
    }
    c.yy = (int64_t) m;
    c.yx = m ? E - 1075 : -8192;
    return c;
}

// |y|^2 / 2 of a group of centres, the largest yx of which is top, as integers of one
// exponent: |y|^2 / 2 = half_square 2^(top - 10), below 2^62, towards minus infinity.  For
// a point with u >= top - 10 none of them is FAR, and |y|^2 / 2 in its units is
// half_square >> (u - top + 10): the same integer as by level().
OZ_HD int64_t half_square(const Centre &c, int top) { return shifted(c.yy, c.yx - top + 9); }

OZ_HD bool near_group(int top, int u) { return u >= top - 10; }

// v from the product I, in units of 2^(p + f) (2^p the point's: its |t_d| < 2^e, and the digits')
OZ_HD int64_t level(int64_t I, const Centre &c, int p, int u)
{
    const int s = c.yx - 1 - u;
    return s >= 10 ? FAR : shifted(I, p + c.f - u) - shifted(c.yy, s);
}

// A signed 96-bit sum, as three words.
struct Sum96 {
    uint32_t w0, w1, w2;
};

// s += hi 2^28 + lo
OZ_HD void add96(Sum96 &s, int64_t hi, int64_t lo)
{
    const uint32_t a0 = (uint32_t) ((uint64_t) hi << 28), a1 = (uint32_t) (hi >> 4), a2 = (uint32_t) (hi >> 36);
    const uint32_t b0 = (uint32_t) lo, b1 = (uint32_t) ((uint64_t) lo >> 32), b2 = (uint32_t) (lo >> 63);
#if defined(__CUDA_ARCH__)
    asm("add.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, %4;\n\taddc.u32 %2, %2, %5;"
        : "+r"(s.w0), "+r"(s.w1), "+r"(s.w2) : "r"(a0), "r"(a1), "r"(a2));
    asm("add.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, %4;\n\taddc.u32 %2, %2, %5;"
        : "+r"(s.w0), "+r"(s.w1), "+r"(s.w2) : "r"(b0), "r"(b1), "r"(b2));
#else
    uint64_t c = (uint64_t) s.w0 + a0 + b0;
    s.w0 = (uint32_t) c;
    c = (uint64_t) s.w1 + a1 + b1 + (c >> 32);
    s.w1 = (uint32_t) c;
    s.w2 += a2 + b2 + (uint32_t) (c >> 32);
#endif
}

OZ_HD int clz64(uint64_t x)
{
#if defined(__CUDA_ARCH__)
    return __clzll((long long) x);
#else
    return x ? __builtin_clzll(x) : 64;
#endif
}

// the sum as a double, rounded once; integer operations only
OZ_HD double to_double96(const Sum96 &s)
{
    const bool neg = (s.w2 >> 31) != 0;
    uint64_t lo = ((uint64_t) s.w1 << 32) | s.w0, top = s.w2;  // |s| = top 2^64 + lo
    if (neg) {
        lo = ~lo + 1;
        top = (uint32_t) ~s.w2 + (lo == 0 ? 1u : 0u);
    }
    const uint64_t up = (top << 32) | (lo >> 32);              // the upper 64 of 96 bits
    // T 2^e, T's top bit set; what T does not hold is below 2^-63 of it
    const int n = up >> 31 ? clz64(up) : 64;
    const uint64_t T = n < 64 ? (n < 32 ? (up << n) | (n ? (uint32_t) lo >> (32 - n) : 0u) : lo << (n - 32)) : shl(lo, clz64(lo));
    if (T == 0)
        return 0.0;
    const int e = n < 64 ? 95 - n : 63 - clz64(lo);
    const uint64_t m = ((T << 1) >> 12) + ((T >> 10) & 1);      // 52 fraction bits (may carry)
    return bits_double(((uint64_t) neg << 63) | ((((uint64_t) (e + 1023)) << 52) + m));
}

// an unsigned fixed-point value in units of 2^-53 from a double (v >= 0)
OZ_HD uint64_t to_wfix(double v) { return (uint64_t) scaled_int(v, WFRAC); }

// table entry: 2^-(i / 4096) in units of 2^-63
static inline void fill_table(uint64_t *tab)
{
    for (int i = 0; i < TAB; i++)
        tab[i] = (uint64_t) (exp2l(-(long double) i / TAB) * 9223372036854775808.0L + 0.5L);
}

}  // namespace oz
}  // namespace dgtm
