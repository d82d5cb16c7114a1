// Host check of csrc/ozfix.cuh: digits, the fixed-point product and exp2_neg
// against long-double references.  Prints the largest errors.
#include "../da-gtm_gb300/csrc/ozfix.cuh"
#include <random>
#include <stdio.h>
#include <vector>
using namespace dgtm::oz;

int main()
{
    std::mt19937_64 g(7);
    std::uniform_real_distribution<double> u(-1.0, 1.0);
    // digits rebuild the integer, and the integer is the value to half a unit
    double bad = 0;
    for (int it = 0; it < 200000; it++) {
        const double v = u(g) * pow(2.0, -40.0 * (it % 3 == 0) * fabs(u(g)));
        const int e = (it & 1) ? 0 : 3;
        const int64_t q = to_fixed(v, e);
        const long double err = fabsl((long double) q - ldexpl((long double) v, FIX - e));
        if (err > 0.5L || llabs(q) > (1ll << 55))
            bad += 1;
        int64_t r = q, back = 0;
        int d[DIGITS];
        for (int i = 0; i < DIGITS; i++)
            d[i] = (int) digit_field((uint64_t) r + digit_bias(), i) - 64;
        for (int i = 0; i < DIGITS; i++) {
            if (d[i] < -64 || d[i] > 64)
                bad += 1;
            back = back * 128 + d[i];
        }
        if (back != q)
            bad += 1;
    }
    // the extremes of the range
    const double ext[] = {1.0 - 0x1p-53, -(1.0 - 0x1p-53), 0.0, 0x1p-1074, 0x1p-60};
    for (double v : ext) {
        int64_t r = to_fixed(v, 0), q = r, back = 0;
        int d[DIGITS];
        for (int i = 0; i < DIGITS; i++)
            d[i] = (int) digit_field((uint64_t) r + digit_bias(), i) - 64;
        for (int i = 0; i < DIGITS; i++) {
            back = back * 128 + d[i];
            if (d[i] < -64 || d[i] > 64)
                bad += 1;
        }
        if (back != q)
            bad += 1;
    }
    std::vector<uint64_t> tab(TAB);
    fill_table(tab.data());
    // exp2_neg and its double, relative to 2^-W of the same W
    long double worst = 0, worstd = 0;
    for (int it = 0; it < 2000000; it++) {
        uint64_t W = g() >> (it % 12);
        if (it < 8192)
            W = ((uint64_t) it << 41) + (it & 1 ? (1ull << 41) - 1 : 0);
        const int n = (int) (W >> WFRAC);
        const uint64_t E = exp2_neg(W, tab.data());
        const long double f = (long double) (W & ((1ull << 53) - 1)) * 0x1p-53L;
        const long double ref = exp2l(-f);
        worst = fmaxl(worst, fabsl((long double) E * 0x1p-63L / ref - 1.0L));
        if (n <= 1000)
            worstd = fmaxl(worstd, fabsl((long double) to_double(E, n) / (ref * exp2l(-n)) - 1.0L));
    }
    // products
    long double worstm = 0;
    const double ks[] = {1.5, 0x1.234p3, 3e-4, 0x1.fp-8, 900.0};
    for (double k : ks)
        for (int e = -60; e <= 0; e += 3) {
            const Mul m = mul_at(make_mul(k), e);
            for (int it = 0; it < 20000; it++) {
                uint64_t x = (uint64_t) (fabs(u(g)) * (double) m.lim);
                if (x > m.lim)
                    x = m.lim;
                const long double ref = (long double) x * (long double) k * ldexpl(1.0L, e + 53);
                const long double err = fabsl((long double) mul_w(m, x) - ref);
                if (ref > 2001.0L * 0x1p53L)
                    bad += 1;
                worstm = fmaxl(worstm, err);
            }
        }
    printf("%.0f %.3Le %.3Le %.3Le\n", bad, worst, worstd, worstm);
    return 0;
}
