// Host check of csrc/ozfix.cuh: the exponents w = x kappa over the whole range of
// FP64's powers (0 to 1074 bits), for mantissas of kappa over a binade and units
// around those a context uses.  Prints how many powers were dropped, how many came
// out beyond 2010 bits instead of being dropped, and the largest error of w in units.
#include "../da-gtm_gb300/csrc/ozfix.cuh"
#include <random>
#include <stdio.h>
using namespace dgtm::oz;

static uint64_t whole(const Mul &k, uint64_t x) { return x <= k.lim ? mul_w(k, x) : mul_far(k, x); }

int main()
{
    std::mt19937_64 g(11);
    long dropped = 0, beyond = 0;
    long double worst = 0;
    for (int i = 0; i < 256; i++)
        for (int u = -70; u <= 12; u++) {
            const double k0 = 1.0 + i / 256.0;
            const Mul k = mul_at(make_mul(k0), u);
            const long double unit = (long double) k0 * ldexpl(1.0L, u);  // one x, in bits
            for (int it = 0; it < 40; it++) {
                const long double bits = it == 0 ? 1074.0L : it < 20 ? 1074.0L * (g() % 10000) / 10000 : 4000.0L * (g() % 10000) / 10000;
                const long double xl = floorl(bits / unit);
                if (xl >= 9223372036854775808.0L)
                    continue;  // not a difference of two 63-bit integers
                const uint64_t x = (uint64_t) xl, w = whole(k, x);
                const long double ref = xl * unit;
                if (ref <= 1075.0L && w == ~0ull)
                    dropped++;
                if (ref >= 2010.0L && w != ~0ull)
                    beyond++;
                if (w != ~0ull)
                    worst = fmaxl(worst, fabsl((long double) w - ref * 0x1p53L));
            }
        }
    printf("%ld %ld %.3Le\n", dropped, beyond, worst);
    return 0;
}
