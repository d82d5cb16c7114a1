// Host check of csrc/f32pair.cuh: the FP32 arguments of the exponentials against the FP64
// expressions they stand for, bit for bit, on random distances and on ones built so that
// the exact argument lies on, just below or just above a rounding boundary; and widen()
// against the conversion over every exponent.  Prints wrong pass-1 arguments, wrong pass-2
// arguments, wrong widenings, and the share of arguments that take the FP64 expression.
#include "../da-gtm_gb300/csrc/f32pair.cuh"
#include <random>
#include <stdio.h>
using namespace dgtm;

static uint32_t bits(float f) { return float_bits(f); }

static float of_bits(uint32_t b)
{
    float f;
    memcpy(&f, &b, sizeof f);
    return f;
}

int main()
{
    std::mt19937_64 g(5);
    auto uni = [&]() { return (double) (g() >> 11) * 0x1p-53; };
    long bad1 = 0, bad2 = 0, badw = 0, slow = 0, total = 0;
    // few and many bits, ties (3, 0.75), subnormal and huge products
    const double cs[] = {3.0, 0.7, 1.0, 0.75, 5.0 / 3.0, 6.25, 30.0, 0.1, 123456.789, 0x1.000001p0, 0x1.fffffep5, 1e-20, 1e20};
    for (double c : cs) {
        const Pair p = split(c);
        for (int it = 0; it < 3000000; it++) {
            float dm, d;
            switch (it % 5) {
            case 0:  // anywhere
                dm = (float) (100.0 * uni());
                d = dm + (float) (200.0 * uni());
                break;
            case 1:  // close distances: many low bits in x
                dm = (float) (50.0 + uni());
                d = of_bits(bits(dm) + (uint32_t) (g() % 4096));
                break;
            case 2: {  // c x near half way between two FP32 numbers
                const float r = of_bits(bits((float) (90.0 * uni() + 1.0)));
                const double mid = 0.5 * ((double) r + (double) of_bits(bits(r) + 1));
                dm = (float) (uni() * 1e-3);
                d = (float) (mid / c + (double) dm);
                d = of_bits(bits(d) + (uint32_t) (g() % 5) - 2);
                break;
            }
            case 3:  // whole numbers and quarters (0/1 data)
                dm = (float) (g() % 64) * 0.25f;
                d = dm + (float) (g() % 4096) * 0.25f;
                break;
            default:  // over many exponents
                dm = (float) exp2(40.0 * uni() - 20.0);
                d = dm * (float) (1.0 + exp2(30.0 * uni() - 24.0));
            }
            if (!(d >= dm) || !(d < 3e38f))
                continue;
            float xh, xl;
            two_sum(d, -dm, xh, xl);
            bool ok = true;
            float a = pass1_argument(p, xh, xl, ok);
            total++;
            slow += !ok;
            const float ref = (float) (-c * ((double) d - (double) dm));
            if (!ok && !exact_product(p, xh, xl))
                a = ref;
            if (bits(a) != bits(ref))
                bad1++;
            // ln s as pass 1 leaves it, at least 0 (the best centre adds 1 to s); and one that
            // puts the argument near a boundary
            double ls = (it & 1) ? 12.0 * uni() : log(1.0 + 1000.0 * uni());
            if (it % 7 == 0) {
                const double arg = fma(-c, (double) d - (double) dm, -ls);
                const float r = (float) arg;
                ls -= (0.5 * ((double) r + (double) of_bits(bits(r) + 1)) - arg);
                ls += (double) ((int) (g() % 3) - 1) * 0x1p-49 * fabs(arg);
                ls = ls < 0.0 ? 0.0 : ls;
            }
            const Pair l = split(ls);
            ok = true;
            a = pass2_argument(p, d, dm, l.h, l.l, ok);
            total++;
            slow += !ok;
            const float ref2 = (float) fma(-c, (double) d - (double) dm, -ls);
            if (!ok)
                a = ref2;
            if (bits(a) != bits(ref2))
                bad2++;
        }
    }
    for (uint32_t e = 0; e < 512; e++)
        for (int it = 0; it < 3000; it++) {
            const uint32_t man = it == 0 ? 0u : it == 1 ? 0x7FFFFFu : it == 2 ? 1u : (uint32_t) g() & 0x7FFFFFu;
            const float f = of_bits((e << 23) | man);
            const double w = widen(f), r = (double) f;
            if (memcmp(&w, &r, 8) != 0 && !(w != w && r != r))
                badw++;
        }
    printf("%ld %ld %ld %.3e\n", bad1, bad2, badw, (double) slow / (double) total);
    return 0;
}
