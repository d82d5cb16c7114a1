// Host check of csrc/ozfix.cuh: 96-bit sums of hi 2^28 + lo against 128-bit integers, and
// their doubles, over sums of every size and sign.  Prints wrong sums and the largest error
// of a double relative to half a unit in its last place.
#include "../da-gtm_gb300/csrc/ozfix.cuh"
#include <random>
#include <stdio.h>
using namespace dgtm::oz;

int main()
{
    std::mt19937_64 g(2);
    long wrong = 0;
    long double worst = 0;
    for (int it = 0; it < 400000; it++) {
        Sum96 s{0, 0, 0};
        __int128 ref = 0;
        const int n = 1 + (int) (g() % 40), bits = (int) (g() % 44), cancel = (int) (g() % 3);
        int64_t ph = 0, pl = 0;
        for (int i = 0; i < n; i++) {
            int64_t hi = (int64_t) (g() >> (63 - bits)) - (int64_t) (g() >> (63 - bits));
            int64_t lo = (int64_t) (g() >> 20) - (int64_t) (g() >> 20);
            if (it % 5 == 0)
                hi = 0;
            if (it % 7 == 0)
                lo >>= g() % 44;
            if (cancel == 1 && (i & 1)) {  // sums that nearly vanish
                hi = -ph;
                lo = -pl + (int64_t) (g() % 3) - 1;
            }
            ph = hi;
            pl = lo;
            add96(s, hi, lo);
            ref += (__int128) hi * (1 << 28) + lo;
        }
        const __int128 got = ((__int128) (int32_t) s.w2 << 64) | (((unsigned __int128) s.w1 << 32) | s.w0);
        if (got != ref)
            wrong++;
        const double d = to_double96(s);
        const __int128 diff = (__int128) d - ref;  // d is a whole number
        if (ref == 0) {
            if (d != 0.0)
                wrong++;
            continue;
        }
        int e;
        frexp((double) ref, &e);
        const long double half = ldexpl(1.0L, e - 54);
        const long double err = fabsl((long double) diff) / (half < 0.5L ? 0.5L : half);
        worst = fmaxl(worst, err);
        if ((ref < 0) != (d < 0.0))
            wrong++;
    }
    printf("%ld %.6Lf\n", wrong, worst);
    return 0;
}
