// Host check of csrc/ozfix.cuh: v = t.y - |y|^2 / 2 in the point's units (oz::level) for
// points and centres whose sizes span many powers of two, zeros, and squares outside
// FP64 among them.  Prints
//   1. the largest error of v relative to what is allowed,
//      2^-51 (|t| |y| + |t|^2 + |y|^2), plus the exponents' own 2^-50 / c1 + 2^-54 / c2;
//   2. how many centres got FAR although exp(-c1 d) > 0 or c2 (d - d_min) < 64;
//   3. how many others left 63 bits, or came out otherwise by way of half_square.
#include "../da-gtm_gb300/csrc/ozfix.cuh"
#include <random>
#include <stdio.h>
#include <vector>
using namespace dgtm::oz;

int main()
{
    std::mt19937_64 g(3);
    std::normal_distribution<double> nrm;
    auto uni = [&](double a, double b) { return a + (b - a) * (double) (g() >> 11) * 0x1p-53; };
    long far = 0, over = 0, nearby = 0;
    long double worst = 0;
    const int dims[] = {1, 2, 8, 9, 37, 64, 200, 256};
    for (int it = 0; it < 4000; it++) {
        const int D = dims[it % 8], K = 12;
        const int spread = (it / 8) % 4;  // of the sizes, in powers of two
        const double range = spread == 0 ? 1.0 : spread == 1 ? 10.0 : spread == 2 ? 100.0 : 200.0;
        std::vector<double> t(D);
        const double ts = it % 50 == 7 ? 0.0 : exp2(uni(-range, range));
        for (auto &x : t)
            x = ts * nrm(g);
        if (it % 5 == 0)
            t[g() % D] *= exp2(uni(0.0, range));
        std::vector<std::vector<double>> y(K, std::vector<double>(D));
        for (int k = 0; k < K; k++) {
            const double ys = k % 5 == 4 && it % 3 == 0 ? 0.0 : k < 3 ? ts * exp2(uni(-1.0, 1.0)) : exp2(uni(-range, range));
            for (int d = 0; d < D; d++)
                y[k][d] = k == 0 ? t[d] * (1.0 + 0x1p-20 * nrm(g)) : ys * nrm(g);
            if (k == 11 && it % 7 == 0)
                y[k][0] = 0x1p600;  // its square is no FP64 number
        }
        long double tt = 0;
        uint64_t tb = 0;
        for (double x : t) {
            tt += (long double) x * x;
            const uint64_t b = double_bits(x) & ABS_MASK;
            tb = b > tb ? b : tb;
        }
        const int e = exponent_of(tb);
        std::vector<Centre> c(K);
        std::vector<long double> dist(K), yyl(K), ty(K);
        int least = 1 << 20;
        long double dmin = INFINITY;
        for (int k = 0; k < K; k++) {
            long double yy = 0, p = 0, dd = 0;
            uint64_t yb = 0;
            for (int d = 0; d < D; d++) {
                yy += (long double) y[k][d] * y[k][d];
                p += (long double) t[d] * y[k][d];
                const long double z = (long double) t[d] - y[k][d];
                dd += z * z;
                const uint64_t b = double_bits(y[k][d]) & ABS_MASK;
                yb = b > yb ? b : yb;
            }
            c[k] = make_centre(yb, (double) yy);
            const int x = exponent_of(double_bits((double) yy) & ABS_MASK);
            least = x < least ? x : least;
            dist[k] = dd;
            yyl[k] = yy;
            ty[k] = p;
            dmin = dd < dmin ? dd : dmin;
        }
        // c1 such that the point's distances matter, or are all alike, or all far
        const double c1 = fmin(1e280, fmax(1e-280, (double) (exp2l(uni(-20.0, 20.0)) / (tt + yyl[1] + 1e-250L))));
        const double c2 = c1 / (it % 4 == 0 ? 1.0 : exp2(uni(0.0, 8.0)));
        const int u = point_unit(exponent_of(double_bits((double) tt)), least, unit_cap(c1, c2));
        for (int k = 0; k < K; k++) {
            const int p = e - 53;
            const long double il = roundl(ldexpl(ty[k], -(p + c[k].f)));
            if (fabsl(il) > 0x1p62L)
                over++;
            const int64_t v = level((int64_t) il, c[k], p, u);
            int top = c[k].yx;  // of the centre and its neighbours
            for (int j = 0; j < K; j++)
                if (j / 3 == k / 3 && c[j].yx > top)
                    top = c[j].yx;
            if (near_group(top, u) &&
                v != shifted((int64_t) il, p + c[k].f - u) - sar(half_square(c[k], top), u - top + 10))
                over++;
            nearby += near_group(top, u);
            if (v == FAR) {
                if (c1 * dist[k] < 745.0L || c2 * (dist[k] - dmin) < 64.0L)
                    far++;
                continue;
            }
            if (v < -(3ll << 61) || v > (1ll << 61))
                over++;
            const long double ref = ty[k] - yyl[k] / 2;
            // half a unit of the product, 2^(e + f - 54) <= 4 max|t| max|y| 2^-54, and less than
            // one of the point's
            const long double allowed = 0x1p-51L * (sqrtl(tt) * sqrtl(yyl[k]) + tt + yyl[k]) + 0x1p-50L / c1 + 0x1p-54L / c2;
            worst = fmaxl(worst, fabsl(ldexpl((long double) v, u) - ref) / allowed);
        }
    }
    if (nearby < 10000)
        over++;
    printf("%.3Lf %ld %ld\n", worst, far, over);
    return 0;
}
