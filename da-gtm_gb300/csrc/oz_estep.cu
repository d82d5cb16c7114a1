// oz_estep.cu -- the E-step, the responsibility pass and the MAP projection in
// FP64 accuracy from digit-slice distances (oz.cu): real-valued data of the FP64
// form, and the map of every form.
//
// The CUDA-core kernels (estep_simt.cu) spend D FP64 multiply-adds and about 20
// FP64 operations of exp a centre-point pair, on a pipe of two per clock and SM.
// Here the contraction runs on the tensor cores and what is left per pair on the
// integer pipe:
//
//   distances.  v_kn = y_k.t_n - |y_k|^2 / 2 = (|t_n|^2 - d_kn) / 2 as a 64-bit integer in
//     units 2^u of the point's own (ozfix.cuh), so the best centre is an integer
//     comparison and d_kn - d_min = 2 (v_max - v_kn) 2^u an exact integer difference.
//     Every point and every centre is cut into digits on the power-of-two grid of its
//     own largest coordinate: the error of d_kn follows |t_n| and |y_k|, as that of an
//     FP64 sum does, whatever other points and centres hold.
//   exponentials.  2^-W for the fixed-point W = c log2(e) (d_kn - d_min) (+ log2 of
//     the column sum), units of 2^-53 (ozfix.cuh): no FP64 operation.
//   column sums.  2^-63 integers with a carry word: exact, order-free.
//   G and R T.  R_kn on its centre's power-of-two grid (the chunk's largest
//     R of the centre within [2^-56, 1] of it: small responsibilities keep their
//     relative precision), in eight digit planes, times the digit planes of
//     T^T and a row of ones: exact sums over the splits of a chunk, FP64 across them.  The
//     points are what is summed over, so T^T has a grid per column; data with a column
//     whose largest value is far above its others (plain_columns) stay on the CUDA cores
//     altogether: their pass with these distances' d_ref would put R of the large point
//     off by its |t|^2.
//
// Points go in chunks whose K x nn integers stay in L2 (1e7 of them, 80 MB of 129).
// Everything per chunk is a launch of its own: the distances cross L2 once more
// than in a fused kernel (16 bytes a pair, against ~150 integer operations), and
// one layout serves the statistics, the responsibilities and the map.
#include "common.cuh"
#include "kernels.cuh"
#include "oz.cuh"
#include "oz_slice.cuh"

#include <math.h>
#include <new>
#include <type_traits>

namespace dgtm {

namespace {

constexpr int PANEL = 64;
constexpr long long CHUNK = 10000000;   // centre-point pairs a chunk
constexpr int ST_PTS = 8;               // points of a statistics or map block
constexpr int DG_K = 2;                 // centres of a digits block
constexpr int NARROW = 8;               // depths whose products are formed as 64-bit integers
constexpr int NARROW_K = 16;            // centres of a block of them
constexpr int64_t ZERO_COLUMN = INT64_MIN;  // aref of a point whose R is 1/K
constexpr size_t TAB_BYTES = sizeof(uint64_t) * oz::TAB;

__host__ __device__ constexpr int rup(int a, int b) { return (a + b - 1) / b * b; }

// what the centres' kernel leaves for the units; two of them take turns, the idle one
// reset by oz_units_kernel
struct OzScale {
    int ymin;  // least exponent of a centre's |y|^2
    int bad;   // a centre is not finite
};
constexpr int YMIN_START = 1 << 20;

// a point's reference and the exponent its responsibilities start from
struct OzPoint {
    int64_t aref;   // v of its d_ref, or ZERO_COLUMN
    uint64_t lam;   // log2 s + WBIAS (2^-53)
};

// planes[i][r][d] = digit i of X[r][d] on the grid of row r's largest value; zero past rows
// and D.  fixed (instead of planes): [r][d] = X[r][d] as an integer below 2^61, ld of a row.
// ex: the rows' exponents (may be null).  cen: the rows as centres, with xx = |x|^2, and
// their sc (both may be null).  start: the two sc before their first use (may be null).  A
// warp a row, ld <= 256.
__global__ void __launch_bounds__(256) oz_slice_rows_kernel(const double *__restrict__ X, int rows, int D,
                                                            int prows, int ld,
                                                            __nv_bfloat16 *__restrict__ planes,
                                                            int64_t *__restrict__ fixed, int *__restrict__ ex,
                                                            const double *__restrict__ xx,
                                                            oz::Centre *__restrict__ cen, OzScale *sc,
                                                            OzScale *start)
{
    if (start && blockIdx.x == 0 && threadIdx.x < 2)
        start[threadIdx.x] = OzScale{YMIN_START, 0};
    const int lane = threadIdx.x & 31;
    const size_t n2 = (size_t) prows * ld / 2;
    int ymin = YMIN_START, bad = 0;
    for (int r = blockIdx.x * 8 + (threadIdx.x >> 5); r < prows; r += gridDim.x * 8) {
        double x[8];  // depths 2 lane + 64 i, + 1
        unsigned long long m = 0ull;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int d = 2 * lane + 64 * (i >> 1) + (i & 1);
            x[i] = r < rows && d < D ? X[(size_t) r * D + d] : 0.0;
            const unsigned long long b = oz::double_bits(x[i]) & oz::ABS_MASK;
            m = b > m ? b : m;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long b = __shfl_xor_sync(0xffffffffu, m, o);
            m = b > m ? b : m;
        }
        const int e = oz::exponent_of(m);
        if (r < rows && lane == 0) {
            if (ex)
                ex[r] = e;
            if (cen) {
                cen[r] = oz::make_centre(m, xx[r]);
                ymin = min(ymin, oz::exponent_of(oz::double_bits(xx[r]) & oz::ABS_MASK));
                bad |= m >= oz::INF_BITS;
            }
        }
        if (fixed) {
            if (r < rows)
#pragma unroll
                for (int i = 0; i < 2; i++)
                    if (2 * lane + i < ld)
                        fixed[(size_t) r * ld + 2 * lane + i] = oz::scaled_int(x[i], 61 - e);
            continue;
        }
#pragma unroll
        for (int i = 0; i < 8; i += 2) {
            const int d = 2 * lane + 32 * i;
            if (d >= ld)
                break;
            uint32_t w[oz::DIGITS];
            digit_pairs(oz::to_fixed(x[i], e), oz::to_fixed(x[i + 1], e), w);
            uint32_t *dst = (uint32_t *) planes + ((size_t) r * ld + d) / 2;
#pragma unroll
            for (int p = 0; p < oz::DIGITS; p++)
                dst[(size_t) p * n2] = w[p];
        }
    }
    if (sc && lane == 0) {
        atomicMin(&sc->ymin, ymin);
        if (bad)
            atomicOr(&sc->bad, 1);
    }
}

// The points' units for the centres that left sc; idle: the next call's sc.  The product is
// in units of 2^(e + f - bits), or 2^(f - bits) where the data are exact (0/1).
__global__ void __launch_bounds__(256) oz_units_kernel(const int *__restrict__ ex, const double *__restrict__ tt, int N,
                                                       const OzScale *__restrict__ sc, OzScale *__restrict__ idle,
                                                       int bits, bool exact, int ucap, OzUnit *__restrict__ units)
{
    const int ymin = sc->ymin;
    for (int n = blockIdx.x * 256 + threadIdx.x; n < N; n += gridDim.x * 256) {
        units[n] = OzUnit{exact ? -bits : ex[n] - bits,
                          oz::point_unit(oz::exponent_of(oz::double_bits(tt[n])), ymin, ucap)};
    }
    if (blockIdx.x == 0 && threadIdx.x == 0)
        *idle = OzScale{YMIN_START, 0};
}

// The products of up to 8 depths as 64-bit integers: each product's upper 64 bits (in
// 2^-58 of the operands' 2^e, eight of them below 2^61) added exactly, then oz::level.  Eight
// digits of either operand leave 2^-54 of the largest product, which at few depths is more
// than an FP64 sum loses: on one grid for all points the error of R at D = 5 was 1.9e-15 of
// its norm, 1.2e-15 by FP64 products, and is 5.6e-16 this way (D >= 9: the digits were the more
// exact, 2.2e-15 against 2.6e-15 at D = 9, 4.1e-15 against 1.4e-14 at D = 37).  A thread
// holds a point, DP >= D depths of it, and goes through 16 centres; bound by integer issue,
// about 10 instructions a product, on small problems by the latency of that loop (N = 992,
// K = 289, D = 4: 29 us with 64 centres).
template <int DP>
__global__ void __launch_bounds__(256) oz_narrow_kernel(const int64_t *__restrict__ T, const int64_t *__restrict__ Y,
                                                        int nn, int K, const OzUnit *__restrict__ units,
                                                        const oz::Centre *__restrict__ cen, size_t ldm,
                                                        int64_t *__restrict__ out)
{
    __shared__ longlong2 cols[NARROW_K];  // |y|^2 / 2 on one exponent (as in oz_gemm_kernel) and f
    __shared__ int s_top;
    const int kb = blockIdx.x * NARROW_K;
    if (threadIdx.x < 32) {
        const oz::Centre c = cen[min(kb + (int) threadIdx.x % NARROW_K, K - 1)];
        const int top = __reduce_max_sync(0xffffffffu, c.yx);
        if (threadIdx.x < NARROW_K)
            cols[threadIdx.x] = make_longlong2(oz::half_square(c, top), c.f);
        if (threadIdx.x == 0)
            s_top = top;
    }
    __syncthreads();
    const int top = s_top;
    const int m = blockIdx.y * 256 + threadIdx.x;
    if (m >= nn)
        return;
    const OzUnit un = units[m];
    const bool near = oz::near_group(top, un.u);
    const int rh = un.u - top + 10;
    int64_t t[DP];
#pragma unroll
    for (int d = 0; d < DP; d++)
        t[d] = T[(size_t) m * DP + d];
    const int k1 = min(K, kb + NARROW_K);
#pragma unroll 4
    for (int k = kb; k < k1; k++) {
        int64_t sum = 0;
#pragma unroll
        for (int d = 0; d < DP; d++)
            sum += __mul64hi(t[d], Y[(size_t) k * DP + d]);
        const longlong2 y = cols[k - kb];
        out[(size_t) k * ldm + m] = near ? oz::shifted(sum, un.p + (int) y.y - un.u) - oz::sar(y.x, rh)
                                         : oz::level(sum, cen[k], un.p, un.u);
    }
}

__device__ __forceinline__ void load_table(uint64_t *tab, const uint64_t *__restrict__ gtab)
{
    for (int i = threadIdx.x; i < oz::TAB; i += blockDim.x)
        tab[i] = gtab[i];
}

// the base-2 exponent of a double's natural logarithm term, as a fixed-point value
__device__ __forceinline__ uint64_t lam_of(double ln_s)
{
    return oz::to_wfix(ln_s * 1.4426950408889634 + (double) oz::WBIAS);
}

struct OzStatsArgs {
    const int64_t *acc;    // K x ldm
    size_t ldm;
    const OzScale *sc;
    const OzUnit *units;   // this chunk's points
    const uint64_t *tab;
    const double *tt;      // this chunk's points
    int nn, K, isDA;
    double c1, c2, dcut;
    oz::MulBase k1, k2;    // 2 c log2(e) for the two exponents
    double2 *colstat;
    OzPoint *pt;
    int64_t *thr;
    double *part;          // 2 per block of the call
    double *block_part;    // of this launch
    double *sums;          // totals, from the last block of the call
    int nblocks;           // of the call
    unsigned *done;        // blocks finished (zero between calls)
};

// (hi, lo) += 2^-(x kappa) in units of 2^-63
__device__ __forceinline__ void add_power(uint64_t x, const oz::Mul &k, const uint64_t *tab, uint64_t &lo,
                                          uint32_t &hi)
{
    const uint64_t W = oz::mul_w(k, x <= k.lim ? x : k.lim);  // lim is 992 bits down at least (or 0)
    const int n = (int) (W >> oz::WFRAC);
    if (n < 64 && x <= k.lim) {
        const uint64_t t = oz::exp2_neg(W, tab) >> n;
        lo += t;
        hi += lo < t;
    }
}

// Column statistics of a chunk.  Block: 8 points x 64 or 128 centre groups (a
// warp reads four 64-byte rows at once); the maximum first, then the sums against it.
// Bound by the integer pipe: about 75 instructions an exponential.
template <int NT, bool TWO>
__global__ void __launch_bounds__(NT) oz_stats_kernel(const OzStatsArgs a)
{
    constexpr int ST_WARPS = NT / 32, ST_KG = NT / ST_PTS;  // warps, centre groups
    extern __shared__ uint64_t tab[];
    __shared__ int64_t smax[ST_WARPS][ST_PTS];
    __shared__ uint64_t slo[2][ST_WARPS][ST_PTS];
    __shared__ uint32_t shi[2][ST_WARPS][ST_PTS];
    __shared__ double red[32];
    __shared__ int last;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int pl = lane & (ST_PTS - 1), kg = w * (32 / ST_PTS) + lane / ST_PTS;
    const int p = blockIdx.x * ST_PTS + pl;
    const bool live = p < a.nn;
    const int64_t *acc = a.acc + (live ? p : 0);
    const int u = a.units[live ? p : 0].u;
    load_table(tab, a.tab);
    int64_t m = INT64_MIN;
    for (int k0 = kg; k0 < a.K; k0 += 8 * ST_KG) {
        int64_t v[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const int k = min(k0 + j * ST_KG, a.K - 1);  // a repeated centre changes no maximum
            v[j] = acc[(size_t) k * a.ldm];
        }
#pragma unroll
        for (int j = 0; j < 8; j++)
            m = v[j] > m ? v[j] : m;
    }
#pragma unroll
    for (int o = ST_PTS; o < 32; o <<= 1) {
        const int64_t v = __shfl_xor_sync(0xffffffffu, m, o);
        m = v > m ? v : m;
    }
    if (lane < ST_PTS)
        smax[w][lane] = m;
    __syncthreads();
    m = smax[0][pl];
#pragma unroll
    for (int i = 1; i < ST_WARPS; i++)
        m = smax[i][pl] > m ? smax[i][pl] : m;
    const oz::Mul k1 = oz::mul_at(a.k1, u), k2 = oz::mul_at(a.k2, u);
    uint64_t lo1 = 0, lo2 = 0;
    uint32_t hi1 = 0, hi2 = 0;
    for (int k0 = kg; k0 < a.K; k0 += 4 * ST_KG) {
        uint64_t x[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int k = min(k0 + j * ST_KG, a.K - 1);
            x[j] = (uint64_t) (m - acc[(size_t) k * a.ldm]);
            if (k0 + j * ST_KG >= a.K)
                x[j] = ~0ull;
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
            add_power(x[j], k1, tab, lo1, hi1);
            if (TWO)
                add_power(x[j], k2, tab, lo2, hi2);
        }
    }
#pragma unroll
    for (int o = ST_PTS; o < 32; o <<= 1) {
        uint64_t v = __shfl_xor_sync(0xffffffffu, lo1, o);
        hi1 += __shfl_xor_sync(0xffffffffu, hi1, o);
        lo1 += v;
        hi1 += lo1 < v;
        if (TWO) {
            v = __shfl_xor_sync(0xffffffffu, lo2, o);
            hi2 += __shfl_xor_sync(0xffffffffu, hi2, o);
            lo2 += v;
            hi2 += lo2 < v;
        }
    }
    if (lane < ST_PTS) {
        slo[0][w][lane] = lo1;
        shi[0][w][lane] = hi1;
        slo[1][w][lane] = lo2;
        shi[1][w][lane] = hi2;
    }
    __syncthreads();
    double t1 = 0.0, t2 = 0.0;
    if (w == 0 && lane < ST_PTS && live) {
#pragma unroll
        for (int i = 1; i < ST_WARPS; i++) {
            const uint64_t v1 = slo[0][i][lane], v2 = slo[1][i][lane];
            lo1 += v1;
            hi1 += shi[0][i][lane] + (lo1 < v1);
            lo2 += v2;
            hi2 += shi[1][i][lane] + (lo2 < v2);
        }
        const double s1 = (double) hi1 * 2.0 + (double) lo1 * 0x1p-63;
        const double s2 = TWO ? (double) hi2 * 2.0 + (double) lo2 * 0x1p-63 : s1;
        const double dmin = a.tt[p] - 2.0 * scalbn((double) m, u);
        const double ln1 = log(s1), ln2 = TWO ? log(s2) : ln1;
        t1 = -a.c1 * dmin + ln1;
        t2 = a.isDA ? -a.c2 * dmin + ln2 : 0.0;
        double lsn = a.isDA ? ln2 : ln1;
        int64_t aref = m;
        uint64_t lam = lam_of(lsn);
        // comm/mpicomm.c:382-389: a column whose every exp(-beta d/2) underflows
        // is replaced by R = 1/K with v = K
        if (exp(-a.c1 * dmin) == 0.0 || a.sc->bad) {
            lsn = NAN;
            aref = ZERO_COLUMN;
            lam = lam_of(log((double) a.K));
            if (a.isDA) {
                t1 = -INFINITY;
                t2 = log((double) a.K);
            } else {
                t1 = log((double) a.K);
            }
            if (a.sc->bad)
                t1 = t2 = NAN;
        }
        a.colstat[p] = make_double2(dmin, lsn);
        a.pt[p] = OzPoint{aref, lam};
        // R = 0 beyond the distance where the reference's exp(-beta d / 2) underflows
        a.thr[p] = aref == ZERO_COLUMN ? INT64_MIN : oz::scaled_int(a.tt[p] - a.dcut, -1 - u);
    }
    if (w == 0) {
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) {
            t1 += __shfl_down_sync(0xffffffffu, t1, o);
            t2 += __shfl_down_sync(0xffffffffu, t2, o);
        }
        if (lane == 0) {
            a.block_part[2 * blockIdx.x] = t1;
            a.block_part[2 * blockIdx.x + 1] = t2;
            __threadfence();
            last = atomicAdd(a.done, 1u) == (unsigned) a.nblocks - 1;
        }
    }
    __syncthreads();
    if (!last)
        return;
    // the call's last block: all terms, in a fixed order
    __threadfence();
    double u1 = 0.0, u2 = 0.0;
    for (int i = threadIdx.x; i < a.nblocks; i += NT) {
        u1 += __ldcg(a.part + 2 * (size_t) i);
        u2 += __ldcg(a.part + 2 * (size_t) i + 1);
    }
    u1 = block_sum_fixed(u1, red);
    u2 = block_sum_fixed(u2, red);
    if (threadIdx.x == 0) {
        a.sums[0] = u1;
        a.sums[1] = u2;
        *a.done = 0u;
    }
}

// references and exponents from a context's column statistics (d_ref, ln s)
__global__ void oz_points_kernel(const double2 *__restrict__ colstat, const double *__restrict__ tt, int N,
                                 int K, const OzScale *__restrict__ sc, const OzUnit *__restrict__ units,
                                 double dcut, OzPoint *__restrict__ pt, int64_t *__restrict__ thr)
{
    for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < N; n += gridDim.x * blockDim.x) {
        const double2 cs = colstat[n];
        const int u = units[n].u;
        OzPoint o;
        if (isnan(cs.y) || sc->bad) {
            o.aref = ZERO_COLUMN;
            o.lam = lam_of(log((double) K));
        } else {
            o.aref = oz::scaled_int(tt[n] - cs.x, -1 - u);
            o.lam = lam_of(cs.y);
        }
        pt[n] = o;
        thr[n] = o.aref == ZERO_COLUMN ? INT64_MIN : oz::scaled_int(tt[n] - dcut, -1 - u);
    }
}

// W of R = 2^(WBIAS - W): w(aref - v) + lam; ~0 where R is 0
__device__ __forceinline__ uint64_t r_exponent(const OzPoint &o, int64_t v, const oz::Mul &k)
{
    if (o.aref == ZERO_COLUMN)
        return o.lam;
    const int64_t x = o.aref - v;
    const uint64_t ax = (uint64_t) (x < 0 ? -x : x);
    if (ax > k.lim) {
        const uint64_t far = x < 0 ? ~0ull : oz::mul_far(k, ax);
        return x < 0 ? 0ull : far == ~0ull ? far : o.lam + far;
    }
    const uint64_t wv = oz::mul_w(k, ax);
    if (x >= 0)
        return o.lam + wv;
    return o.lam > wv ? o.lam - wv : 0ull;
}

// the exponent of R^2
__device__ __forceinline__ uint64_t r_square(uint64_t W)
{
    constexpr uint64_t bias = (uint64_t) oz::WBIAS << oz::WFRAC;
    return W >> 63 ? ~0ull : 2 * W > bias ? 2 * W - bias : 0ull;
}

// W of a centre's values from W of its R: the grid bound and the digits agree on it
template <bool SQ>
__device__ __forceinline__ int grid_of_w(float w)
{
    if (SQ)
        w = 2.f * w - (float) oz::WBIAS;
    // the integer part of a W at most 2^-5 + 2^-9 w below w
    w = floorf(w - 0.03125f - w * 0.001953125f);
    return w < 0.f ? 0 : (int) w;
}

// The least exponents W of R_kn of DG_K centres over the points na .. nb (each
// warp's own share), in FP32: enough for the grid of a centre's responsibilities
// (grid_of_w takes a margin), and one conversion and one FMA a pair.
__device__ __forceinline__ void least_exponents(const int64_t *const (&row)[DG_K], int na, int nb,
                                                const oz::MulBase &kb, const OzUnit *__restrict__ units,
                                                const OzPoint *__restrict__ pt, const int64_t *__restrict__ thr,
                                                float (&w)[DG_K])
{
    const float kf0 = (float) (kb.m >> 40) * 0x1p-24f;
#pragma unroll
    for (int i = 0; i < DG_K; i++)
        w[i] = 4096.f;
    for (int n = na + threadIdx.x; n < nb; n += 256) {
        const OzPoint o = pt[n];
        const int64_t t = thr[n];
        // exponents from x >> xs, xs such that one of its units is at most 2^-8
        const int q = kb.ex + units[n].u, xs = min(max(-8 - q, 0), 40);
        const float kf = kf0 * __int_as_float((min(q + xs, 64) + 127) << 23);
        const float lf = (float) (uint32_t) (o.lam >> 32) * 0x1p-21f;  // 53 - 32 bits of fraction
#pragma unroll
        for (int i = 0; i < DG_K; i++) {
            const int64_t v = row[i][n];
            const int64_t x = (o.aref - v) >> xs;
            const int xi = x > 0x7FFFFFFF ? 0x7FFFFFFF : (int) x;  // x >= -(a few): d_ref is the least
            const float f = o.aref == ZERO_COLUMN ? lf : fmaf((float) xi, kf, lf);
            w[i] = fminf(w[i], v < t ? 4096.f : f);
        }
    }
#pragma unroll
    for (int i = 0; i < DG_K; i++) {
#pragma unroll
        for (int s = 16; s > 0; s >>= 1)
            w[i] = fminf(w[i], __shfl_xor_sync(0xffffffffu, w[i], s));
        w[i] = fmaxf(w[i], 0.f);
    }
}

// wmin[k] = that of the whole chunk as FP32 bits (4096 where all R are 0).  Block:
// DG_K centres (a point's constants are read once for all of them), a range of points.
__global__ void __launch_bounds__(256) oz_rmax_kernel(const int64_t *__restrict__ acc, size_t ldm, int nn, int K,
                                                      const OzUnit *__restrict__ units,
                                                      const OzPoint *__restrict__ pt,
                                                      const int64_t *__restrict__ thr, oz::MulBase kb, int range,
                                                      unsigned *__restrict__ wmin)
{
    const int k0 = blockIdx.x * DG_K, na = blockIdx.y * range, nb = min(nn, na + range);
    const int64_t *row[DG_K];
    float w[DG_K];
#pragma unroll
    for (int i = 0; i < DG_K; i++)
        row[i] = acc + (size_t) min(k0 + i, K - 1) * ldm;
    least_exponents(row, na, nb, kb, units, pt, thr, w);
#pragma unroll
    for (int i = 0; i < DG_K; i++)
        if ((threadIdx.x & 31) == 0 && k0 + i < K)
            atomicMin(&wmin[k0 + i], __float_as_uint(w[i]));
}

// Responsibilities (SQ: their squares) of a chunk as digit planes, planes[i][k][n]
// (n fastest), each centre on the grid of its largest value in the chunk; nmin[k] is
// an integer bound of that value's exponent.  Zero past nn up to ldn.  Blocks as in
// oz_rmax_kernel, two points a thread.  FIND: the block covers the whole chunk and
// finds the grids itself (a second launch reads the distances from L2 again: 100 us
// a chunk of 1e7 pairs against 87).  Bound by the integer pipe: about 120
// instructions a pair, half of them the exponential.
template <bool SQ, bool FIND>
__global__ void __launch_bounds__(256) oz_digits_kernel(const int64_t *__restrict__ acc, size_t ldm, int nn, int K,
                                                        const OzUnit *__restrict__ units,
                                                        const uint64_t *__restrict__ gtab,
                                                        const OzPoint *__restrict__ pt,
                                                        const int64_t *__restrict__ thr, oz::MulBase kb, int range,
                                                        unsigned *__restrict__ wmin, int prows, int ldn,
                                                        __nv_bfloat16 *__restrict__ planes,
                                                        int *__restrict__ nmin_out)
{
    extern __shared__ uint64_t tab[];
    const int k0 = blockIdx.x * DG_K, ja = blockIdx.y * (range / 2), jb = min(ldn / 2, ja + range / 2);
    const int64_t *row[DG_K];
    int nmin[DG_K];
    load_table(tab, gtab);
#pragma unroll
    for (int i = 0; i < DG_K; i++)
        row[i] = acc + (size_t) min(k0 + i, K - 1) * ldm;
    if constexpr (FIND) {
        __shared__ float red[8][DG_K];
        float w[DG_K];
        least_exponents(row, 0, nn, kb, units, pt, thr, w);
        if ((threadIdx.x & 31) == 0) {
#pragma unroll
            for (int i = 0; i < DG_K; i++)
                red[threadIdx.x >> 5][i] = w[i];
        }
        __syncthreads();
        if (threadIdx.x < DG_K && k0 + (int) threadIdx.x < K) {
            float m = red[0][threadIdx.x];
            for (int i = 1; i < 8; i++)
                m = fminf(m, red[i][threadIdx.x]);
            wmin[k0 + threadIdx.x] = __float_as_uint(m);
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < DG_K; i++) {
        nmin[i] = grid_of_w<SQ>(__uint_as_float(wmin[min(k0 + i, K - 1)]));
        if (threadIdx.x == 0 && blockIdx.y == 0 && k0 + i < K)
            nmin_out[k0 + i] = nmin[i];
    }
    const size_t plane = (size_t) prows * ldn / 2;
    for (int j = ja + threadIdx.x; j < jb; j += 256) {
        OzPoint o[2];
        int64_t t[2];
        oz::Mul km[2];
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const int n = min(2 * j + e, nn - 1);
            o[e] = pt[n];
            km[e] = oz::mul_at(kb, units[n].u);
            t[e] = 2 * j + e < nn ? thr[n] : INT64_MAX;  // padding: R = 0
        }
#pragma unroll
        for (int i = 0; i < DG_K; i++) {
            if (k0 + i >= K)
                break;
            int64_t q[2];
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int64_t v = row[i][min(2 * j + e, nn - 1)];
                uint64_t W = v < t[e] ? ~0ull : r_exponent(o[e], v, km[e]);
                if (SQ)
                    W = r_square(W);
                const int ex = (int) (W >> oz::WFRAC);
                // R 2^(55 - (5 - nmin)) = E >> (9 + ex - nmin), rounded
                const int sh = 9 + ex - nmin[i];
                q[e] = 0;
                if (ex < 2047 && sh < 64)
                    q[e] = (int64_t) ((oz::exp2_neg(W, tab) + (1ull << (sh - 1))) >> sh);
            }
            uint32_t *dst = (uint32_t *) planes + (size_t) (k0 + i) * ldn / 2 + j;
            uint32_t w[oz::DIGITS];
            digit_pairs(q[0], q[1], w);
#pragma unroll
            for (int d = 0; d < oz::DIGITS; d++)
                dst[(size_t) d * plane] = w[d];
        }
    }
}

// G and R T of a chunk from the products' split sums; the first chunk sets, the
// others add.  Column D of the product is the row of ones: G.
__global__ void __launch_bounds__(256) oz_rt_kernel(const double *__restrict__ part, int ntiles, int splits,
                                                    const int *__restrict__ nmin,
                                                    const unsigned long long *__restrict__ cbits, int K, int D,
                                                    int first, double *__restrict__ G, double *__restrict__ RT)
{
    const int t = blockIdx.x, mt = t / ntiles, nt = t - mt * ntiles;
    for (int e = blockIdx.y * 256 + threadIdx.x; e < 128 * 64; e += 256 * gridDim.y) {
        const int k = mt * 128 + (e & 127), d = nt * 64 + (e >> 7);
        if (k >= K || d > D)
            continue;
        double sum = 0.0;
        for (int sp = 0; sp < splits; sp++)
            sum += part[((size_t) t * splits + sp) * (128 * 64) + e];
        const int nm = nmin[k];
        const double v = nm < 2047 ? scalbn(sum, 5 - nm + oz::exponent_of(cbits[d]) - OZ_SUM_BITS) : 0.0;
        double *dst = d < D ? RT + (size_t) k * D + d : G + k;
        *dst = first ? v : *dst + v;
    }
}

// M = R^T X of a chunk, blocks as in oz_stats_kernel.
template <int NT, int LMAX>
__global__ void __launch_bounds__(NT) oz_map_kernel(const int64_t *__restrict__ acc, size_t ldm, int nn,
                                                            const OzUnit *__restrict__ units,
                                                            const uint64_t *__restrict__ gtab,
                                                            const OzPoint *__restrict__ pt, oz::MulBase kb,
                                                            int K, const double *__restrict__ X, int L,
                                                            double *__restrict__ M)
{
    constexpr int ST_WARPS = NT / 32, ST_KG = NT / ST_PTS;
    extern __shared__ uint64_t tab[];
    __shared__ double sm[ST_WARPS][LMAX][ST_PTS];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int pl = lane & (ST_PTS - 1), kg = w * (32 / ST_PTS) + lane / ST_PTS;
    const int p = blockIdx.x * ST_PTS + pl;
    const bool live = p < nn;
    const int64_t *a = acc + (live ? p : 0);
    const OzPoint o = pt[live ? p : 0];
    const oz::Mul km = oz::mul_at(kb, units[live ? p : 0].u);
    load_table(tab, gtab);
    __syncthreads();
    double m[LMAX] = {};
    for (int k0 = kg; k0 < K; k0 += 4 * ST_KG) {
        int64_t v[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int k = min(k0 + j * ST_KG, K - 1);
            v[j] = a[(size_t) k * ldm];
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int k = k0 + j * ST_KG;
            // (no R is cut here but FAR, which stands for any distance beyond the unit's range)
            const uint64_t W = k < K && (v[j] > oz::FAR || o.aref == ZERO_COLUMN) ? r_exponent(o, v[j], km) : ~0ull;
            const int n = (int) (W >> oz::WFRAC) - oz::WBIAS;
            if (n > 1080)  // R is 0 in FP64
                continue;
            const double r = oz::to_double(oz::exp2_neg(W, tab), n);
#pragma unroll
            for (int l = 0; l < LMAX; l++)
                if (l < L)
                    m[l] = fma(r, X[(size_t) k * L + l], m[l]);
        }
    }
#pragma unroll
    for (int l = 0; l < LMAX; l++) {
#pragma unroll
        for (int s = ST_PTS; s < 32; s <<= 1)
            m[l] += __shfl_xor_sync(0xffffffffu, m[l], s);
        if (lane < ST_PTS)
            sm[w][l][lane] = m[l];
    }
    __syncthreads();
    if (threadIdx.x < LMAX * ST_PTS) {
        const int l = threadIdx.x / ST_PTS, q = blockIdx.x * ST_PTS + threadIdx.x % ST_PTS;
        if (l < L && q < nn) {
            double s = 0.0;
            for (int i = 0; i < ST_WARPS; i++)
                s += sm[i][l][threadIdx.x % ST_PTS];
            M[(size_t) q * L + l] = s;
        }
    }
}

// R of a block of centres and points from its distances (acc: nk rows of ldm)
__global__ void __launch_bounds__(256) oz_rblock_kernel(const int64_t *__restrict__ acc, size_t ldm, int nk, int nn,
                                                        const OzUnit *__restrict__ units,
                                                        const uint64_t *__restrict__ gtab,
                                                        const OzPoint *__restrict__ pt,
                                                        const int64_t *__restrict__ thr, oz::MulBase kb, size_t ldR,
                                                        double *__restrict__ R)
{
    extern __shared__ uint64_t tab[];
    load_table(tab, gtab);
    __syncthreads();
    const size_t total = (size_t) nk * nn;
    for (size_t i = blockIdx.x * (size_t) 256 + threadIdx.x; i < total; i += (size_t) gridDim.x * 256) {
        const int k = (int) (i / nn), n = (int) (i - (size_t) k * nn);
        const int64_t v = acc[(size_t) k * ldm + n];
        const uint64_t W = v < thr[n] ? ~0ull : r_exponent(pt[n], v, oz::mul_at(kb, units[n].u));
        R[(size_t) k * ldR + n] =
            W == ~0ull ? 0.0 : oz::to_double(oz::exp2_neg(W, tab), (int) (W >> oz::WFRAC) - oz::WBIAS);
    }
}

int grid_of(size_t n, int cap)
{
    const size_t b = (n + 255) / 256;
    return (int) (b < 1 ? 1 : b > (size_t) cap ? (size_t) cap : b);
}

}  // namespace

struct OzE {
    OzEArgs a;
    unsigned char *arena = nullptr;  // every buffer below, one allocation
    int narrow = 0;  // depths of a row of 64-bit integers in Town and Yp, 0: digit planes
    int sa = 8, panels = 0, ldT = 0, ldY = 0, Np = 0, Kp = 0, chunk = 0, nchunks = 0;  // lds: of a row of planes
    const __nv_bfloat16 *Tp = nullptr;  // data planes (own or the caller's)
    __nv_bfloat16 *Town = nullptr, *Yp = nullptr;
    unsigned long long *bits = nullptr;  // maxima of the columns of T, then of the ones; then, 32 bits
                                         // each, how many of their values are short of bits
    OzScale *sc = nullptr;   // [2], sc_now the one of the centres in Yp
    int sc_now = 0;
    int *ex = nullptr;       // the points' exponents
    OzUnit *units = nullptr; // and units for the centres in Yp
    oz::Centre *cen = nullptr;
    uint64_t *tab = nullptr;
    int64_t *acc = nullptr;
    size_t ldm = 0;
    OzPoint *pt = nullptr;
    int64_t *thr = nullptr;  // acc below it: the reference's R is 0
    int acc_whole = 0;  // acc holds all points of the centres in Yp
    int own_stats = 0;  // Yp, cen, units and pt are those of the last oze_estep
    // responsibility pass
    int Wp = 0, Kp128 = 0, Npk = 0, rt_tiles = 0, rt_per = 0;
    __nv_bfloat16 *Tt = nullptr, *Rp = nullptr;
    double *part = nullptr;
    int *nmin = nullptr;
    unsigned *wmin = nullptr;
    unsigned *done = nullptr;  // statistics blocks finished in a call
};

// The digit-slice path has fixed costs (planes of the centres, four launches a
// chunk, tiles of 128 x 64), about 60 us an EM iteration.  The CUDA-core kernels
// take that for about 3e4 pairs: few blocks, each walking all centres (N = 1000,
// K = 400, D = 12: 600 us).
bool oze_wanted(int N, int D, int K)
{
    return D <= 4 * PANEL && K <= (1 << 20) && (double) N * K >= 32768;
}

void oze_destroy(OzE *st)
{
    if (!st)
        return;
    if (st->arena)
        cudaFree(st->arena);
    delete st;
}

// the table of exp2_neg, filled once in the process (4096 long-double powers)
static const uint64_t *host_table()
{
    struct Table {
        uint64_t v[oz::TAB];
        Table() { oz::fill_table(v); }
    };
    static const Table t;
    return t.v;
}

// Whether every column of T (maxima, then counts of values short of bits) has squares
// within FP64 and keeps its precision on one grid: at most a quarter of its values are
// below 2^-6 of the grid's end and not exact there.  A value at that line
// keeps 50 bits, the column's sums then 2^-51 of its bulk.  Gaussian and uniform
// columns, and 0/1 and other coarse values, pass (a Gaussian column of 1e6 points: 20 %);
// a column with one value 16 standard deviations out does not (38 %).
static bool plain_columns(const unsigned long long *top, int D, int N)
{
    const unsigned *low = (const unsigned *) (top + D + 1);
    for (int d = 0; d < D; d++)
        if (top[d] >= oz::double_bits(0x1p500) || 4.0 * low[d] > (double) N)
            return false;
    return true;
}

int oze_create(OzE **out, const OzEArgs &a, cudaStream_t s)
{
    *out = nullptr;
    OzE *st = new (std::nothrow) OzE();
    if (!st) {
        set_error(DGTM_ENOMEM, "host allocation failed");
        return DGTM_ENOMEM;
    }
    st->a = a;
    const int N = a.N, D = a.D, K = a.K;
    st->sa = a.Tb ? 1 : 8;
    st->narrow = a.Tb || D > NARROW ? 0 : D <= 2 ? 2 : D <= 4 ? 4 : 8;
    // rows of planes in whole panels, at few depths in whole 32 bytes (the product's panel is
    // filled up with zeros on the way: a quarter of the memory at D = 9); or of 64-bit
    // integers.  Rows of 16-byte multiples at D = 37 made a chunk's product 25 us longer.
    st->ldY = st->narrow ? st->narrow : D <= PANEL / 2 ? rup(D, 16) : rup(D, PANEL);
    st->ldT = a.Tb ? a.Tb_ld : st->ldY;
    st->panels = ceil_div(D, PANEL);
    st->Np = a.Tb ? a.Tb_rows : rup(N, 128);
    st->Kp = rup(K, 64);
    // points a chunk: no more than whole waves of statistics blocks (8 points on each SM)
    // where one fits, in whole tiles of 128 (which leave the last wave of an odd number of
    // waves a little short: 1152 points for 1216 on 152 SMs)
    const long long wave = (long long) ST_PTS * a.sms;
    long long c = CHUNK / K;
    c = c >= wave ? c / wave * wave : c;
    c = c / 128 * 128;
    c = c < 128 ? 128 : c > st->Np ? st->Np : c;
    st->chunk = (int) c;
    st->nchunks = ceil_div(N, st->chunk);
    st->ldm = (size_t) st->chunk;
    st->Wp = rup(D + 1, 64);
    st->Kp128 = rup(K, 128);
    st->Npk = rup(N, PANEL);
    const size_t planes = sizeof(__nv_bfloat16) * oz::DIGITS;
    const size_t value = st->narrow ? sizeof(int64_t) : planes;  // bytes of one of T or Y
    const int cp = rup(st->chunk, PANEL) / PANEL;
    st->rt_tiles = (st->Kp128 / 128) * (st->Wp / 64);
    st->rt_per = oz_item_panels(st->rt_tiles, cp, a.sms);
    size_t bytes = 0;
    auto lay = [&](auto **pp, size_t n, unsigned char *base) {
        if (base)
            *pp = reinterpret_cast<std::remove_reference_t<decltype(*pp)>>(base + bytes);
        bytes += (n + 255) / 256 * 256;
    };
    auto lay_out = [&](unsigned char *base) {
        bytes = 0;
        if (!a.Tb)
            lay(&st->Town, value * st->Np * st->ldT, base);
        lay(&st->Yp, value * st->Kp * st->ldY, base);
        lay(&st->bits, (sizeof(unsigned long long) + sizeof(unsigned)) * (D + 1), base);
        lay(&st->sc, 2 * sizeof(OzScale), base);
        lay(&st->ex, sizeof(int) * N, base);
        lay(&st->units, sizeof(OzUnit) * N, base);
        lay(&st->cen, sizeof(oz::Centre) * K, base);
        lay(&st->tab, TAB_BYTES, base);
        lay(&st->acc, sizeof(int64_t) * st->ldm * K, base);
        lay(&st->pt, sizeof(OzPoint) * N, base);
        lay(&st->thr, sizeof(int64_t) * N, base);
        lay(&st->wmin, sizeof(unsigned) * K, base);
        lay(&st->done, sizeof(unsigned), base);
        if (a.mstep) {
            lay(&st->Tt, planes * (D + 1) * st->Npk, base);
            lay(&st->Rp, planes * st->Kp128 * st->chunk, base);
            lay(&st->part, sizeof(double) * 8192 * (size_t) st->rt_tiles * ceil_div(cp, st->rt_per), base);
            lay(&st->nmin, sizeof(int) * K, base);
        }
    };
    lay_out(nullptr);
    cudaError_t e = cudaMalloc((void **) &st->arena, bytes);
    if (e == cudaSuccess)
        lay_out(st->arena);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(st->tab, host_table(), TAB_BYTES, cudaMemcpyHostToDevice, s);
    const size_t nbits = (sizeof(unsigned long long) + sizeof(unsigned)) * (D + 1);
    unsigned *low = (unsigned *) (st->bits + D + 1);
    if (e == cudaSuccess)
        e = cudaMemsetAsync(st->bits, 0, nbits, s);
    if (e == cudaSuccess)
        e = cudaMemsetAsync(st->done, 0, sizeof(unsigned), s);
    if (e == cudaSuccess) {
        // of 0/1 data, which are in Tb, only the exponents are wanted: rows of no columns
        oz_slice_rows_kernel<<<grid_of((size_t) st->Np * 32, 16384), 256, 0, s>>>(
            a.T64, N, D, a.Tb ? N : st->Np, a.Tb ? 0 : st->ldT, st->Town,
            st->narrow ? (int64_t *) st->Town : nullptr, st->ex, nullptr, nullptr, nullptr, st->sc);
        e = cudaGetLastError();
        st->Tp = a.Tb ? a.Tb : st->Town;
    }
    const OzSource src{nullptr, a.T64, nullptr, D, D, 0};
    if (e == cudaSuccess) {
        oz_colmax_kernel<<<dim3(ceil_div(N, 512), ceil_div(D + 1, 32)), 256, 0, s>>>(src, N, D + 1, 512, st->bits);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess && a.mstep) {
        oz_slice_t_kernel<<<dim3(st->Npk / PANEL, ceil_div(D + 1, 32)), 256, 0, s>>>(
            src, N, D + 1, D + 1, st->Npk, st->bits, st->Tt, low, nullptr);
        if (e == cudaSuccess)
            e = cudaGetLastError();
    }
    unsigned long long cols[(4 * PANEL + 1) * 3 / 2 + 1];  // nbits, D <= 256 (oze_wanted)
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(cols, st->bits, nbits, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess)
        e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
        const int code = e == cudaErrorMemoryAllocation ? DGTM_ENOMEM : DGTM_ECUDA;
        cudaGetLastError();
        set_error(code, "oze_create: %s", cudaGetErrorString(e));
        oze_destroy(st);
        return code;
    }
    // the CUDA-core kernels carry data, or squares of it, that are not finite, and sums
    // that the grids would cost bits
    if (!plain_columns(cols, D, N)) {
        oze_destroy(st);
        return DGTM_OK;
    }
    *out = st;
    return DGTM_OK;
}

int oze_estep_blocks(const OzE *st)
{
    return (st->nchunks - 1) * (st->chunk / ST_PTS) +
           ceil_div(st->a.N - (st->nchunks - 1) * st->chunk, ST_PTS);
}

namespace {

// the centres' planes, and the points' units for exponents c1 d and c2 d
int slice_centres(OzE *st, const double *Y, const double *yy, double c1, double c2, cudaStream_t s)
{
    const int N = st->a.N, K = st->a.K, D = st->a.D;
    st->sc_now ^= 1;
    oz_slice_rows_kernel<<<grid_of((size_t) st->Kp * 32, 4864), 256, 0, s>>>(
        Y, K, D, st->Kp, st->ldY, st->Yp, st->narrow ? (int64_t *) st->Yp : nullptr,
        nullptr, yy, st->cen, st->sc + st->sc_now, nullptr);
    DGTM_CUDA_TRY(cudaGetLastError());
    oz_units_kernel<<<grid_of((size_t) N, 1216), 256, 0, s>>>(
        st->ex, st->a.tt, N, st->sc + st->sc_now, st->sc + (st->sc_now ^ 1), st->narrow ? 58 : st->sa == 1 ? 55 : 53,
        st->sa == 1, oz::unit_cap(c1, c2), st->units);
    DGTM_CUDA_TRY(cudaGetLastError());
    st->acc_whole = st->own_stats = 0;
    return DGTM_OK;
}

// points m0 .. m0 + nn - 1 with centres k0 .. k0 + nk - 1 into out (narrow state)
int narrow_products(OzE *st, int m0, int nn, int k0, int nk, size_t ldm, int64_t *out, cudaStream_t s)
{
    const int dp = st->narrow;
    const auto kernel = dp == 2 ? oz_narrow_kernel<2> : dp == 4 ? oz_narrow_kernel<4> : oz_narrow_kernel<8>;
    const dim3 grid(ceil_div(nk, NARROW_K), ceil_div(nn, 256));
    kernel<<<grid, 256, 0, s>>>((const int64_t *) st->Tp + (size_t) m0 * dp, (const int64_t *) st->Yp + (size_t) k0 * dp,
                                nn, nk, st->units + m0, st->cen + k0, ldm, out);
    DGTM_CUDA_TRY(cudaGetLastError());
    return DGTM_OK;
}

// the integer products of chunk c
int chunk_products(OzE *st, int c, cudaStream_t s)
{
    if (st->narrow) {
        const int n0 = c * st->chunk, nn = st->a.N - n0 < st->chunk ? st->a.N - n0 : st->chunk;
        return narrow_products(st, n0, nn, 0, st->a.K, st->ldm, st->acc, s);
    }
    OzGemm g;
    g.A = st->Tp;
    g.B = st->Yp;
    g.sa = st->sa;
    g.a_rows = st->Np;
    g.b_rows = st->Kp;
    g.panels = st->panels;
    g.a_ld = st->ldT;
    g.b_ld = st->ldY;
    const int n0 = c * st->chunk, nn = st->a.N - n0 < st->chunk ? st->a.N - n0 : st->chunk;
    g.a_tile0 = n0 / 128;
    g.mtiles = ceil_div(nn, 128);
    g.ntiles = st->Kp / 64;
    g.out = st->acc;
    g.ldm = st->ldm;
    g.mrows = nn;
    g.ncols = st->a.K;
    g.units = st->units + n0;
    g.cen = st->cen;
    return launch_oz_gemm(g, st->a.sms, st->a.status, s);
}

template <typename Kernel>
int table_smem(Kernel k)
{
    DGTM_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) TAB_BYTES));
    return DGTM_OK;
}

// Few points a chunk (many centres): fewer than two blocks an SM, so that a block
// of 1024 threads keeps the SM's schedulers busier than one of 512
bool wide_blocks(int K) { return K > 4096; }

constexpr double LOG2E_2 = 2.0 * 1.4426950408889634;

}  // namespace

#define OZ_TRY(expr)           \
    do {                       \
        const int _r = (expr); \
        if (_r != DGTM_OK)     \
            return _r;         \
    } while (0)

int oze_estep(OzE *st, const double *Y, const double *yy, double c1, double c2, int isDA, double2 *colstat,
              double *part, double dcut, double *sums, int *nlaunch, cudaStream_t s)
{
    OZ_TRY(slice_centres(st, Y, yy, c1, isDA ? c2 : c1, s));
    const bool two = isDA && c1 != c2;
    const int nt = wide_blocks(st->a.K) ? 1024 : 512;
    const auto kernel = nt == 512 ? (two ? oz_stats_kernel<512, true> : oz_stats_kernel<512, false>)
                                  : (two ? oz_stats_kernel<1024, true> : oz_stats_kernel<1024, false>);
    OZ_TRY(table_smem(kernel));
    for (int c = 0; c < st->nchunks; c++) {
        OZ_TRY(chunk_products(st, c, s));
        const int n0 = c * st->chunk, nn = st->a.N - n0 < st->chunk ? st->a.N - n0 : st->chunk;
        OzStatsArgs a{};
        a.acc = st->acc;
        a.ldm = st->ldm;
        a.sc = st->sc + st->sc_now;
        a.units = st->units + n0;
        a.tab = st->tab;
        a.tt = st->a.tt + n0;
        a.nn = nn;
        a.K = st->a.K;
        a.isDA = isDA;
        a.c1 = c1;
        a.c2 = c2;
        a.k1 = oz::make_mul(c1 * LOG2E_2);
        a.k2 = oz::make_mul(c2 * LOG2E_2);
        a.colstat = colstat + n0;
        a.pt = st->pt + n0;
        a.thr = st->thr + n0;
        a.dcut = dcut;
        a.part = part;
        a.block_part = part + 2 * (size_t) (n0 / ST_PTS);
        a.sums = sums;
        a.nblocks = oze_estep_blocks(st);
        a.done = st->done;
        kernel<<<ceil_div(nn, ST_PTS), nt, TAB_BYTES, s>>>(a);
        DGTM_CUDA_TRY(cudaGetLastError());
    }
    st->acc_whole = st->nchunks == 1;
    st->own_stats = 1;
    if (nlaunch)
        *nlaunch = 2 + 2 * st->nchunks;
    return DGTM_OK;
}

int oze_mstep_pass(OzE *st, double c, double *G, double *RT, int *nlaunch, cudaStream_t s)
{
    const int K = st->a.K, D = st->a.D;
    int nl = 0;
    for (int ch = 0; ch < st->nchunks; ch++) {
        if (!st->acc_whole) {
            OZ_TRY(chunk_products(st, ch, s));
            nl++;
        }
        const int n0 = ch * st->chunk, nn = st->a.N - n0 < st->chunk ? st->a.N - n0 : st->chunk;
        const int ldn = rup(nn, PANEL);
        OZ_TRY(oze_r_digits(st, ch, 0, K, c, false, false, st->Kp128, st->Rp, st->nmin, s));
        OzGemm g;
        g.A = st->Rp;
        g.B = st->Tt;
        g.a_rows = st->Kp128;
        g.b_rows = D + 1;
        g.panels = ldn / PANEL;
        g.a_ld = ldn;
        g.b_ld = st->Npk;
        g.b_panel0 = n0 / PANEL;
        g.mtiles = st->Kp128 / 128;
        g.ntiles = st->Wp / 64;
        g.sums = st->part;
        g.item_panels = st->rt_per;
        OZ_TRY(launch_oz_gemm(g, st->a.sms, st->a.status, s));
        oz_rt_kernel<<<dim3(st->rt_tiles, 32), 256, 0, s>>>(st->part, g.ntiles, ceil_div(g.panels, st->rt_per),
                                                            st->nmin, st->bits, K, D,
                                                            ch == 0 ? 1 : 0, G, RT);
        DGTM_CUDA_TRY(cudaGetLastError());
        nl += 4;
    }
    if (nlaunch)
        *nlaunch = nl;
    return DGTM_OK;
}

// the centres' planes and the points' references for a context's column statistics
int oze_refer(OzE *st, const double *Y, const double *yy, const double2 *colstat, double c1, double c, double dcut,
              cudaStream_t s)
{
    if (st->own_stats)
        return DGTM_OK;
    OZ_TRY(slice_centres(st, Y, yy, c1, c, s));
    oz_points_kernel<<<grid_of((size_t) st->a.N, 1216), 256, 0, s>>>(colstat, st->a.tt, st->a.N, st->a.K,
                                                                    st->sc + st->sc_now, st->units, dcut, st->pt,
                                                                    st->thr);
    DGTM_CUDA_TRY(cudaGetLastError());
    return DGTM_OK;
}

int oze_chunks(const OzE *st, int *points)
{
    *points = st->chunk;
    return st->nchunks;
}

int oze_r_digits(OzE *st, int ch, int k0, int kb, double c, bool squares, bool products, int prows,
                 __nv_bfloat16 *planes, int *nmin, cudaStream_t s)
{
    if (products && !st->acc_whole)
        OZ_TRY(chunk_products(st, ch, s));
    const int n0 = ch * st->chunk, nn = st->a.N - n0 < st->chunk ? st->a.N - n0 : st->chunk;
    const int ldn = rup(nn, PANEL), kblocks = ceil_div(kb, DG_K);
    // ranges of points: about four blocks an SM, at least 1024 points each
    int parts = ceil_div(4LL * st->a.sms, kblocks);
    const int range = rup(ceil_div(ldn, parts) < 1024 ? 1024 : ceil_div(ldn, parts), PANEL);
    parts = ceil_div(ldn, range);
    const int64_t *acc = st->acc + (size_t) k0 * st->ldm;
    const oz::MulBase base = oz::make_mul(c * LOG2E_2);
    // the squares' grids follow from the same exponents
    const auto kernel = squares ? oz_digits_kernel<true, false>
                                : parts == 1 ? oz_digits_kernel<false, true> : oz_digits_kernel<false, false>;
    OZ_TRY(table_smem(kernel));
    if (!squares && parts > 1) {
        DGTM_CUDA_TRY(cudaMemsetAsync(st->wmin, 0x7F, sizeof(unsigned) * kb, s));
        oz_rmax_kernel<<<dim3(kblocks, parts), 256, 0, s>>>(acc, st->ldm, nn, kb, st->units + n0, st->pt + n0,
                                                            st->thr + n0, base, range, st->wmin);
        DGTM_CUDA_TRY(cudaGetLastError());
    }
    kernel<<<dim3(kblocks, parts), 256, TAB_BYTES, s>>>(acc, st->ldm, nn, kb, st->units + n0, st->tab,
                                                        st->pt + n0, st->thr + n0, base, range, st->wmin, prows,
                                                        ldn, planes, nmin);
    DGTM_CUDA_TRY(cudaGetLastError());
    return DGTM_OK;
}

int oze_r_block(OzE *st, const double *Y, const double *yy, const double2 *colstat, double c1, double c, double dcut,
                int k0, int nk, int n0, int nn, double *R, cudaStream_t s)
{
    OZ_TRY(oze_refer(st, Y, yy, colstat, c1, c, dcut, s));
    OZ_TRY(table_smem(oz_rblock_kernel));
    const oz::MulBase base = oz::make_mul(c * LOG2E_2);
    auto launch = [&](const int64_t *acc, size_t ldm, int n, int np) -> int {
        oz_rblock_kernel<<<grid_of((size_t) nk * np, 1216), 256, TAB_BYTES, s>>>(
            acc, ldm, nk, np, st->units + n, st->tab, st->pt + n, st->thr + n, base, (size_t) nn, R + (n - n0));
        DGTM_CUDA_TRY(cudaGetLastError());
        return DGTM_OK;
    };
    if (st->acc_whole)
        return launch(st->acc + (size_t) k0 * st->ldm + n0, st->ldm, n0, nn);
    // as many points at a time as the chunk buffer has room for with nk rows
    OzGemm g;
    g.A = st->Tp;
    g.B = st->Yp;
    g.sa = st->sa;
    g.a_rows = st->Np;
    g.b_rows = st->Kp;
    g.b_row0 = k0;
    g.panels = st->panels;
    g.a_ld = st->ldT;
    g.b_ld = st->ldY;
    g.ntiles = ceil_div(nk, 64);
    g.out = st->acc;
    g.ncols = nk;
    g.cen = st->cen + k0;
    const int first = n0 / 128 * 128;
    const long long room = (long long) st->ldm * st->a.K / nk / 128 * 128;
    for (long long m0 = first; m0 < n0 + nn; m0 += room) {
        const int m1 = (int) (m0 + room < n0 + nn ? m0 + room : n0 + nn);
        g.a_tile0 = (int) (m0 / 128);
        g.units = st->units + m0;
        g.mtiles = ceil_div(m1 - m0, 128);
        g.mrows = (int) (m1 - m0);
        g.ldm = (size_t) g.mrows;
        if (st->narrow)
            OZ_TRY(narrow_products(st, (int) m0, m1 - (int) m0, k0, nk, g.ldm, st->acc, s));
        else
            OZ_TRY(launch_oz_gemm(g, st->a.sms, st->a.status, s));
        const int na = m0 < n0 ? n0 : (int) m0;
        OZ_TRY(launch(st->acc + (na - m0), g.ldm, na, m1 - na));
    }
    return DGTM_OK;
}

int oze_map(OzE *st, const double *Y, const double *yy, const double2 *colstat, double c1, double c, const double *X,
            int L, double *M, cudaStream_t s)
{
    const int N = st->a.N, K = st->a.K;
    OZ_TRY(oze_refer(st, Y, yy, colstat, c1, c, 1e300, s));
    const int nt = wide_blocks(K) ? 1024 : 512;
    const auto kernel = nt == 512 ? (L <= 2 ? oz_map_kernel<512, 2> : L == 3 ? oz_map_kernel<512, 3> : oz_map_kernel<512, 8>)
                                  : (L <= 2 ? oz_map_kernel<1024, 2> : L == 3 ? oz_map_kernel<1024, 3> : oz_map_kernel<1024, 8>);
    OZ_TRY(table_smem(kernel));
    for (int ch = 0; ch < st->nchunks; ch++) {
        if (!st->acc_whole)
            OZ_TRY(chunk_products(st, ch, s));
        const int n0 = ch * st->chunk, nn = N - n0 < st->chunk ? N - n0 : st->chunk;
        kernel<<<ceil_div(nn, ST_PTS), nt, TAB_BYTES, s>>>(st->acc, st->ldm, nn, st->units + n0, st->tab,
                                                                   st->pt + n0, oz::make_mul(c * LOG2E_2), K,
                                                                   X, L, M + (size_t) n0 * L);
        DGTM_CUDA_TRY(cudaGetLastError());
    }
    return DGTM_OK;
}

}  // namespace dgtm
