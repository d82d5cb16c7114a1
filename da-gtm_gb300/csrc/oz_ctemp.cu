// oz_ctemp.cu -- the scatter of the AUTO schedule's critical temperature in FP64
// accuracy on the tensor cores (the FP64 form).
//
// For every centre k the schedule needs S1 = sum_n R_kn x x^T and S2 = sum_n
// R_kn^2 x x^T with x = t_n - y_k (ctemp.cu): K N D^2 FP64 multiply-adds for the
// CUDA-core scatter, on a pipe of two a clock and SM (N = 20,000, K = 125,
// D = 64: 53 ms; this file's launches at that size 0.9 ms).  About the data's mean m, with z = t - m and w = y - m,
//     S1 = P - w a^T - a w^T + g w w^T,  P = sum R z z^T, a = sum R z, g = sum R,
// so the points' pair features u_n = (z_i z_j for i <= j, z_i, 1) serve all
// centres and [R; R^2] U^T is one digit-slice product (oz.cu) over the points.
// The features are FP64 products; each feature has its own power-of-two grid,
// and so has each centre's R.
//
// The expansion cancels where a centre's points lie close together and far from
// the mean: tr P / tr S1 says by how much (a few units on spread-out data).  And every
// point leaves what the digit products below level 7 would add, about 2^-56 of the grids of
// the centre's R and of the feature, whatever its own R and z: sqrt(N) of that in a sum
// (on few points in grids far above theirs it is much: N = 5001, D = 5, centres on a few
// dozen points: 2e-13 of a critical temperature).  The caller redoes the centres for which
// either is more than 8 bits of 2^-53 of tr S1 with the CUDA-core scatter.
#include "common.cuh"
#include "kernels.cuh"
#include "oz.cuh"
#include "oz_slice.cuh"

#include <math.h>

namespace dgtm {

int launch_ctemp_eig(const CtempPlan &pl, int kb, int D, const double *S, void *Mg, const double *gg,
                     double lim_scale, double *out, cudaStream_t s);

namespace {

constexpr int PANEL = 64;
constexpr int U_FEATURES = 128;  // features of a block
constexpr int SUM_ROWS = 256;    // points of a block of the mean

__host__ __device__ constexpr int rup(int a, int b) { return (a + b - 1) / b * b; }

// mean[d] += sum over the block's points / N, by columns (32 of them, 8 rows at a time)
__global__ void __launch_bounds__(256) mean_kernel(const double *__restrict__ T, int N, int D,
                                                   double *__restrict__ part)
{
    __shared__ double red[8][33];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, d = blockIdx.y * 32 + lane;
    const int n0 = blockIdx.x * SUM_ROWS, n1 = min(N, n0 + SUM_ROWS);
    double s = 0.0;
    if (d < D)
        for (int n = n0 + w; n < n1; n += 8)
            s += T[(size_t) n * D + d];
    red[w][lane] = s;
    __syncthreads();
    if (w == 0 && d < D) {
        for (int i = 1; i < 8; i++)
            s += red[i][lane];
        part[(size_t) blockIdx.x * D + d] = s;
    }
}

__global__ void mean_finish_kernel(const double *__restrict__ part, int blocks, int N, int D,
                                   double *__restrict__ mean)
{
    const int d = blockIdx.x * blockDim.x + threadIdx.x;
    if (d >= D)
        return;
    double s = 0.0;
    for (int b = 0; b < blocks; b++)
        s += part[(size_t) b * D + d];
    mean[d] = s / N;
}

// bits[d] = the largest |t_nd - mean_d|
__global__ void __launch_bounds__(256) zmax_kernel(const double *__restrict__ T, int N, int D,
                                                   const double *__restrict__ mean,
                                                   unsigned long long *__restrict__ bits)
{
    __shared__ unsigned long long red[8][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, d = blockIdx.y * 32 + lane;
    const int n0 = blockIdx.x * SUM_ROWS, n1 = min(N, n0 + SUM_ROWS);
    unsigned long long m = 0ull;
    if (d < D) {
        const double mu = mean[d];
        for (int n = n0 + w; n < n1; n += 8) {
            const unsigned long long b = oz::double_bits(T[(size_t) n * D + d] - mu) & oz::ABS_MASK;
            m = b > m ? b : m;
        }
    }
    red[w][lane] = m;
    __syncthreads();
    if (w == 0 && d < D) {
        for (int i = 1; i < 8; i++)
            m = red[i][lane] > m ? red[i][lane] : m;
        atomicMax(&bits[d], m);
    }
}

// feature f of pairs (i <= j) row by row, then the D coordinates, then 1: (i, j)
// with j = -1 for a coordinate and i = j = -1 for the one
__device__ __forceinline__ void feature_of(int f, int D, int &i, int &j)
{
    const int np = D * (D + 1) / 2;
    if (f >= np) {
        i = f - np < D ? f - np : -1;
        j = -1;
        return;
    }
    // rows from the end hold 1, 2, 3, .. pairs
    const int g = np - 1 - f;
    int r = (int) ((sqrtf(8.0f * (float) g + 1.0f) - 1.0f) * 0.5f);
    while ((r + 1) * (r + 2) / 2 <= g)
        r++;
    while (r * (r + 1) / 2 > g)
        r--;
    i = D - 1 - r;
    j = D - 1 - (g - r * (r + 1) / 2);
}

// A feature's coordinates and power-of-two grid, |z_i z_j| < 2^e; padding features
// have i = j = -2.
struct Feature {
    short i, j;
    int e;
};

__global__ void feature_table_kernel(int F, int Fp, int D, const unsigned long long *__restrict__ zbits,
                                     Feature *__restrict__ tab)
{
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= Fp)
        return;
    int i = -2, j = -2, e = 1;
    if (f < F) {
        feature_of(f, D, i, j);
        if (i >= 0) {
            const double a = oz::bits_double(zbits[i]);
            e = oz::exponent_of(oz::double_bits(j < 0 ? a : a * oz::bits_double(zbits[j])));
        }
    }
    tab[f] = Feature{(short) i, (short) j, e};
}

// planes[p][f][n]: the features of 64 points (z in shared memory) and U_FEATURES
// features a block, one warp per feature, two points a lane; zero past nn and F.
// Bound by the stores: 16 bytes a value.
__global__ void __launch_bounds__(256) features_kernel(const double *__restrict__ T, int nn, int D,
                                                       const double *__restrict__ mean,
                                                       const Feature *__restrict__ ftab, int Fp, int ldn,
                                                       __nv_bfloat16 *__restrict__ planes)
{
    extern __shared__ double z[];  // [D][66]
    const int n0 = blockIdx.x * 64, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int e = threadIdx.x; e < 64 * D; e += 256) {
        const int p = e / D, d = e - p * D;
        z[d * 66 + p] = n0 + p < nn ? T[(size_t) (n0 + p) * D + d] - mean[d] : 0.0;
    }
    __syncthreads();
    const size_t plane = (size_t) Fp * ldn / 2;
    const int f0 = blockIdx.y * U_FEATURES, f1 = min(Fp, f0 + U_FEATURES);
    for (int f = f0 + w; f < f1; f += 8) {
        const Feature t = ftab[f];
        double a = 0.0, b = 0.0;
        if (t.i == -1) {
            a = n0 + 2 * lane < nn ? 1.0 : 0.0;
            b = n0 + 2 * lane + 1 < nn ? 1.0 : 0.0;
        } else if (t.i >= 0) {
            const double2 zi = *(const double2 *) &z[t.i * 66 + 2 * lane];
            a = zi.x;
            b = zi.y;
            if (t.j >= 0) {
                const double2 zj = *(const double2 *) &z[t.j * 66 + 2 * lane];
                a *= zj.x;
                b *= zj.y;
            }
        }
        uint32_t v[oz::DIGITS];
        digit_pairs(oz::to_fixed(a, t.e), oz::to_fixed(b, t.e), v);
        uint32_t *dst = (uint32_t *) planes + ((size_t) f * ldn + n0) / 2 + lane;
#pragma unroll
        for (int p = 0; p < oz::DIGITS; p++)
            dst[(size_t) p * plane] = v[p];
    }
}

// P[f][row] (+)= the product's sums, rows = R then R^2; noise[row] (+)= sqrt(points) times
// the grid of the row's R
__global__ void __launch_bounds__(256) sums_kernel(const double *__restrict__ part, int ntiles, int splits,
                                                   const int *__restrict__ nmin, int rows, int F,
                                                   const Feature *__restrict__ ftab, int first, double rootn,
                                                   double *__restrict__ P, double *__restrict__ noise)
{
    const int t = blockIdx.x, mt = t / ntiles, nt = t - mt * ntiles;
    for (int e = blockIdx.y * 256 + threadIdx.x; e < 128 * 64; e += 256 * gridDim.y) {
        const int r = mt * 128 + (e & 127), f = nt * 64 + (e >> 7);
        if (f >= F)
            continue;
        double sum = 0.0;
        for (int sp = 0; sp < splits; sp++)
            sum += part[((size_t) t * splits + sp) * (128 * 64) + e];
        const int nm = nmin[r];
        const double v = nm >= 0 && nm < 2047 ? scalbn(sum, 5 - nm + ftab[f].e - OZ_SUM_BITS) : 0.0;
        double *dst = P + (size_t) f * rows + r;
        *dst = first ? v : *dst + v;
        if (f == 0) {
            const double d = nm >= 0 && nm < 2047 ? rootn * scalbn(1.0, 5 - nm) : 0.0;
            noise[r] = first ? d : noise[r] + d;
        }
    }
}

// S1, S2 (upper triangles), g and tr P / tr S1 of the batch's centres, one block each
__global__ void __launch_bounds__(256) assemble_kernel(const double *__restrict__ P, int rows, int kpad, int D,
                                                       const Feature *__restrict__ ftab,
                                                       const double *__restrict__ Y,
                                                       const double *__restrict__ mean,
                                                       const double *__restrict__ noise, double *__restrict__ S, double *__restrict__ gsum,
                                                       double *__restrict__ spread)
{
    extern __shared__ double sh[];  // w, a1, a2
    __shared__ double red[32];
    const int k = blockIdx.x, np = D * (D + 1) / 2;
    double *w = sh, *a1 = sh + D, *a2 = sh + 2 * D;
    for (int d = threadIdx.x; d < D; d += 256) {
        w[d] = Y[(size_t) k * D + d] - mean[d];
        a1[d] = P[(size_t) (np + d) * rows + k];
        a2[d] = P[(size_t) (np + d) * rows + kpad + k];
    }
    __syncthreads();
    const double g1 = P[(size_t) (np + D) * rows + k], g2 = P[(size_t) (np + D) * rows + kpad + k];
    double *S1 = S + (size_t) k * 2 * D * D, *S2 = S1 + (size_t) D * D;
    double tp = 0.0, ts = 0.0, tz = 0.0;  // traces: P, S1, the grids of the squares
    for (int f = threadIdx.x; f < np; f += 256) {
        const int i = ftab[f].i, j = ftab[f].j;
        const double p1 = P[(size_t) f * rows + k], p2 = P[(size_t) f * rows + kpad + k];
        const double wi = w[i], wj = w[j];
        // sum R (z_i - w_i)(z_j - w_j) = p - w_i (a_j - g w_j) - a_i w_j
        const double s1 = p1 - wi * fma(-g1, wj, a1[j]) - a1[i] * wj;
        const double s2 = p2 - wi * fma(-g2, wj, a2[j]) - a2[i] * wj;
        S1[(size_t) i * D + j] = s1;
        S2[(size_t) i * D + j] = s2;
        if (i == j) {
            tp += p1;
            ts += s1;
            tz += scalbn(1.0, ftab[f].e);
        }
    }
    tp = block_sum_fixed(tp, red);
    ts = block_sum_fixed(ts, red);
    tz = block_sum_fixed(tz, red);
    if (threadIdx.x == 0) {
        gsum[k] = g1;
        // 2^-56 of the grids against 2^-53 of P: an eighth
        const double lost = fmax(tp, 0.125 * noise[k] * tz);
        spread[k] = lost > 0.0 ? (ts > 0.0 ? lost / ts : INFINITY) : lost;
    }
}

size_t align_up(size_t b) { return (b + 255) / 256 * 256; }

}  // namespace

#define OZ_TRY(expr)           \
    do {                       \
        const int _r = (expr); \
        if (_r != DGTM_OK)     \
            return _r;         \
    } while (0)

int oz_ctemp(OzE *st, const double *T64, const double *Y, const double *yy, const double2 *colstat, int N,
             int D, int K, int sms, double c1, double c, double dcut, const double *gg_dev, double lim_scale,
             size_t budget, double *gsum_dev, double *out_dev, double *spread_dev, int *status,
             cudaStream_t s)
{
    const int F = D * (D + 1) / 2 + D + 1, Fp = rup(F, 64), ntiles = Fp / 64;
    int chunk = 0;
    const int nchunks = oze_chunks(st, &chunk);
    const int cpanels = rup(chunk < N ? chunk : rup(N, PANEL), PANEL) / PANEL;
    // batch of centres (a multiple of 128) within the budget
    const CtempPlan pl = ctemp_plan(N, D, K, false, false, (size_t) 1 << 40, 1);
    const int blocks = ceil_div(N, SUM_ROWS);
    size_t fixed = align_up(sizeof(__nv_bfloat16) * oz::DIGITS * (size_t) Fp * cpanels * PANEL) +
                   align_up(sizeof(double) * D) + align_up(sizeof(unsigned long long) * D) +
                   align_up(sizeof(double) * (size_t) blocks * D) + align_up(sizeof(Feature) * Fp);
    int kpad = rup(K, 128), per = 0, splits = 0;
    size_t need = 0;
    for (;; kpad = rup(kpad / 2, 128)) {
        per = oz_item_panels(2 * (kpad / 128) * ntiles, cpanels, sms);
        splits = ceil_div(cpanels, per);
        need = fixed + align_up(sizeof(__nv_bfloat16) * oz::DIGITS * 2 * (size_t) kpad * cpanels * PANEL) +
               align_up(sizeof(double) * 2 * (size_t) kpad * Fp * splits) +
               align_up(sizeof(double) * 2 * (size_t) kpad * F) +
               (pl.eig_in_smem ? 1 : 2) * align_up(sizeof(double) * (size_t) kpad * 2 * D * D) +
               align_up(sizeof(int) * 2 * kpad) + align_up(sizeof(double) * 2 * kpad);
        if (need <= budget || kpad == 128)
            break;
    }
    unsigned char *base = nullptr;
    if (need > budget || cudaMalloc((void **) &base, need) != cudaSuccess) {
        cudaGetLastError();
        set_error(DGTM_ENOMEM, "oz_ctemp: %zu bytes of scratch", need);
        return DGTM_ENOMEM;
    }
    unsigned char *at = base;
    auto take = [&](size_t bytes) {
        unsigned char *p = at;
        at += align_up(bytes);
        return (void *) p;
    };
    __nv_bfloat16 *U = (__nv_bfloat16 *) take(sizeof(__nv_bfloat16) * oz::DIGITS * (size_t) Fp * cpanels * PANEL);
    double *mean = (double *) take(sizeof(double) * D);
    unsigned long long *zbits = (unsigned long long *) take(sizeof(unsigned long long) * D);
    double *mpart = (double *) take(sizeof(double) * (size_t) blocks * D);
    Feature *ftab = (Feature *) take(sizeof(Feature) * Fp);
    const int rows = 2 * kpad;
    __nv_bfloat16 *R = (__nv_bfloat16 *) take(sizeof(__nv_bfloat16) * oz::DIGITS * (size_t) rows * cpanels * PANEL);
    double *part = (double *) take(sizeof(double) * (size_t) rows * Fp * splits);
    double *P = (double *) take(sizeof(double) * (size_t) rows * F);
    double *S = (double *) take(sizeof(double) * (size_t) kpad * 2 * D * D);
    double *Mg = pl.eig_in_smem ? nullptr : (double *) take(sizeof(double) * (size_t) kpad * 2 * D * D);
    int *nmin = (int *) take(sizeof(int) * rows);
    double *noise = (double *) take(sizeof(double) * rows);
    const size_t zsmem = sizeof(double) * 66 * (size_t) D, asmem = sizeof(double) * 3 * (size_t) D;

    auto body = [&]() -> int {
        DGTM_CUDA_TRY(cudaMemsetAsync(zbits, 0, sizeof(unsigned long long) * D, s));
        DGTM_CUDA_TRY(cudaFuncSetAttribute(features_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) zsmem));
        mean_kernel<<<dim3(blocks, ceil_div(D, 32)), 256, 0, s>>>(T64, N, D, mpart);
        mean_finish_kernel<<<ceil_div(D, 64), 64, 0, s>>>(mpart, blocks, N, D, mean);
        zmax_kernel<<<dim3(blocks, ceil_div(D, 32)), 256, 0, s>>>(T64, N, D, mean, zbits);
        feature_table_kernel<<<ceil_div(Fp, 256), 256, 0, s>>>(F, Fp, D, zbits, ftab);
        DGTM_CUDA_TRY(cudaGetLastError());
        OZ_TRY(oze_refer(st, Y, yy, colstat, c1, c, dcut, s));
        for (int k0 = 0; k0 < K; k0 += kpad) {
            const int kb = K - k0 < kpad ? K - k0 : kpad;
            // rows without a centre count as zero
            DGTM_CUDA_TRY(cudaMemsetAsync(nmin, 0xFF, sizeof(int) * rows, s));
            for (int ch = 0; ch < nchunks; ch++) {
                const int n0 = ch * chunk, nn = N - n0 < chunk ? N - n0 : chunk, ldn = rup(nn, PANEL);
                OZ_TRY(oze_r_digits(st, ch, k0, kb, c, false, true, rows, R, nmin, s));
                OZ_TRY(oze_r_digits(st, ch, k0, kb, c, true, false, rows, R + (size_t) kpad * ldn, nmin + kpad, s));
                features_kernel<<<dim3(ldn / 64, ceil_div(Fp, U_FEATURES)), 256, zsmem, s>>>(
                    T64 + (size_t) n0 * D, nn, D, mean, ftab, Fp, ldn, U);
                DGTM_CUDA_TRY(cudaGetLastError());
                OzGemm g;
                g.A = R;
                g.B = U;
                g.a_rows = rows;
                g.b_rows = Fp;
                g.panels = ldn / PANEL;
                g.a_ld = g.b_ld = ldn;
                g.mtiles = rows / 128;
                g.ntiles = ntiles;
                g.sums = part;
                g.item_panels = per;
                OZ_TRY(launch_oz_gemm(g, sms, status, s));
                sums_kernel<<<dim3(g.mtiles * ntiles, 8), 256, 0, s>>>(part, ntiles, ceil_div(g.panels, per),
                                                                       nmin, rows, F, ftab, ch == 0 ? 1 : 0, sqrt((double) nn),
                                                                       P, noise);
                DGTM_CUDA_TRY(cudaGetLastError());
            }
            assemble_kernel<<<kb, 256, asmem, s>>>(P, rows, kpad, D, ftab, Y + (size_t) k0 * D, mean, noise, S, gsum_dev + k0,
                                                   spread_dev + k0);
            DGTM_CUDA_TRY(cudaGetLastError());
            OZ_TRY(launch_ctemp_eig(pl, kb, D, S, Mg, gg_dev ? gg_dev + k0 : gsum_dev + k0, lim_scale,
                                    out_dev + (size_t) 2 * k0, s));
        }
        return DGTM_OK;
    };
    int rc = body();
    const cudaError_t e = cudaStreamSynchronize(s);  // the scratch goes back below
    cudaFree(base);
    if (rc == DGTM_OK && e != cudaSuccess) {
        set_error(DGTM_ECUDA, "oz_ctemp: %s", cudaGetErrorString(e));
        rc = DGTM_ECUDA;
    }
    return rc;
}

}  // namespace dgtm
