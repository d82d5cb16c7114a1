// mstep.cu -- the small FP64 kernels of the M-step, shared by every form.
//
//   reduce_slices : G_k = sum_s Gpart[s][k], RT = sum_s RTpart[s] (fixed order)
//   form_ab       : A = FI^T diag(G) FI, B = FI^T RT     (dagtm/dagtm.cxx:1715-1761),
//                   K-sliced 4 x 4 register tiles, slice partials summed in order
//   solve         : A W = B, FP64 Cholesky (numerically dependent pivots dropped;
//                   one block for M1 <= 110, panels over the GPU above that; one
//                   warp per right-hand side in the substitution)
//                   or symmetric-eigen pseudo-inverse
//                   with exactly-zero eigenvalues dropped (the semantics of
//                   gsl_linalg_SV_solve used by dagtm_solve2, comm/comm.c:1299-1348)
//   update_y      : Y = FI W (dagtm/dagtm.cxx:1769), |y_k|^2, the beta terms, and
//                   the copies of Y the E-step of the FP32 / split form reads
//   sum_ratio     : beta = N D / (sum_k G_k|y_k|^2 - 2 y_k.RT_k + sum_n |t_n|^2)
//                   = N D / sum_kn R_kn |y_k - t_n|^2 (comm/mpicomm.c:276-302
//                   evaluates the same sum over an explicit K x N distance matrix;
//                   every column of R sums to one, which gives the closed form)
//
// Every reduction runs in a fixed order, so repeated runs are bit-identical.
#include "common.cuh"
#include "f32pair.cuh"
#include "kernels.cuh"

#include <cuda_bf16.h>

#include <math.h>
#include <type_traits>

namespace dgtm {

__global__ void reduce_slices_kernel(const double *__restrict__ Gpart,
                                     const double *__restrict__ RTpart, int nsplit, int K, int D,
                                     double *__restrict__ G, double *__restrict__ RT)
{
    const size_t KD = (size_t) K * D;
    for (size_t i = blockIdx.x * (size_t) blockDim.x + threadIdx.x; i < KD + K;
         i += (size_t) gridDim.x * blockDim.x) {
        double s = 0.0;
        if (i < KD) {
            for (int p = 0; p < nsplit; p++)
                s += RTpart[(size_t) p * KD + i];
            RT[i] = s;
        } else {
            const size_t k = i - KD;
            for (int p = 0; p < nsplit; p++)
                s += Gpart[(size_t) p * K + k];
            G[k] = s;
        }
    }
}

int launch_reduce_slices(const double *Gpart, const double *RTpart, int nsplit, int K, int D,
                         double *G, double *RT, cudaStream_t s)
{
    const size_t n = (size_t) K * D + K;
    int blocks = (int) ((n + 255) / 256);
    if (blocks > 4096)
        blocks = 4096;
    reduce_slices_kernel<<<blocks, 256, 0, s>>>(Gpart, RTpart, nsplit, K, D, G, RT);
    DGTM_CUDA_TRY(cudaGetLastError());
    return DGTM_OK;
}

// C = FI^T [RT | diag(G) FI] (M1 x (D + M1)): B = C[:, :D], A = C[:, D:]
// (the upper triangle of A and its diagonal tiles only).
// The K rows are cut into slices; each thread keeps a 4 x 4 FP64 tile of C over its
// slice, fed from shared memory; the slices' partial tiles are then summed in slice
// order.  Every element is one multiply-add chain over its slice, whichever kernel
// forms it.  The FP64 pipe (about 2 FMA per clock per SM on this part) bounds both.
//
// form_ab_rows_kernel (M1 <= AB_ROWS_MAX): a block stages whole rows of both
// operands for 256 consecutive 4 x 4 tiles, so no tile of a small basis is padding.
// form_ab_partial_kernel (above): a block forms a 64 x 64 tile of C over its
// slice, a thread 4 x 4 of it, from shared-memory copies of AB_KC rows of its
// FI and right-operand columns (the next rows' loads in flight meanwhile).  A warp
// covers 8 rows x 64 columns; warps past M1 or below A's diagonal do nothing.
// K = 32768, M1 = 513, D = 166: 14.3 ms (11.3 ms at the pipe's 0.63 TFMA/s), by
// whole rows, staged and scaled by 86 blocks, 19.4 ms.  K = 8000, M1 = 65: 0.37 ms,
// its second tile row holding one row, against 0.25 ms by whole rows.
constexpr int AB_ROWS_MAX = 128;
constexpr int AB_THREADS = 256;
constexpr int AB_SLICES = 76;
constexpr int AB_TILE = 64;
constexpr int AB_KC = 16;
constexpr int AB_LD = AB_TILE + 2;

__global__ void __launch_bounds__(AB_THREADS) form_ab_rows_kernel(
    const double *__restrict__ FI, const double *__restrict__ G, const double *__restrict__ RT,
    int K, int M1, int D, int M1p, int Wp, int kc, int slice_len, double *__restrict__ Cpart,
    const int *__restrict__ only)
{
    if (only && !*only)
        return;
    extern __shared__ double sh[];
    double *FIs = sh;                       // kc x M1p
    double *Rs = sh + (size_t) kc * M1p;    // kc x Wp
    const int W = D + M1;
    const int nct = Wp / 4;
    const int tile = blockIdx.y * AB_THREADS + threadIdx.x;
    const bool in_range = tile < (M1p / 4) * nct;
    const int m0 = in_range ? (tile / nct) * 4 : 0, c0 = in_range ? (tile % nct) * 4 : 0;
    // a tile of A strictly below the diagonal is not formed: the reduction
    // takes A from its upper triangle and mirrors it
    const bool active = in_range && !(c0 >= D && c0 + 3 - D < m0);
    const int kb = blockIdx.x * slice_len, ke = min(K, kb + slice_len);
    double acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++)
            acc[i][j] = 0.0;
    for (int k0 = kb; k0 < ke; k0 += kc) {
        const int nk = min(kc, ke - k0);
        __syncthreads();
        for (int e = threadIdx.x; e < kc * M1p; e += AB_THREADS) {
            const int r = e / M1p, m = e % M1p;
            FIs[e] = (r < nk && m < M1) ? FI[(size_t) (k0 + r) * M1 + m] : 0.0;
        }
        for (int e = threadIdx.x; e < kc * Wp; e += AB_THREADS) {
            const int r = e / Wp, c = e % Wp;
            double v = 0.0;
            if (r < nk) {
                const int k = k0 + r;
                if (c < D)
                    v = RT[(size_t) k * D + c];
                else if (c < W)
                    v = G[k] * FI[(size_t) k * M1 + (c - D)];
            }
            Rs[e] = v;
        }
        __syncthreads();
        if (active) {
            for (int r = 0; r < nk; r++) {
                const double2 a01 = *(const double2 *) &FIs[(size_t) r * M1p + m0];
                const double2 a23 = *(const double2 *) &FIs[(size_t) r * M1p + m0 + 2];
                const double2 b01 = *(const double2 *) &Rs[(size_t) r * Wp + c0];
                const double2 b23 = *(const double2 *) &Rs[(size_t) r * Wp + c0 + 2];
                const double av[4] = {a01.x, a01.y, a23.x, a23.y};
                const double bv[4] = {b01.x, b01.y, b23.x, b23.y};
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++)
                        acc[i][j] = fma(av[i], bv[j], acc[i][j]);
            }
        }
    }
    if (!active)
        return;
    double *dst = Cpart + (size_t) blockIdx.x * M1 * W;
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (m0 + i < M1 && c0 + j < W)
                dst[(size_t) (m0 + i) * W + c0 + j] = acc[i][j];
}

__global__ void __launch_bounds__(AB_THREADS) form_ab_partial_kernel(
    const double *__restrict__ FI, const double *__restrict__ G, const double *__restrict__ RT,
    int K, int M1, int D, int nct, int slice_len, double *__restrict__ Cpart, const int *__restrict__ only)
{
    if (only && !*only)
        return;
    __shared__ __align__(16) double FIs[AB_KC * AB_LD], Rs[AB_KC * AB_LD];
    const int W = D + M1;
    const int mt = (blockIdx.y / nct) * AB_TILE, ct = (blockIdx.y % nct) * AB_TILE;
    // a tile of A strictly below the diagonal is not formed: the reduction
    // takes A from its upper triangle and mirrors it
    if (ct >= D && ct + AB_TILE - 1 - D < mt)
        return;
    const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
    const int m0 = mt + 4 * ty, c0 = ct + 4 * tx;
    const int wm = mt + 8 * (threadIdx.x >> 5);  // the warp's first row
    const bool active = wm < M1 && !(ct >= D && ct + AB_TILE - 1 - D < wm);
    const int kb = blockIdx.x * slice_len, ke = min(K, kb + slice_len);
    // staging: row sr + 4 q, column sc of both operands
    const int sr = threadIdx.x >> 6, sc = threadIdx.x & 63;
    const int gm = mt + sc, gc = ct + sc;
    double fv[AB_KC / 4], rv[AB_KC / 4];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int q = 0; q < AB_KC / 4; q++) {
            const int k = k0 + sr + 4 * q;
            fv[q] = (k < ke && gm < M1) ? FI[(size_t) k * M1 + gm] : 0.0;
            double v = 0.0;
            if (k < ke) {
                if (gc < D)
                    v = RT[(size_t) k * D + gc];
                else if (gc < W)
                    v = G[k] * FI[(size_t) k * M1 + (gc - D)];
            }
            rv[q] = v;
        }
    };
    double acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++)
            acc[i][j] = 0.0;
    fetch(kb);
    for (int k0 = kb; k0 < ke; k0 += AB_KC) {
        const int nk = min(AB_KC, ke - k0);
        __syncthreads();
#pragma unroll
        for (int q = 0; q < AB_KC / 4; q++) {
            FIs[(sr + 4 * q) * AB_LD + sc] = fv[q];
            Rs[(sr + 4 * q) * AB_LD + sc] = rv[q];
        }
        __syncthreads();
        if (k0 + AB_KC < ke)
            fetch(k0 + AB_KC);
        if (active) {
#pragma unroll 4
            for (int r = 0; r < nk; r++) {
                const double2 a01 = *(const double2 *) &FIs[r * AB_LD + 4 * ty];
                const double2 a23 = *(const double2 *) &FIs[r * AB_LD + 4 * ty + 2];
                const double2 b01 = *(const double2 *) &Rs[r * AB_LD + 4 * tx];
                const double2 b23 = *(const double2 *) &Rs[r * AB_LD + 4 * tx + 2];
                const double av[4] = {a01.x, a01.y, a23.x, a23.y};
                const double bv[4] = {b01.x, b01.y, b23.x, b23.y};
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++)
                        acc[i][j] = fma(av[i], bv[j], acc[i][j]);
            }
        }
    }
    if (!active)
        return;
    double *dst = Cpart + (size_t) blockIdx.x * M1 * W;
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (m0 + i < M1 && c0 + j < W)
                dst[(size_t) (m0 + i) * W + c0 + j] = acc[i][j];
}

// sum over slices in slice order; A is written from its upper triangle and
// mirrored, so it is exactly symmetric
__global__ void form_ab_reduce_kernel(const double *__restrict__ Cpart, int nslice, int M1, int D,
                                      double *__restrict__ A, double *__restrict__ B,
                                      int *__restrict__ flag, const int *__restrict__ only)
{
    if (only && !*only)
        return;
    if (blockIdx.x == 0 && threadIdx.x < 3)
        flag[threadIdx.x] = 0;
    const int W = D + M1;
    const size_t total = (size_t) M1 * W;
    for (size_t i = blockIdx.x * (size_t) blockDim.x + threadIdx.x; i < total;
         i += (size_t) gridDim.x * blockDim.x) {
        const int m = (int) (i / W), c = (int) (i % W);
        if (c >= D && c - D < m)
            continue;
        // in slice order; sixteen loads in flight (one at a time the 67 to 76 slices
        // of a small basis cost their memory latency each)
        double sum = 0.0;
        int sl = 0;
        for (; sl + 16 <= nslice; sl += 16) {
            double v[16];
#pragma unroll
            for (int q = 0; q < 16; q++)
                v[q] = Cpart[(size_t) (sl + q) * total + i];
#pragma unroll
            for (int q = 0; q < 16; q++)
                sum += v[q];
        }
        for (; sl < nslice; sl++)
            sum += Cpart[(size_t) sl * total + i];
        if (c < D) {
            B[(size_t) m * D + c] = sum;
        } else {
            const int j = c - D;
            A[(size_t) m * M1 + j] = sum;
            A[(size_t) j * M1 + m] = sum;
        }
    }
}

size_t form_ab_scratch_doubles(int M1, int D) { return (size_t) AB_SLICES * M1 * (D + M1); }

int launch_form_ab(const double *FI, const double *G, const double *RT, int K, int M1, int D,
                   double *A, double *B, double *scratch, int *flag, cudaStream_t s, const int *only)
{
    const int slice_len = ceil_div(K, AB_SLICES);
    const int nslice = ceil_div(K, slice_len);
    if (M1 <= AB_ROWS_MAX) {
        const int M1p = (M1 + 3) / 4 * 4, Wp = (D + M1 + 3) / 4 * 4;
        int kc = (int) ((48 * 1024) / (sizeof(double) * (size_t) (M1p + Wp)));
        kc = kc > 16 ? 16 : kc;  // at least 11: M1 + D <= 384
        form_ab_rows_kernel<<<dim3(nslice, ceil_div((M1p / 4) * (Wp / 4), AB_THREADS)), AB_THREADS,
                              sizeof(double) * (size_t) kc * (M1p + Wp), s>>>(FI, G, RT, K, M1, D, M1p, Wp, kc,
                                                                              slice_len, scratch, only);
    } else {
        const int nct = ceil_div(D + M1, AB_TILE);
        form_ab_partial_kernel<<<dim3(nslice, ceil_div(M1, AB_TILE) * nct), AB_THREADS, 0, s>>>(
            FI, G, RT, K, M1, D, nct, slice_len, scratch, only);
    }
    DGTM_CUDA_TRY(cudaGetLastError());
    const size_t total = (size_t) M1 * (D + M1);
    // small blocks: a small basis has few elements, and their loads spread over the SMs
    const int blocks = (int) ((total + 63) / 64);
    form_ab_reduce_kernel<<<blocks, 64, 0, s>>>(scratch, nslice, M1, D, A, B, flag, only);
    DGTM_CUDA_TRY(cudaGetLastError());
    return DGTM_OK;
}

// ---------------------------------------------------------------------------
// solvers
// ---------------------------------------------------------------------------
constexpr int SMEM_SOLVE_MAX = 110;  // M1 up to which L lives in shared memory
constexpr int CHOL_MAX_M1 = 1024;  // the large substitution's shared vector

// 1/sqrt(d) for a positive normal d: an FP32 estimate refined by two
// Newton-Raphson steps for f(r) = 1/r^2 - d, r <- r (3 - d r^2) / 2 (each
// step doubles the correct bits: 23 -> 46 -> full FP64).  Outside the FP32
// exponent range the FP64 library square root is used.
__device__ __forceinline__ double rsqrt_nr(double d)
{
    if (!(d > 1e-30 && d < 1e30))
        return 1.0 / sqrt(d);
    double r = (double) rsqrtf((float) d);
#pragma unroll
    for (int it = 0; it < 2; it++)
        r = r * fma(-0.5 * d * r, r, 1.5);
    return r;
}

// Cholesky with pivot drops.  A pivot that keeps less than CHOL_DROP of its
// diagonal (the column adds no new direction at FP64 precision) is dropped:
// its diagonal and column are stored as 0 and that unknown is fixed at 0,
// which keeps the solve defined when A = FI^T diag(G) FI is numerically
// singular (wide basis functions).  L (lower triangle) goes to
// work[0 .. M1*M1), the reciprocal diagonal to work[M1*M1 .. M1*M1 + M1) (0
// for a dropped pivot); flag[1] counts the drops.
constexpr double CHOL_DROP = 1e-12;
constexpr int CHOL_THREADS = 256;

__device__ __forceinline__ void chol_pivot(double *L, const double *adiag, int M1, int j,
                                           double *rinv, int *bad, int *ndrop)
{
    const size_t jj = (size_t) j * M1 + j;
    const double d = L[jj], ajj = adiag[j];
    double r = 0.0;
    if (!isfinite(d)) {
        *bad = 1;
        L[jj] = 0.0;
    } else if (!(d > CHOL_DROP * ajj)) {
        (*ndrop)++;
        L[jj] = 0.0;  // marks a dropped unknown
    } else {
        r = rsqrt_nr(d);
        L[jj] = d * r;
    }
    rinv[j] = r;
}

// Blocked right-looking Cholesky for M1 > SMEM_SOLVE_MAX, in panels of CHB
// columns: chol_diag_kernel factorises the panel's diagonal block with
// chol_pivot's drop rule (in registers), chol_rows_kernel
// takes every row below through the same columns (one row a thread, so the rows
// spread over the SMs), and chol_update_kernel (one CTA per 32 x 32 tile) subtracts
// the panel's L21 L21^T from the trailing lower triangle.  Per element the
// operations and their order are those of a factorisation column by column.  One
// CTA doing a panel's columns over all rows in global memory, four barriers a
// column, took 0.26 ms a panel at M1 = 513; diagonal block and rows take 0.055.
// The layout is that of the shared-memory kernel below: the
// scaled L (L_ij = a_ij / sqrt(d_j)) in the lower
// triangle of work, the reciprocal diagonal after it (0 for a dropped pivot),
// flag[0] for a non-finite pivot and flag[1] counting the drops.
constexpr int CHB = 32;

// Four warps, because a sub-partition issues one FP64 instruction in 64 clocks: lane
// = row, warp w holds the columns 4 q + w.  The owner of column j + 1 updates it
// first and finishes it while the others still take column j off theirs.
constexpr int CHD_WARPS = 4;

__global__ void __launch_bounds__(32 * CHD_WARPS) chol_diag_kernel(const double *__restrict__ A, int M1, int p0,
                                                                   int w, double *__restrict__ work, int *flag)
{
    __shared__ double col[2][CHB];
    constexpr int Q = CHB / CHD_WARPS;
    double *L = work;
    double *rinv = work + (size_t) M1 * M1;
    const int i = threadIdx.x & 31, wp = threadIdx.x >> 5;
    double a[Q];  // row p0 + i, columns CHD_WARPS q + wp
    const double *row = L + (size_t) (p0 + min(i, w - 1)) * M1 + p0;
#pragma unroll
    for (int q = 0; q < Q; q++)
        a[q] = CHD_WARPS * q + wp < w ? row[CHD_WARPS * q + wp] : 0.0;
    const double diag = A[(size_t) (p0 + min(i, w - 1)) * M1 + p0 + min(i, w - 1)];
    int bad = 0, ndrop = 0;
    // column j in registers q of its owner: pivot and scaling
    auto finish = [&](double &x, int j) {
        const double d = __shfl_sync(0xffffffffu, x, j), ajj = __shfl_sync(0xffffffffu, diag, j);
        double r = 0.0, ljj = 0.0;  // 0 marks a dropped unknown
        if (!isfinite(d)) {
            bad = 1;
        } else if (!(d > CHOL_DROP * ajj)) {
            ndrop++;
        } else {
            r = rsqrt_nr(d);
            ljj = d * r;
        }
        x = i == j ? ljj : i > j ? x * r : x;
        col[j & 1][i] = x;
        if (i == j)
            rinv[p0 + j] = r;
    };
    if (wp == 0)
        finish(a[0], 0);
    __syncthreads();
#pragma unroll
    for (int j = 0; j < CHB; j++) {
        if (j + 1 < w) {  // uniform
            const double lij = col[j & 1][i];
            // column j + 1 first, by its owner
            const int qn = (j + 1) / CHD_WARPS;
            if (wp == (j + 1) % CHD_WARPS) {
                const double lkj = col[j & 1][j + 1];
                if (i >= j + 1)
                    a[qn < Q ? qn : 0] = fma(-lij, lkj, a[qn < Q ? qn : 0]);
                finish(a[qn < Q ? qn : 0], j + 1);
            }
#pragma unroll
            for (int q = 0; q < Q; q++) {
                const int k = CHD_WARPS * q + wp;
                if (CHD_WARPS * q + CHD_WARPS - 1 > j + 1 && k > j + 1) {
                    const double lkj = col[j & 1][k];
                    if (i >= k)
                        a[q] = fma(-lij, lkj, a[q]);
                }
            }
        }
        __syncthreads();
    }
    if (i < w) {
        double *dst = L + (size_t) (p0 + i) * M1 + p0;
#pragma unroll
        for (int q = 0; q < Q; q++)
            if (CHD_WARPS * q + wp <= i)
                dst[CHD_WARPS * q + wp] = a[q];
    }
    if (i == 0) {
        if (bad)
            flag[0] = DGTM_ENONFINITE;
        if (ndrop)
            atomicAdd(&flag[1], ndrop);
    }
}

// rows below the diagonal block: column j scaled by r_j, then the later columns less
// l_ij l_kj
__global__ void __launch_bounds__(32) chol_rows_kernel(int M1, int p0, double *__restrict__ work)
{
    __shared__ double Ld[CHB][CHB + 1], r[CHB];
    double *L = work;
    const double *rinv = work + (size_t) M1 * M1;
    const int i0 = p0 + CHB + blockIdx.x * 32, lane = threadIdx.x;
    __shared__ double T[32][CHB + 1];  // the 32 rows, through shared memory for whole lines
    for (int q = 0; q < 32; q++) {
        Ld[q][lane] = L[(size_t) (p0 + q) * M1 + p0 + lane];
        T[q][lane] = i0 + q < M1 ? L[(size_t) (i0 + q) * M1 + p0 + lane] : 0.0;
    }
    r[lane] = rinv[p0 + lane];
    __syncwarp();
    double a[CHB];
#pragma unroll
    for (int k = 0; k < CHB; k++)
        a[k] = T[lane][k];
#pragma unroll
    for (int j = 0; j < CHB; j++) {
        a[j] *= r[j];
#pragma unroll
        for (int k = j + 1; k < CHB; k++)
            a[k] = fma(-a[j], Ld[k][j], a[k]);
    }
#pragma unroll
    for (int k = 0; k < CHB; k++)
        T[lane][k] = a[k];
    __syncwarp();
    for (int q = 0; q < 32 && i0 + q < M1; q++)
        L[(size_t) (i0 + q) * M1 + p0 + lane] = T[q][lane];
}

// L[i][k] -= sum_q L[i][p0 + q] L[k][p0 + q] over the panel's w columns, for
// i >= k >= p0 + w: tile (ti, tk), tk <= ti, from the block index
__global__ void __launch_bounds__(256) chol_update_kernel(int M1, int p0, int w,
                                                          double *__restrict__ work)
{
    __shared__ double Li[32][CHB + 1], Lk[32][CHB + 1];
    const int t0 = p0 + w;
    int x = blockIdx.x, ti = 0;
    while (x > ti) {
        x -= ti + 1;
        ti++;
    }
    const int tk = x;
    const int i0 = t0 + 32 * ti, k0 = t0 + 32 * tk;
    double *L = work;
    for (int e = threadIdx.x; e < 32 * w; e += 256) {
        const int r = e / w, q = e - (e / w) * w;
        Li[r][q] = (i0 + r < M1) ? L[(size_t) (i0 + r) * M1 + p0 + q] : 0.0;
        Lk[r][q] = (k0 + r < M1) ? L[(size_t) (k0 + r) * M1 + p0 + q] : 0.0;
    }
    __syncthreads();
    const int r = threadIdx.x >> 3, c0 = threadIdx.x & 7;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    for (int q = 0; q < w; q++) {
        const double a = Li[r][q];
#pragma unroll
        for (int m = 0; m < 4; m++)
            acc[m] = fma(a, Lk[c0 + 8 * m][q], acc[m]);
    }
    const int i = i0 + r;
#pragma unroll
    for (int m = 0; m < 4; m++) {
        const int k = k0 + c0 + 8 * m;
        if (i < M1 && k <= i)
            L[(size_t) i * M1 + k] -= acc[m];
    }
}

// The same factorisation with L in shared memory (M1 <= SMEM_SOLVE_MAX),
// balanced over the threads.  The trailing triangle of step j, the (i, k) with
// j < k <= i < M1, is the first n_j (n_j + 1) / 2 entries of a table ordered by
// k, then i, both descending (entry a (a + 1) / 2 + b holds k = M1 - 1 - a,
// i = M1 - 1 - b), so each step's elements spread evenly.  Per column j: the
// scaled column u_i = a_ij r_j goes to a shared vector (and to the free upper
// triangle), then every element takes one FMA, L[i][k] -= u_i u_k.  The next
// pivot (j+1, j+1) is the last entry of step j; its thread walks its entries
// in reverse, so it updates the pivot first and takes its reciprocal square
// root while the other threads work.
__global__ void __launch_bounds__(CHOL_THREADS) cholesky_small_kernel(const double *__restrict__ A,
                                                                     int M1,
                                                                     double *__restrict__ work,
                                                                     int *flag)
{
    extern __shared__ double sh[];
    double *rinv = sh, *adiag = sh + M1, *u = sh + 2 * M1, *L = sh + 3 * M1;
    uint32_t *tab = (uint32_t *) (L + M1 * M1);
    __shared__ int bad, ndrop;
    const int tid = threadIdx.x;
    const int n2 = M1 * M1, npair0 = M1 * (M1 - 1) / 2;
    if (tid == 0) {
        bad = 0;
        ndrop = 0;
    }
#pragma unroll 4
    for (int e = tid; e < n2; e += CHOL_THREADS)
        L[e] = A[e];
    for (int j = tid; j < M1; j += CHOL_THREADS)
        adiag[j] = A[j * M1 + j];
    for (int t = tid; t < npair0; t += CHOL_THREADS) {
        int a = (int) ((sqrtf(8.0f * (float) t + 1.0f) - 1.0f) * 0.5f);
        while ((a + 1) * (a + 2) / 2 <= t)
            a++;
        while (a * (a + 1) / 2 > t)
            a--;
        const int b = t - a * (a + 1) / 2;
        tab[t] = ((uint32_t) (M1 - 1 - b) << 16) | (uint32_t) (M1 - 1 - a);
    }
    __syncthreads();
    if (tid == 0)
        chol_pivot(L, adiag, M1, 0, rinv, &bad, &ndrop);
    for (int j = 0; j < M1; j++) {
        __syncthreads();  // r_j published, step j-1's updates done
        const double rj = rinv[j];
        for (int i = j + 1 + tid; i < M1; i += CHOL_THREADS) {
            const double ui = L[i * M1 + j] * rj;
            u[i] = ui;
            L[j * M1 + i] = ui;
        }
        __syncthreads();
        const int nj = M1 - 1 - j, npair = nj * (nj + 1) / 2;
        if (tid < npair) {
            for (int t = tid + (npair - 1 - tid) / CHOL_THREADS * CHOL_THREADS; t >= tid;
                 t -= CHOL_THREADS) {
                const uint32_t ik = tab[t];
                const int i = (int) (ik >> 16), k = (int) (ik & 0xFFFFu);
                L[i * M1 + k] = fma(-u[i], u[k], L[i * M1 + k]);
                if (t == npair - 1)
                    chol_pivot(L, adiag, M1, j + 1, rinv, &bad, &ndrop);
            }
        }
    }
    __syncthreads();
    for (int e = tid; e < n2; e += CHOL_THREADS) {
        const int i = e / M1, k = e - i * M1;
        if (k < i)
            work[e] = L[k * M1 + i];
        else if (k == i)
            work[e] = L[e];
    }
    for (int j = tid; j < M1; j += CHOL_THREADS)
        work[n2 + j] = rinv[j];
    if (tid == 0) {
        flag[0] = bad ? DGTM_ENONFINITE : 0;
        flag[1] = ndrop;
    }
}

// Forward (L y = b) and back (L^T w = y) substitution, right-looking, one
// right-hand side (column of B) a CTA.  For an entry p the finished entries i are
// taken off in the order i = 0, 1, .. (forward) and from the end (back), one FMA
// each, in both kernels.
//
// L in shared memory (M1 <= SMEM_SOLVE_MAX): one warp, lane l holding entries l,
// l + 32, ... in NR = ceil(M1 / 32) registers; step i broadcasts the finished entry
// and every lane updates the registers that can still change.  The CTA's other
// warps only load L.
constexpr int TRI_THREADS = 128;

template <int NR>
__global__ void __launch_bounds__(TRI_THREADS) tri_solve_kernel(const double *__restrict__ Lg,
                                                                const double *__restrict__ B,
                                                                int M1, int D,
                                                                const int *__restrict__ flag,
                                                                double *__restrict__ W)
{
    extern __shared__ double sh[];
    if (flag[0] != 0)
        return;  // non-finite factorisation: reported by the host
    const int n = M1 * M1 + M1;
#pragma unroll 8
    for (int i = threadIdx.x; i < n; i += TRI_THREADS)
        sh[i] = Lg[i];
    __syncthreads();
    if (threadIdx.x >= 32)
        return;
    const double *L = sh, *inv = sh + (size_t) M1 * M1;
    const int lane = threadIdx.x, c = blockIdx.x;
    double x[NR];
#pragma unroll
    for (int r = 0; r < NR; r++) {
        const int p = lane + 32 * r;
        x[r] = (p < M1) ? B[(size_t) p * D + c] : 0.0;
    }
    // forward: y_i = x_i / L_ii, then x_p -= L_pi y_i for p > i; entry i sits
    // in register rb = i / 32 of lane i % 32, and only registers rb.. hold p > i
#pragma unroll
    for (int rb = 0; rb < NR; rb++) {
        const int iend = min(32, M1 - 32 * rb);
        for (int il = 0; il < iend; il++) {
            const int i = 32 * rb + il;
            const double yi = __shfl_sync(0xffffffffu, x[rb], il) * inv[i];
#pragma unroll
            for (int r = rb; r < NR; r++) {
                const int p = lane + 32 * r;
                if (p == i)
                    x[r] = yi;
                else if (p > i && p < M1)
                    x[r] = fma(-L[(size_t) p * M1 + i], yi, x[r]);
            }
        }
    }
    // back: w_i = y_i / L_ii, then y_p -= L_ip w_i for p < i (registers ..rb)
#pragma unroll
    for (int rb = NR - 1; rb >= 0; rb--) {
        const int iend = min(32, M1 - 32 * rb);
        for (int il = iend - 1; il >= 0; il--) {
            const int i = 32 * rb + il;
            const double wi = __shfl_sync(0xffffffffu, x[rb], il) * inv[i];
#pragma unroll
            for (int r = 0; r <= rb; r++) {
                const int p = lane + 32 * r;
                if (p == i)
                    x[r] = wi;
                else if (p < i)
                    x[r] = fma(-L[(size_t) i * M1 + p], wi, x[r]);
            }
        }
    }
#pragma unroll
    for (int r = 0; r < NR; r++) {
        const int p = lane + 32 * r;
        if (p < M1)
            W[(size_t) p * D + c] = x[r];
    }
}

// L beyond shared memory: blocks of 32 entries.  Warp 0 solves a block against L's
// 32 x 32 diagonal block; then all four warps (a sub-partition issues one FP64
// instruction in 64 clocks) take its 32 entries off the others, a thread an entry at
// a time, with L read by whole lines: a forward step needs columns, from the
// transposed copy LT.  M1 = 513, D = 166: 0.54 ms; 3.0 ms with one warp reading
// columns across rows, four right-hand sides a CTA.
__global__ void __launch_bounds__(TRI_THREADS) tri_solve_large_kernel(const double *__restrict__ L,
                                                                      const double *__restrict__ LT,
                                                                      const double *__restrict__ inv,
                                                                      const double *__restrict__ B, int M1, int D,
                                                                      const int *__restrict__ flag,
                                                                      double *__restrict__ W)
{
    __shared__ double x[1024 + 32], y[32], dg[32][33];
    if (flag[0] != 0)
        return;
    const int tid = threadIdx.x, lane = tid & 31, c = blockIdx.x;
    for (int p = tid; p < M1; p += TRI_THREADS)
        x[p] = B[(size_t) p * D + c];
    const int nb = (M1 + 31) / 32;
    for (int pass = 0; pass < 2; pass++) {
        for (int q = 0; q < nb; q++) {
            const int b = pass ? nb - 1 - q : q, i0 = 32 * b, w = min(32, M1 - i0);
            // dg[s][l]: what step s takes off entry l of the block (L_{l s} forward, L_{s l} back)
            for (int s = tid >> 5; s < 32; s += TRI_THREADS / 32)
                dg[s][lane] = (s < w && lane < w) ? (pass ? L : LT)[(size_t) (i0 + s) * M1 + i0 + lane] : 0.0;
            __syncthreads();
            if (tid < 32) {
                double v = lane < w ? x[i0 + lane] : 0.0;
                const double iv = lane < w ? inv[i0 + lane] : 0.0;
                for (int t = 0; t < w; t++) {
                    const int s = pass ? w - 1 - t : t;
                    const double f = __shfl_sync(0xffffffffu, v, s) * __shfl_sync(0xffffffffu, iv, s);
                    if (lane == s)
                        v = f;
                    else if (pass ? lane < s : (lane > s && lane < w))
                        v = fma(-dg[s][lane], f, v);
                }
                y[lane] = v;
                if (lane < w)
                    x[i0 + lane] = v;
            }
            __syncthreads();
            // the entries after (before) the block, up to four of a thread side by side
            // (their chains are independent, and so are their loads)
            const int pa = pass ? 0 : i0 + 32, pe = pass ? i0 : M1;
            const double *M = (pass ? L : LT) + (size_t) i0 * M1;
            for (int pb = pa; pb < pe; pb += 4 * TRI_THREADS) {
                double v[4];
                int p[4];
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    p[r] = min(pb + tid + TRI_THREADS * r, pe - 1);
                    v[r] = x[p[r]];
                }
                const int nr = min(4, (pe - pb + TRI_THREADS - 1) / TRI_THREADS);
                auto steps = [&](auto NR) {
                    constexpr int R = decltype(NR)::value;
#pragma unroll 4
                    for (int t = 0; t < w; t++) {
                        const int s = pass ? w - 1 - t : t;
                        double l[R];
#pragma unroll
                        for (int r = 0; r < R; r++)
                            l[r] = M[(size_t) s * M1 + p[r]];
#pragma unroll
                        for (int r = 0; r < R; r++)
                            v[r] = fma(-l[r], y[s], v[r]);
                    }
                };
                if (nr == 1)
                    steps(std::integral_constant<int, 1>());
                else if (nr == 2)
                    steps(std::integral_constant<int, 2>());
                else if (nr == 3)
                    steps(std::integral_constant<int, 3>());
                else
                    steps(std::integral_constant<int, 4>());
#pragma unroll
                for (int r = 0; r < 4; r++)
                    if (pb + tid + TRI_THREADS * r < pe)
                        x[p[r]] = v[r];
            }
            __syncthreads();
        }
    }
    for (int p = tid; p < M1; p += TRI_THREADS)
        W[(size_t) p * D + c] = x[p];
}

// LT[i][p] = L[p][i], p >= i
__global__ void __launch_bounds__(256) transpose_kernel(const double *__restrict__ L, int M1,
                                                        double *__restrict__ LT)
{
    __shared__ double t[32][33];
    const int p0 = blockIdx.x * 32, i0 = blockIdx.y * 32, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int r = w; r < 32; r += 8)
        t[r][lane] = (p0 + r < M1 && i0 + lane < M1) ? L[(size_t) (p0 + r) * M1 + i0 + lane] : 0.0;
    __syncthreads();
    for (int r = w; r < 32; r += 8)
        if (i0 + r < M1 && p0 + lane < M1)
            LT[(size_t) (i0 + r) * M1 + p0 + lane] = t[lane][r];
}

using TriKernel = void (*)(const double *, const double *, int, int, const int *, double *);

// ceil(M1 / 32) for M1 <= SMEM_SOLVE_MAX
TriKernel tri_solve_for(int nr)
{
    return nr == 1 ? tri_solve_kernel<1> : nr == 2 ? tri_solve_kernel<2>
           : nr == 3 ? tri_solve_kernel<3> : tri_solve_kernel<4>;
}

// Parallel cyclic Jacobi (round-robin pairing) on the symmetric A; the
// eigenvectors go to work[M1 M1 ..) and the inverted eigenvalues (0 where an
// eigenvalue is exactly 0) to work[2 M1 M1 ..); then W = V diag(inv) V^T B.
//
// One CTA, because the M1 - 1 rounds of a sweep depend on each other.  A round's
// rotations act on S as independent 2 x 2 blocks, one per pair of pivot pairs
// (t <= u, mirrored): J_t^T S_tu J_u in one step.  What bounds it is FP64: an SM
// sub-partition issues one FP64 instruction in 64 clocks, so a chain of them in one
// warp costs 64 clocks each.  Therefore:
//   * S and V stay in shared memory (in global memory beyond M1 = SVD_SMEM_MAX);
//   * the angle is taken in FP32 (on the pivot elements' leading bits, scaled by
//     their larger exponent) as tan(theta / 2), and c = 2 r - 1, s = 2 tan r with
//     r = 1 / (1 + tan^2) in FP64, so c^2 + s^2 = 1 to FP64: ten FP64 instructions.
//     A pivot element is left at ~1e-7 of itself instead of at rounding, and the
//     next sweep removes it;
//   * the eigenvectors of a round are rotated by the other warps while the first
//     ones take the next round's angles.
// M1 = 26: 5.73 ms a solve with S and V in global memory and FP64 angles, 0.74 ms
// with the angles' FP64 division and square root and V after S; 0.41 ms this way.
constexpr int SVD_THREADS = 512;
constexpr int SVD_SMEM_MAX = 112;  // 2 M1^2 doubles within 200 KB

__device__ __forceinline__ int jacobi_slot(int x, int n) { return x >= n - 1 ? x - (n - 1) : x; }

// x 2^-(e - 1023) to FP32's leading bits (truncated), for an exponent field of x at most e
__device__ __forceinline__ float leading_bits(double x, int e)
{
    const uint32_t hi = (uint32_t) __double2hiint(x), lo = (uint32_t) __double2loint(x);
    const int fe = (int) ((hi >> 20) & 0x7FF) - e + 127;
    if (fe <= 0)
        return 0.f;
    return __uint_as_float((hi & 0x80000000u) | ((uint32_t) fe << 23) | ((hi & 0xFFFFFu) << 3) | (lo >> 29));
}

template <bool SM>
__global__ void __launch_bounds__(SVD_THREADS) jacobi_kernel(const double *__restrict__ A, int M1,
                                                            double *__restrict__ work, int *flag)
{
    extern __shared__ double sh[];
    double *S = SM ? sh : work;                       // M1 x M1 (becomes diagonal)
    double *V = SM ? sh + (size_t) M1 * M1            // M1 x M1 eigenvectors (columns)
                   : work + (size_t) M1 * M1;
    __shared__ double cs[2][SVD_THREADS], sn[2][SVD_THREADS];  // two rounds' rotations
    __shared__ short2 pq[2][SVD_THREADS];
    __shared__ double red[32];
    const int tid = threadIdx.x;
    const int n = M1 + (M1 & 1);  // even number of slots; slot M1 (if any) is a dummy
    const int h = n / 2, noff = h * (h - 1) / 2, noff32 = (noff + 31) & ~31;
    const int na = (h + 31) & ~31;              // threads that take angles
    const bool overlap = na <= SVD_THREADS / 2;  // the others rotate V meanwhile
    for (int i = tid; i < M1 * M1; i += SVD_THREADS) {
        S[i] = A[i];
        V[i] = ((i / M1) == (i % M1)) ? 1.0 : 0.0;
    }
    // V <- V J of the rotations in buffer b, by threads t0 .. SVD_THREADS
    auto rotate_v = [&](int b, int t0) {
        for (int idx = tid - t0; idx < h * M1; idx += SVD_THREADS - t0) {
            const int t = idx / M1, k = idx - t * M1;
            const int p = pq[b][t].x, q = pq[b][t].y;
            const double c = cs[b][t], s = sn[b][t];
            if (s == 0.0)
                continue;
            const double vp = V[k * M1 + p], vq = V[k * M1 + q];
            V[k * M1 + p] = c * vp - s * vq;
            V[k * M1 + q] = s * vp + c * vq;
        }
    };
    __syncthreads();
    int round = 0;  // rounds so far; their rotations alternate between the buffers
    for (int sweep = 0; sweep < 60; sweep++) {
        double off = 0.0, tot = 0.0;
        for (int i = tid; i < M1 * M1; i += SVD_THREADS) {
            const double v = S[i] * S[i];
            tot += v;
            if ((i / M1) != (i % M1))
                off += v;
        }
        off = block_sum_fixed(off, red);
        tot = block_sum_fixed(tot, red);
        if (off <= 1e-32 * tot)  // the same value in every thread
            break;
        for (int r = 0; r < n - 1; r++, round++) {
            const int b = round & 1;
            // round-robin: slot 0 fixed, the others rotate
            if (tid < h) {
                const int x = (tid == 0) ? 0 : 1 + jacobi_slot(tid - 1 + r, n);
                const int y = 1 + jacobi_slot(n - 2 - tid + r, n);
                const int p = min(x, y), q = max(x, y);
                double c = 1.0, s = 0.0;
                if (q < M1) {
                    const double apq = S[p * M1 + q], d = S[q * M1 + q] - S[p * M1 + p];
                    if (apq != 0.0) {
                        const int e = max((__double2hiint(apq) >> 20) & 0x7FF, (__double2hiint(d) >> 20) & 0x7FF);
                        // fast FP32 forms: the angle only has to be near
                        const float th = fminf(fmaxf(__fdividef(0.5f * leading_bits(d, e), leading_bits(apq, e)),
                                                     -1e18f), 1e18f);
                        const float a2 = fmaf(th, th, 1.0f);
                        const float t = copysignf(__fdividef(1.0f, fabsf(th) + a2 * rsqrtf(a2)), th);
                        const float b2 = fmaf(t, t, 1.0f);
                        const float hf = __fdividef(t, 1.0f + b2 * rsqrtf(b2));  // tan(theta / 2)
                        const double hd = widen(hf), den = fma(hd, hd, 1.0);
                        double ri = widen(__fdividef(1.0f, fmaf(hf, hf, 1.0f)));
                        ri = fma(ri, fma(-den, ri, 1.0), ri);
                        ri = fma(ri, fma(-den, ri, 1.0), ri);
                        c = fma(2.0, ri, -1.0);
                        s = 2.0 * hd * ri;
                    }
                }
                pq[b][tid] = make_short2((short) p, (short) q);
                cs[b][tid] = c;
                sn[b][tid] = s;
            } else if (overlap && tid >= na && round > 0) {
                rotate_v(b ^ 1, na);
            }
            __syncthreads();
            // S <- J^T S J: block (t, u) of the pairs t < u, then (in warps of their own)
            // the pivot blocks t = u
            for (int idx = tid; idx < noff32 + h; idx += SVD_THREADS) {
                int t, u;
                if (idx < noff32) {
                    if (idx >= noff)
                        continue;
                    u = (int) ((sqrtf(8.0f * (float) idx + 1.0f) + 1.0f) * 0.5f);
                    while (u * (u + 1) / 2 <= idx)
                        u++;
                    while (u * (u - 1) / 2 > idx)
                        u--;
                    t = idx - u * (u - 1) / 2;
                } else {
                    t = u = idx - noff32;
                }
                const int p = pq[b][t].x, q = pq[b][t].y;
                const double c1 = cs[b][t], s1 = sn[b][t];
                if (t == u) {
                    if (q >= M1 || s1 == 0.0)
                        continue;
                    const double pp = S[p * M1 + p], qq = S[q * M1 + q], x = S[p * M1 + q];
                    const double cx = c1 * pp - s1 * x, sx = s1 * pp + c1 * x;  // (J^T S) column p
                    const double cy = c1 * x - s1 * qq, sy = s1 * x + c1 * qq;  // column q
                    S[p * M1 + p] = c1 * cx - s1 * cy;
                    S[q * M1 + q] = s1 * sx + c1 * sy;
                    S[p * M1 + q] = S[q * M1 + p] = s1 * cx + c1 * cy;
                    continue;
                }
                const int v = pq[b][u].x, w = pq[b][u].y;
                const double c2 = cs[b][u], s2 = sn[b][u];
                if (s1 == 0.0 && s2 == 0.0)
                    continue;
                const bool hq = q < M1, hw = w < M1;  // p and v are real slots
                const double pv = S[p * M1 + v], pw = hw ? S[p * M1 + w] : 0.0;
                const double qv = hq ? S[q * M1 + v] : 0.0, qw = hq && hw ? S[q * M1 + w] : 0.0;
                const double rpv = c1 * pv - s1 * qv, rpw = c1 * pw - s1 * qw;
                const double rqv = s1 * pv + c1 * qv, rqw = s1 * pw + c1 * qw;
                S[p * M1 + v] = S[v * M1 + p] = c2 * rpv - s2 * rpw;
                if (hw)
                    S[p * M1 + w] = S[w * M1 + p] = s2 * rpv + c2 * rpw;
                if (hq)
                    S[q * M1 + v] = S[v * M1 + q] = c2 * rqv - s2 * rqw;
                if (hq && hw)
                    S[q * M1 + w] = S[w * M1 + q] = s2 * rqv + c2 * rqw;
            }
            if (!overlap)
                rotate_v(b, 0);
            __syncthreads();
        }
    }
    if (overlap && round > 0)
        rotate_v((round - 1) & 1, 0);  // the last round's
    __syncthreads();
    // the inverted eigenvalues after V, which the global variant has in place
    for (int i = tid; i < M1; i += SVD_THREADS) {
        const double lam = S[i * M1 + i];
        work[2 * M1 * M1 + i] = lam != 0.0 ? 1.0 / lam : 0.0;
    }
    if (SM)
        for (int i = tid; i < M1 * M1; i += SVD_THREADS)
            work[M1 * M1 + i] = V[i];
    if (tid == 0)
        flag[0] = 0;
}

// The same decomposition for the FP32 and split forms, whose rounded centres would
// follow a last bit of W that changes (see launch_form_ab's callers): FP64 angles, and
// a row pass and a column pass over the whole of S, element by element as these forms
// have always had them.  S and V in shared memory where they fit.
template <bool SM>
__global__ void __launch_bounds__(SVD_THREADS) jacobi_passes_kernel(const double *__restrict__ A, int M1,
                                                                   double *__restrict__ work, int *flag)
{
    extern __shared__ double sh[];
    double *S = SM ? sh : work;                                  // M1 x M1 (becomes diagonal)
    double *V = (SM ? sh : work) + (size_t) M1 * M1;             // M1 x M1 eigenvectors (columns)
    __shared__ double cs[SVD_THREADS], sn[SVD_THREADS];
    __shared__ int pp[SVD_THREADS], qq[SVD_THREADS];
    __shared__ double red[32];
    __shared__ int done;
    const int n = M1 + (M1 & 1);  // even number of slots; slot M1 (if any) is a dummy
    for (int i = threadIdx.x; i < M1 * M1; i += blockDim.x) {
        S[i] = A[i];
        V[i] = ((i / M1) == (i % M1)) ? 1.0 : 0.0;
    }
    __syncthreads();
    for (int sweep = 0; sweep < 60; sweep++) {
        double off = 0.0, tot = 0.0;
        for (int i = threadIdx.x; i < M1 * M1; i += blockDim.x) {
            const double v = S[i] * S[i];
            tot += v;
            if ((i / M1) != (i % M1))
                off += v;
        }
        off = block_sum_fixed(off, red);
        tot = block_sum_fixed(tot, red);
        if (threadIdx.x == 0)
            done = (off <= 1e-32 * tot);
        __syncthreads();
        if (done)
            break;
        for (int r = 0; r < n - 1; r++) {
            // round-robin: slot 0 fixed, the others rotate
            for (int t = threadIdx.x; t < n / 2; t += blockDim.x) {
                int a = (t == 0) ? 0 : 1 + ((t - 1 + r) % (n - 1));
                int b = 1 + ((n - 2 - t + r) % (n - 1));
                int p = min(a, b), q = max(a, b);
                double c = 1.0, s = 0.0;
                if (q < M1) {
                    const double apq = S[(size_t) p * M1 + q];
                    if (apq != 0.0) {
                        const double app = S[(size_t) p * M1 + p], aqq = S[(size_t) q * M1 + q];
                        const double th = (aqq - app) / (2.0 * apq);
                        const double tt = (th >= 0 ? 1.0 : -1.0) / (fabs(th) + sqrt(th * th + 1.0));
                        c = 1.0 / sqrt(tt * tt + 1.0);
                        s = tt * c;
                    }
                }
                pp[t] = p;
                qq[t] = q;
                cs[t] = c;
                sn[t] = s;
            }
            __syncthreads();
            // rows: S <- J^T S
            for (int idx = threadIdx.x; idx < (n / 2) * M1; idx += blockDim.x) {
                const int t = idx / M1, k = idx % M1;
                const int p = pp[t], q = qq[t];
                if (q >= M1 || sn[t] == 0.0)
                    continue;
                const double c = cs[t], s = sn[t];
                const double sp = S[(size_t) p * M1 + k], sq = S[(size_t) q * M1 + k];
                S[(size_t) p * M1 + k] = c * sp - s * sq;
                S[(size_t) q * M1 + k] = s * sp + c * sq;
            }
            __syncthreads();
            // columns: S <- S J, V <- V J
            for (int idx = threadIdx.x; idx < (n / 2) * M1; idx += blockDim.x) {
                const int t = idx / M1, k = idx % M1;
                const int p = pp[t], q = qq[t];
                if (q >= M1 || sn[t] == 0.0)
                    continue;
                const double c = cs[t], s = sn[t];
                const double sp = S[(size_t) k * M1 + p], sq = S[(size_t) k * M1 + q];
                S[(size_t) k * M1 + p] = c * sp - s * sq;
                S[(size_t) k * M1 + q] = s * sp + c * sq;
                const double vp = V[(size_t) k * M1 + p], vq = V[(size_t) k * M1 + q];
                V[(size_t) k * M1 + p] = c * vp - s * vq;
                V[(size_t) k * M1 + q] = s * vp + c * vq;
            }
            __syncthreads();
        }
    }
    for (int i = threadIdx.x; i < M1; i += blockDim.x) {
        const double lam = S[(size_t) i * M1 + i];
        work[2 * (size_t) M1 * M1 + i] = lam != 0.0 ? 1.0 / lam : 0.0;
    }
    if (SM)
        for (int i = threadIdx.x; i < M1 * M1; i += blockDim.x)
            work[(size_t) M1 * M1 + i] = V[i];
    if (threadIdx.x == 0)
        flag[0] = 0;
}

// W = V diag(inv) V^T B, SVD_COLS columns of B per CTA (the columns are
// independent, so they spread over the SMs)
constexpr int SVD_COLS = 4;

__global__ void __launch_bounds__(128) svd_apply_kernel(const double *__restrict__ V,
                                                        const double *__restrict__ inv,
                                                        const double *__restrict__ B, int M1, int D,
                                                        double *__restrict__ W)
{
    extern __shared__ double sh[];
    double *b = sh, *y = sh + SVD_COLS * M1;  // [M1][SVD_COLS] each
    const int c0 = blockIdx.x * SVD_COLS;
    for (int e = threadIdx.x; e < M1 * SVD_COLS; e += blockDim.x) {
        const int r = e / SVD_COLS, c = c0 + e % SVD_COLS;
        b[e] = c < D ? B[(size_t) r * D + c] : 0.0;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < M1; i += blockDim.x) {
        double acc[SVD_COLS] = {};
        for (int r = 0; r < M1; r++) {
            const double v = V[(size_t) r * M1 + i];
#pragma unroll
            for (int c = 0; c < SVD_COLS; c++)
                acc[c] = fma(v, b[r * SVD_COLS + c], acc[c]);
        }
#pragma unroll
        for (int c = 0; c < SVD_COLS; c++)
            y[i * SVD_COLS + c] = inv[i] * acc[c];
    }
    __syncthreads();
    for (int r = threadIdx.x; r < M1; r += blockDim.x) {
        double acc[SVD_COLS] = {};
        for (int i = 0; i < M1; i++) {
            const double v = V[(size_t) r * M1 + i];
#pragma unroll
            for (int c = 0; c < SVD_COLS; c++)
                acc[c] = fma(v, y[i * SVD_COLS + c], acc[c]);
        }
#pragma unroll
        for (int c = 0; c < SVD_COLS; c++)
            if (c0 + c < D)
                W[(size_t) r * D + c0 + c] = acc[c];
    }
}

int solve_launches(int M1, int solver)
{
    if (solver == DGTM_SOLVE_SVD)
        return 2;
    if (M1 <= SMEM_SOLVE_MAX)
        return 2;
    // np diagonal blocks, np - 1 of the rows below and trailing updates (none after
    // the last), L's transpose, the substitution
    const int np = ceil_div(M1, CHB);
    return np + 2 * (np - 1) + 2;
}

int launch_solve(const double *A, const double *B, int M1, int D, int solver, bool fp64, double *W,
                 double *work, int *flag, cudaStream_t s)
{
    if (solver != DGTM_SOLVE_SVD && M1 > CHOL_MAX_M1) {
        set_error(DGTM_ENOTSUP, "the Cholesky solver supports M1 <= %d", CHOL_MAX_M1);
        return DGTM_ENOTSUP;
    }
    if (solver == DGTM_SOLVE_SVD && M1 > 2 * SVD_THREADS - 2) {
        set_error(DGTM_ENOTSUP, "the eigen-SVD solver supports M1 <= %d", 2 * SVD_THREADS - 2);
        return DGTM_ENOTSUP;
    }
    if (solver == DGTM_SOLVE_SVD) {
        const bool sm = M1 <= SVD_SMEM_MAX;
        const size_t smem = sm ? sizeof(double) * 2 * (size_t) M1 * M1 : 0;
        const auto jacobi = fp64 ? (sm ? jacobi_kernel<true> : jacobi_kernel<false>)
                                 : (sm ? jacobi_passes_kernel<true> : jacobi_passes_kernel<false>);
        DGTM_CUDA_TRY(cudaFuncSetAttribute(jacobi, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem));
        jacobi<<<1, SVD_THREADS, smem, s>>>(A, M1, work, flag);
        DGTM_CUDA_TRY(cudaGetLastError());
        const size_t asmem = sizeof(double) * 2 * SVD_COLS * (size_t) M1;
        DGTM_CUDA_TRY(cudaFuncSetAttribute(svd_apply_kernel,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int) asmem));
        svd_apply_kernel<<<ceil_div(D, SVD_COLS), 128, asmem, s>>>(
            work + (size_t) M1 * M1, work + 2 * (size_t) M1 * M1, B, M1, D, W);
    } else {
        if (M1 <= SMEM_SOLVE_MAX) {
            const size_t smem = sizeof(double) * (3 * (size_t) M1 + (size_t) M1 * M1) +
                                sizeof(uint32_t) * ((size_t) M1 * (M1 - 1) / 2);
            DGTM_CUDA_TRY(cudaFuncSetAttribute(cholesky_small_kernel,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int) smem));
            cholesky_small_kernel<<<1, CHOL_THREADS, smem, s>>>(A, M1, work, flag);
        } else {
            DGTM_CUDA_TRY(cudaMemcpyAsync(work, A, sizeof(double) * (size_t) M1 * M1,
                                          cudaMemcpyDeviceToDevice, s));
            for (int p0 = 0; p0 < M1; p0 += CHB) {
                const int w = M1 - p0 < CHB ? M1 - p0 : CHB;
                chol_diag_kernel<<<1, 32 * CHD_WARPS, 0, s>>>(A, M1, p0, w, work, flag);
                const int nt = ceil_div(M1 - p0 - w, 32);
                if (nt > 0) {
                    chol_rows_kernel<<<nt, 32, 0, s>>>(M1, p0, work);
                    chol_update_kernel<<<nt * (nt + 1) / 2, 256, 0, s>>>(M1, p0, w, work);
                }
            }
        }
        DGTM_CUDA_TRY(cudaGetLastError());
        if (M1 <= SMEM_SOLVE_MAX) {
            const size_t tsmem = sizeof(double) * ((size_t) M1 * M1 + M1);
            const TriKernel tri = tri_solve_for(ceil_div(M1, 32));
            DGTM_CUDA_TRY(cudaFuncSetAttribute(tri, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int) tsmem));
            tri<<<D, TRI_THREADS, tsmem, s>>>(work, B, M1, D, flag, W);
        } else {
            const double *inv = work + (size_t) M1 * M1;
            double *LT = work + (size_t) M1 * M1 + M1;  // within the solver's 2 M1^2 + M1 D
            const int nt = ceil_div(M1, 32);
            transpose_kernel<<<dim3(nt, nt), 256, 0, s>>>(work, M1, LT);
            DGTM_CUDA_TRY(cudaGetLastError());
            tri_solve_large_kernel<<<D, TRI_THREADS, 0, s>>>(work, LT, inv, B, M1, D, flag, W);
        }
    }
    DGTM_CUDA_TRY(cudaGetLastError());
    return DGTM_OK;
}

// ---------------------------------------------------------------------------
// Y = FI W, the per-centre terms of beta and the E-step's copies of Y
// ---------------------------------------------------------------------------
// A warp computes two centres over all depths: lane l owns depths l + 32 c,
// c < NC (passes of 32 NC depths when D > 256).  Per basis function it loads
// the two FI values once (broadcast) and W[m][l + 32 c] from shared memory,
// where W is padded with zeros to whole passes so the loop has no guards.
// Each warp takes the next centre pair from a counter (*ticket, zero at
// launch), so the pairs spread evenly over the SM sub-partitions whatever the
// CTA placement.  The warp sums |y|^2, y.RT and, for the split form,
// |y_hi + y_lo|^2 of each centre by lane partials and shuffles in a fixed
// order (FP64).
//
// Two arithmetics.  DF = false (the FP64 form): 2 NC FP64 accumulators per
// lane; the FP64 pipe (about 2 FMA per clock per SM) bounds the kernel.
// DF = true (the FP32 and split-BF16 forms): FI and W as unevaluated sums of
// two FP32 (hi + lo, 48 bits) and each product accumulated by Dot2 of Ogita,
// Rump and Oishi ("Accurate sum and dot product", SIAM J. Sci. Comput. 26,
// 2005): the high parts' product split exactly by an FMA, the cross terms
// added to its error, the running sum kept exact by Knuth's TwoSum.  The
// result is as accurate as a product in twice FP32's precision (~1e-14
// relative), far inside those forms' 1e-4, on the FP32 pipe, which is 64
// times as wide as the FP64 one.
constexpr int UY_THREADS = 256;
constexpr int UY_NCMAX = 8;
constexpr size_t UY_WSMEM_MAX = 110 * 1024;  // two CTAs per SM

__device__ __forceinline__ double uy_warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// p + s += (a.x + a.y) (w.x + w.y); the _rn intrinsics keep each rounding
// where Dot2 needs it (no contraction into an FMA)
__device__ __forceinline__ void dot2_step(float &p, float &s, float2 a, float2 w)
{
    const float h = __fmul_rn(a.x, w.x);
    float r = fmaf(a.x, w.x, -h);
    r = fmaf(a.x, w.y, r);
    r = fmaf(a.y, w.x, r);
    const float t = __fadd_rn(p, h);
    const float z = __fsub_rn(t, p);
    const float q = __fadd_rn(__fsub_rn(p, __fsub_rn(t, z)), __fsub_rn(h, z));
    p = t;
    s = __fadd_rn(s, __fadd_rn(q, r));
}

__device__ __forceinline__ float2 f64_to_pair(double x)
{
    const float hi = (float) x;
    return make_float2(hi, (float) (x - (double) hi));
}

__global__ void to_pairs_kernel(const double *__restrict__ src, size_t n, float2 *__restrict__ dst)
{
    for (size_t i = blockIdx.x * (size_t) blockDim.x + threadIdx.x; i < n;
         i += (size_t) gridDim.x * blockDim.x)
        dst[i] = f64_to_pair(src[i]);
}

int launch_to_pairs(const double *src, size_t n, float2 *dst, cudaStream_t s)
{
    size_t blocks = (n + 255) / 256;
    if (blocks > 4096)
        blocks = 4096;
    to_pairs_kernel<<<(int) blocks, 256, 0, s>>>(src, n, dst);
    DGTM_CUDA_TRY(cudaGetLastError());
    return DGTM_OK;
}

template <int NC, bool WS, bool DF>
__global__ void __launch_bounds__(UY_THREADS) update_y_kernel(
    const double *__restrict__ FI, const float2 *__restrict__ FIp, const double *__restrict__ Wg,
    const double *__restrict__ G, const double *__restrict__ RT, int K, int M1, int D, int Dw,
    double *__restrict__ Y, double *__restrict__ yy, double *__restrict__ bterm, YCopies cp,
    int *ticket, const float2 *__restrict__ Wq)
{
    // Wq (DF without WS, may be null): W as FP32 pairs in global memory, M1 x Dw
    // M1 x Dw, zero past D: FP64 values, or (hi, lo) pairs of the same size
    extern __shared__ double Ws[];
    float2 *const Wp = reinterpret_cast<float2 *>(Ws);
    if (WS) {
        const int n = M1 * Dw;
#pragma unroll 4
        for (int i = threadIdx.x; i < n; i += UY_THREADS) {
            const int m = i / Dw, d = i - m * Dw;
            const double w = (d < D) ? Wg[(size_t) m * D + d] : 0.0;
            if constexpr (DF)
                Wp[i] = f64_to_pair(w);
            else
                Ws[i] = w;
        }
        __syncthreads();
    }
    __nv_bfloat16 *const hi = reinterpret_cast<__nv_bfloat16 *>(cp.Yb);
    __nv_bfloat16 *const lo = hi ? hi + (size_t) cp.Kpad * cp.Dp : nullptr;
    const int lane = threadIdx.x & 31;
    for (;;) {
        int pair = 0;
        if (lane == 0)
            pair = atomicAdd(ticket, 1);
        const int k0 = 2 * __shfl_sync(0xffffffffu, pair, 0);
        if (k0 >= K)
            break;
        const int nr = (k0 + 1 < K) ? 2 : 1;
        const int k1 = k0 + nr - 1;
        double syy[2] = {0.0, 0.0}, srt[2] = {0.0, 0.0}, sq[2] = {0.0, 0.0};
        for (int db = 0; db < D; db += 32 * NC) {
            double y0[NC], y1[NC];
            if constexpr (DF) {
                float p0[NC], s0[NC], p1[NC], s1[NC];
#pragma unroll
                for (int c = 0; c < NC; c++)
                    p0[c] = s0[c] = p1[c] = s1[c] = 0.f;
                const float2 *f0 = FIp + (size_t) k0 * M1, *f1 = FIp + (size_t) k1 * M1;
                for (int m = 0; m < M1; m++) {
                    const float2 x0 = f0[m], x1 = f1[m];
#pragma unroll
                    for (int c = 0; c < NC; c++) {
                        const int d = db + lane + 32 * c;
                        const float2 w = WS ? Wp[m * Dw + d]
                                         : Wq ? Wq[(size_t) m * Dw + d]
                                              : ((d < D) ? f64_to_pair(Wg[(size_t) m * D + d])
                                                         : make_float2(0.f, 0.f));
                        dot2_step(p0[c], s0[c], x0, w);
                        dot2_step(p1[c], s1[c], x1, w);
                    }
                }
#pragma unroll
                for (int c = 0; c < NC; c++) {
                    y0[c] = (double) p0[c] + (double) s0[c];
                    y1[c] = (double) p1[c] + (double) s1[c];
                }
            } else {
#pragma unroll
                for (int c = 0; c < NC; c++)
                    y0[c] = y1[c] = 0.0;
                const double *f0 = FI + (size_t) k0 * M1, *f1 = FI + (size_t) k1 * M1;
                for (int m = 0; m < M1; m++) {
                    const double x0 = __ldg(f0 + m), x1 = __ldg(f1 + m);
#pragma unroll
                    for (int c = 0; c < NC; c++) {
                        const int d = db + lane + 32 * c;
                        const double w =
                            WS ? Ws[m * Dw + d] : ((d < D) ? __ldg(Wg + (size_t) m * D + d) : 0.0);
                        y0[c] = fma(x0, w, y0[c]);
                        y1[c] = fma(x1, w, y1[c]);
                    }
                }
            }
#pragma unroll
            for (int c = 0; c < NC; c++) {
                const int d = db + lane + 32 * c;
                if (d >= D)
                    continue;
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    if (r >= nr)
                        break;
                    const int k = k0 + r;
                    const double y = r ? y1[c] : y0[c];
                    const size_t e = (size_t) k * D + d;
                    Y[e] = y;
                    syy[r] = fma(y, y, syy[r]);
                    if (RT)
                        srt[r] = fma(y, RT[e], srt[r]);
                    if (cp.Y32)
                        cp.Y32[e] = (float) y;
                    if (hi) {
                        // BF16 hi + lo of y, as the split form's set-up does
                        const __nv_bfloat16 h = __float2bfloat16_rn((float) y);
                        const double hd = (double) __bfloat162float(h);
                        const __nv_bfloat16 l = __float2bfloat16_rn((float) (y - hd));
                        const double yh = hd + (double) __bfloat162float(l);
                        hi[(size_t) k * cp.Dp + d] = h;
                        lo[(size_t) k * cp.Dp + d] = l;
                        sq[r] = fma(yh, yh, sq[r]);
                    }
                }
            }
        }
#pragma unroll
        for (int r = 0; r < 2; r++) {
            if (r >= nr)
                break;
            const int k = k0 + r;
            const double s_yy = uy_warp_sum(syy[r]);
            const double s_rt = RT ? uy_warp_sum(srt[r]) : 0.0;
            const double s_q = hi ? uy_warp_sum(sq[r]) : 0.0;
            if (lane == 0) {
                yy[k] = s_yy;
                if (bterm)
                    bterm[k] = G[k] * s_yy - 2.0 * s_rt;
            }
            if (hi && lane < 3) {
                // -q/2 in three BF16 pieces (24+ significant bits), columns D .. D+2
                const double v = -0.5 * s_q;
                const __nv_bfloat16 p1 = __float2bfloat16_rn((float) v);
                const double r1 = v - (double) __bfloat162float(p1);
                const __nv_bfloat16 p2 = __float2bfloat16_rn((float) r1);
                const double r2 = r1 - (double) __bfloat162float(p2);
                const __nv_bfloat16 p3 = __float2bfloat16_rn((float) r2);
                hi[(size_t) k * cp.Dp + D + lane] = (lane == 0) ? p1 : (lane == 1) ? p2 : p3;
            }
        }
    }
}

using UpdateYKernel = void (*)(const double *, const float2 *, const double *, const double *,
                               const double *, int, int, int, int, double *, double *, double *,
                               YCopies, int *, const float2 *);

// W (M1 x D) as FP32 pairs, M1 x Dw with zero columns past D
__global__ void w_pairs_kernel(const double *__restrict__ W, int M1, int D, int Dw,
                               float2 *__restrict__ Wq)
{
    const size_t n = (size_t) M1 * Dw;
    for (size_t i = blockIdx.x * (size_t) blockDim.x + threadIdx.x; i < n;
         i += (size_t) gridDim.x * blockDim.x) {
        const int m = (int) (i / Dw), d = (int) (i % Dw);
        Wq[i] = d < D ? f64_to_pair(W[(size_t) m * D + d]) : make_float2(0.f, 0.f);
    }
}

template <bool WS, bool DF>
UpdateYKernel update_y_for(int nc)
{
    switch (nc) {
    case 1: return update_y_kernel<1, WS, DF>;
    case 2: return update_y_kernel<2, WS, DF>;
    case 3: return update_y_kernel<3, WS, DF>;
    case 4: return update_y_kernel<4, WS, DF>;
    case 5: return update_y_kernel<5, WS, DF>;
    case 6: return update_y_kernel<6, WS, DF>;
    case 7: return update_y_kernel<7, WS, DF>;
    default: return update_y_kernel<8, WS, DF>;
    }
}

int launch_update_y(const double *FI, const float2 *FIp, const double *W, const double *G,
                    const double *RT, int K, int M1, int D, double *Y, double *yy, double *bterm,
                    const YCopies &cp, int *ticket, double *scratch, size_t scratch_doubles,
                    int *nlaunch, cudaStream_t s)
{
    int dev = 0, sms = 0;
    DGTM_CUDA_TRY(cudaGetDevice(&dev));
    DGTM_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    int nc = ceil_div(D, 32);
    if (nc > UY_NCMAX)
        nc = UY_NCMAX;
    const int Dw = ceil_div(D, 32 * nc) * 32 * nc;
    const size_t wbytes = sizeof(double) * (size_t) M1 * Dw;  // = pairs of FP32
    const bool ws = wbytes <= UY_WSMEM_MAX;
    const bool df = FIp != nullptr;
    int blocks = ceil_div(K, 2 * (UY_THREADS / 32));
    const int cap = sms * (ws ? 2 : 4);
    if (blocks > cap)
        blocks = cap;
    const UpdateYKernel k = ws ? (df ? update_y_for<true, true>(nc) : update_y_for<true, false>(nc))
                               : (df ? update_y_for<false, true>(nc) : update_y_for<false, false>(nc));
    if (ws)
        DGTM_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int) wbytes));
    // W beyond shared memory: converted to pairs once here, not per centre
    float2 *Wq = nullptr;
    int nl = 1;
    if (!ws && df && scratch && (size_t) M1 * Dw <= scratch_doubles) {
        Wq = reinterpret_cast<float2 *>(scratch);
        w_pairs_kernel<<<ceil_div(M1 * Dw, 256), 256, 0, s>>>(W, M1, D, Dw, Wq);
        DGTM_CUDA_TRY(cudaGetLastError());
        nl++;
    }
    k<<<blocks, UY_THREADS, ws ? wbytes : 0, s>>>(FI, FIp, W, G, RT, K, M1, D, Dw, Y, yy, bterm, cp,
                                                 ticket, Wq);
    DGTM_CUDA_TRY(cudaGetLastError());
    if (nlaunch)
        *nlaunch = nl;
    return DGTM_OK;
}

__global__ void norms_kernel(const double *__restrict__ X, int rows, int D,
                             double *__restrict__ out)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int wpb = blockDim.x >> 5;
    for (int r = blockIdx.x * wpb + warp; r < rows; r += gridDim.x * wpb) {
        double s = 0.0;
        for (int d = lane; d < D; d += 32) {
            const double v = X[(size_t) r * D + d];
            s += v * v;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0)
            out[r] = s;
    }
}

int launch_norms(const double *X, int rows, int D, double *out, cudaStream_t s)
{
    int blocks = ceil_div(rows, 8);
    if (blocks > 4864)
        blocks = 4864;
    norms_kernel<<<blocks, 256, 0, s>>>(X, rows, D, out);
    DGTM_CUDA_TRY(cudaGetLastError());
    return DGTM_OK;
}

__global__ void __launch_bounds__(1024) sum_ratio_kernel(const double *__restrict__ v, int n,
                                                        double add, double num, double *out)
{
    __shared__ double red[32];
    double s = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x)  // coalesced, fixed order
        s += v[i];
    s = block_sum_fixed(s, red);
    if (threadIdx.x == 0) {
        const double den = s + add;
        out[0] = den;
        out[1] = num / den;
    }
}

int launch_sum_ratio(const double *v, int n, double add, double num, double *out, cudaStream_t s)
{
    sum_ratio_kernel<<<1, 1024, 0, s>>>(v, n, add, num, out);
    DGTM_CUDA_TRY(cudaGetLastError());
    return DGTM_OK;
}

__global__ void __launch_bounds__(1024) sum_pairs_kernel(const double *__restrict__ part,
                                                        int nb, double *out)
{
    __shared__ double red[32];
    double s0 = 0.0, s1 = 0.0;
    for (int i = threadIdx.x; i < nb; i += blockDim.x) {  // coalesced, fixed order
        s0 += part[2 * i];
        s1 += part[2 * i + 1];
    }
    s0 = block_sum_fixed(s0, red);
    s1 = block_sum_fixed(s1, red);
    if (threadIdx.x == 0) {
        out[0] = s0;
        out[1] = s1;
    }
}

int launch_sum_pairs(const double *part, int nblocks, double *out, cudaStream_t s)
{
    sum_pairs_kernel<<<1, 1024, 0, s>>>(part, nblocks, out);
    DGTM_CUDA_TRY(cudaGetLastError());
    return DGTM_OK;
}

__global__ void to_f32_kernel(const double *__restrict__ src, size_t n, float *__restrict__ dst)
{
    for (size_t i = blockIdx.x * (size_t) blockDim.x + threadIdx.x; i < n;
         i += (size_t) gridDim.x * blockDim.x)
        dst[i] = (float) src[i];
}

int launch_to_f32(const double *src, size_t n, float *dst, cudaStream_t s)
{
    size_t blocks = (n + 255) / 256;
    if (blocks > 8192)
        blocks = 8192;
    if (blocks == 0)
        return DGTM_OK;
    to_f32_kernel<<<(unsigned) blocks, 256, 0, s>>>(src, n, dst);
    DGTM_CUDA_TRY(cudaGetLastError());
    return DGTM_OK;
}

}  // namespace dgtm
