// estep_f32.cu -- the FP32 form's E-step and responsibility pass on the CUDA
// cores, bit for bit the arithmetic of the generic kernels (estep_simt.cu).
//
// The FP32 form rounds its centres to FP32 every M-step, so a last bit that
// changes anywhere in a pass changes later iterations by the form's own 1e-6;
// these kernels therefore keep every rounding and every summation order of the
// generic ones and change only how the work is laid out:
//
//   * the products run from shared memory by 16-byte loads with row strides that
//     are free of bank conflicts (stride / 4 odd), centres or points resident;
//   * GB300's FP64 pipe does two operations a clock and SM, and the generic
//     kernels spend 11 to 14 of them a pair on forming an FP32 argument in FP64.
//     Here the argument comes from error-free FP32 operations: x = d - d_min as
//     an exact pair (Knuth's TwoSum), the product with c as a pair (FMA), about
//     2^-45 relative.  Rounding that to FP32 gives what the FP64 expression
//     gives unless it lies within 2^-42 of a rounding boundary, which is tested;
//     those arguments (one in 2^17) are formed in FP64;
//   * FP32 values become FP64 by integer operations, and sums over lanes are
//     reduced and scattered at once (the same tree, an eighth of the additions).
//
// N = 100,000, K = 8000, D = 166: pass 1 29.9 -> 13.6 ms (16.8 while a chunk of centres
// was loaded between two barriers), pass 2 85.7 -> 20.7 ms.  What bounds pass 1 now is
// issue and latency at two blocks an SM; pass 2 shared memory: 1010 wavefronts a warp
// and tile of 64 points for 2100 FP32 multiply-adds' clocks over four schedulers.
#include "common.cuh"
#include "f32pair.cuh"
#include "kernels.cuh"
#include "sm100.cuh"

#include <math.h>

namespace dgtm {

using namespace sm100;

namespace {

constexpr int FT = 256;   // threads
constexpr int TILE = 64;  // points (and pass 1's centres) of a tile
constexpr int P2C = 32;   // centres of a pass-2 block: four per warp

// Row stride in floats for J = ceil(D / 32): a multiple of 4 with an odd quarter, and
// room for 32 lanes x J, so that every address is a base and a constant.
template <int J>
__host__ __device__ constexpr int row_stride() { return 32 * J + 4; }

}  // namespace

// ---------------------------------------------------------------------------
// Pass 1: column statistics.  Block: 64 points (resident in shared memory), all
// centres in chunks of 64, half their depths at a time through two buffers that
// cp.async fills ahead of the products; thread: 4 points x 4 centres (tx + 16 j, as the generic
// kernel's lanes, whose summation tree this keeps).  Two blocks an SM.
// ---------------------------------------------------------------------------
// a row of half the depths (an even number of quads: see row_stride)
template <int J>
__host__ __device__ constexpr int half_stride() { return 16 * J + 4; }

__device__ __forceinline__ void copy_async(float *dst, const float *src, bool in, bool two)
{
    const uint32_t d = smem_u32(dst);
    if (two)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(in ? 8 : 0) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(in ? 4 : 0) : "memory");
}

template <int J>
__global__ void __launch_bounds__(FT, J <= 6 ? 2 : 1) pass1_f32_kernel(Pass1Args<float> a, Pair c1, Pair c2)
{
    extern __shared__ __align__(16) float sm[];
    constexpr int ld = row_stride<J>();
    const int D = a.D, D4 = (D + 3) / 4 * 4;
    constexpr int lh = half_stride<J>();
    const int hd = (D4 + 7) / 8 * 4;  // depths of the first half
    float *Ts = sm, *Ys = sm + TILE * ld, *yys = Ys + 2 * TILE * lh;  // points, centres, |y|^2
    __shared__ double red[32];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n0 = blockIdx.x * TILE;
    for (int r = warp; r < TILE; r += FT / 32)
        for (int d = lane; d < D4; d += 32)
            Ts[r * ld + d] = (n0 + r < a.N && d < D) ? a.T[(size_t) (n0 + r) * D + d] : 0.f;
    float ttf[4], dmin[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int n = n0 + ty * 4 + i;
        ttf[i] = (float) (n < a.N ? a.tt[n] : 0.0);
        dmin[i] = INFINITY;
    }
    // this lane's share of the sums after the reduction: point oi, temperature ot
    const int oi = ((tx >> 3) & 1) * 2 + ((tx >> 2) & 1), ot = (tx >> 1) & 1;
    const double oc = ot ? a.c2 : a.c1;
    double s = 0.0;

    // 8-byte copies where every row starts on 8 bytes: an even D, and a pointer that does
    // (Y may be a caller's array, which is only known to start on 4)
    const bool two = (D & 1) == 0 && ((uintptr_t) a.Y & 7) == 0;
    // depths d0 .. d1 - 1 of the centres k .. k + 63 into half buffer b; zeros outside
    auto fill = [&](int k, int b) {
        const int d0 = b * hd, n = b ? D4 - hd : hd;
        float *dst = Ys + b * TILE * lh;
        const int step = two ? 2 : 1;
        for (int r = warp; r < TILE; r += FT / 32) {
            const float *src = a.Y + (size_t) min(k + r, a.K - 1) * D;
            for (int d = step * lane; d < n; d += 32 * step) {
                const bool in = k + r < a.K && d0 + d < D;
                copy_async(dst + r * lh + d, in ? src + d0 + d : a.Y, in, two);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fill(0, 0);

    for (int k0 = 0; k0 < a.K; k0 += TILE) {
        float acc[4][4];
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++)
                acc[i][j] = 0.f;
#pragma unroll 1
        for (int b = 0; b < 2; b++) {
            // this half has arrived for every thread, and the other buffer's readers are done
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncthreads();
            if (b == 0)
                fill(k0, 1);
            else if (k0 + TILE < a.K)
                fill(k0 + TILE, 0);
            float yy = 0.f;
            if (b == 0 && threadIdx.x < TILE)
                yy = (float) (k0 + (int) threadIdx.x < a.K ? a.yy[k0 + threadIdx.x] : 0.0);
            const float *tp = Ts + b * hd, *yp = Ys + b * TILE * lh;
            const int n = b ? D4 - hd : hd;
            // columns D .. D4 are zero in both operands: adding 0 x 0 keeps every bit
            // (a sum that is -0 cannot arise from products added to +0)
#pragma unroll 2
            for (int d = 0; d < n; d += 4) {
                float4 t[4], y[4];
#pragma unroll
                for (int i = 0; i < 4; i++)
                    t[i] = *(const float4 *) &tp[(ty * 4 + i) * ld + d];
#pragma unroll
                for (int j = 0; j < 4; j++)
                    y[j] = *(const float4 *) &yp[(tx + 16 * j) * lh + d];
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        acc[i][j] = __fmaf_rn(t[i].x, y[j].x, acc[i][j]);
                        acc[i][j] = __fmaf_rn(t[i].y, y[j].y, acc[i][j]);
                        acc[i][j] = __fmaf_rn(t[i].z, y[j].z, acc[i][j]);
                        acc[i][j] = __fmaf_rn(t[i].w, y[j].w, acc[i][j]);
                    }
            }
            // read after the second half's barrier; the last chunk's readers passed the first's
            if (b == 0 && threadIdx.x < TILE)
                yys[threadIdx.x] = yy;
        }
        float yf[4];
#pragma unroll
        for (int j = 0; j < 4; j++)
            yf[j] = yys[tx + 16 * j];
        double v[8];  // the point sums of this lane, points x temperatures
        float nmo = 0.f, dmo = 0.f;  // new and old minimum of this lane's point oi
#pragma unroll
        for (int i = 0; i < 4; i++) {
            float dd[4], lm = INFINITY;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                dd[j] = __fadd_rn(__fmaf_rn(-2.f, acc[i][j], yf[j]), ttf[i]);
                if (k0 + tx + 16 * j < a.K)
                    lm = fminf(lm, dd[j]);
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1)
                lm = fminf(lm, __shfl_xor_sync(0xffffffffu, lm, o));
            const float nm = fminf(dmin[i], lm);
            float p1[4], p2[4];
            unsigned bad = 0;  // bit j: p1[j], 4 + j: p2[j] not settled
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const bool in = k0 + tx + 16 * j < a.K;
                float xh, xl;
                two_sum(in ? dd[j] : nm, -nm, xh, xl);
                bool ok = true;
                p1[j] = pass1_argument(c1, xh, xl, ok);
                bad |= ok ? 0u : 1u << j;
                if (a.isDA) {
                    ok = true;
                    p2[j] = pass1_argument(c2, xh, xl, ok);
                    bad |= ok ? 0u : 16u << j;
                }
            }
            if (bad) {
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    float xh, xl;
                    two_sum(dd[j], -nm, xh, xl);
                    if (((bad >> j) & 1) && !exact_product(c1, xh, xl)) {
                        // a volatile statement: the FP64 instructions stay behind the branch
                        asm volatile("");
                        p1[j] = (float) (-a.c1 * ((double) dd[j] - (double) nm));
                    }
                    if (((bad >> (4 + j)) & 1) && !exact_product(c2, xh, xl)) {
                        asm volatile("");
                        p2[j] = (float) (-a.c2 * ((double) dd[j] - (double) nm));
                    }
                }
            }
            double e1 = 0.0, e2 = 0.0;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const bool in = k0 + tx + 16 * j < a.K;
                const float f1 = in ? expf(p1[j]) : 0.f;
                e1 = j ? e1 + widen(f1) : widen(f1);
                if (a.isDA) {
                    const float f2 = in ? expf(p2[j]) : 0.f;
                    e2 = j ? e2 + widen(f2) : widen(f2);
                }
            }
            v[2 * i] = e1;
            v[2 * i + 1] = e2;
            if (i == oi) {
                nmo = nm;
                dmo = dmin[i];
            }
            dmin[i] = nm;
        }
        // the butterfly over 16 lanes, halving what a lane still needs at each step
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const bool up = tx & 8;
            const double mine = up ? v[4 + q] : v[q], send = up ? v[q] : v[4 + q];
            v[q] = mine + __shfl_xor_sync(0xffffffffu, send, 8);
        }
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const bool up = tx & 4;
            const double mine = up ? v[2 + q] : v[q], send = up ? v[q] : v[2 + q];
            v[q] = mine + __shfl_xor_sync(0xffffffffu, send, 4);
        }
        {
            const bool up = tx & 2;
            const double mine = up ? v[1] : v[0], send = up ? v[0] : v[1];
            v[0] = mine + __shfl_xor_sync(0xffffffffu, send, 2);
        }
        v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
        if (nmo < dmo) {
            const double x = (double) dmo - (double) nmo;  // >= 0 (inf on the first chunk)
            s = (s == 0.0) ? 0.0 : s * exp(-oc * x);
        }
        s += v[0];
    }

    // point oi's two sums to one lane (tx & 3 == 0), then as the generic kernel
    const double s2 = __shfl_xor_sync(0xffffffffu, s, 2);
    double l1 = 0.0, l2 = 0.0;
    const int gn = n0 + ty * 4 + oi;
    if ((tx & 3) == 0 && gn < a.N) {
        const float dm = oi == 0 ? dmin[0] : oi == 1 ? dmin[1] : oi == 2 ? dmin[2] : dmin[3];
        const double dmn = (double) dm;
        const double lse1 = -a.c1 * dmn + log(s);
        const double ss = a.isDA ? s2 : s;
        double lsn = log(ss);
        l1 = lse1;
        l2 = a.isDA ? (-a.c2 * dmn + log(s2)) : 0.0;
        // comm/mpicomm.c:382-389: a column whose every exp(-beta d/2)
        // underflows is replaced by R = 1/K with v = K
        if (exp(-a.c1 * dmn) == 0.0) {
            lsn = NAN;
            if (a.isDA) {
                l1 = -INFINITY;          // log(vgc) = log 0
                l2 = log((double) a.K);  // log(vgc2) = log K
            } else {
                l1 = log((double) a.K);
            }
        }
        a.colstat[gn] = make_double2(dmn, lsn);
    }
    l1 = block_sum_fixed(l1, red);
    l2 = block_sum_fixed(l2, red);
    if (threadIdx.x == 0) {
        a.part[2 * blockIdx.x + 0] = l1;
        a.part[2 * blockIdx.x + 1] = l2;
    }
}

// ---------------------------------------------------------------------------
// Pass 2: G and R T of one slice of the points.  Block: 32 centres (resident), a
// warp owns four of them from distance to R T: it forms R of its centres for the 64
// points of a tile (two points a lane), leaves it in its own shared rows and
// multiplies by the tile (J = ceil(D / 64) pairs of depths a lane, packed FP32
// multiply-adds; R is stored twice over so that it comes out as a pair).  So only the
// tile loads synchronise the block.  The FP32 sums over a tile of 64 points go into FP64 sums.
// ---------------------------------------------------------------------------
template <int J>
__global__ void __launch_bounds__(FT, J <= 3 ? 2 : 1) pass2_f32_kernel(Pass2Args<float> a, Pair c, float cut)
{
    extern __shared__ __align__(16) float sm[];
    constexpr int RS = 2 * P2C + 4, ld = row_stride<2 * J>();
    const int D = a.D, D4 = (D + 3) / 4 * 4;
    float *Ts = sm, *Ys = Ts + TILE * ld, *Rs = Ys + P2C * ld;  // [64][ld], [32][ld], [64][RS]
    float4 *pc = (float4 *) (Rs + TILE * RS);  // per point: d_min, ln s as a pair, |t|^2
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int k0 = blockIdx.x * P2C, kw = k0 + 4 * warp;
    const int split_i = blockIdx.y;
    const int nb = split_i * a.n_per_split, ne = min(a.N, nb + a.n_per_split);
    for (int r = warp; r < P2C; r += FT / 32)
        for (int d = lane; d < D4; d += 32)
            Ys[r * ld + d] = (k0 + r < a.K && d < D) ? a.Y[(size_t) (k0 + r) * D + d] : 0.f;
    float yf[4];
#pragma unroll
    for (int i = 0; i < 4; i++)
        yf[i] = (float) (kw + i < a.K ? a.yy[kw + i] : 0.0);
    const float invK = (float) (1.0 / (double) a.K);
    const bool two = (D & 1) == 0 && ((uintptr_t) a.T & 7) == 0;  // every row starts on 8 bytes
    // G of two centres (lanes 0-15: kw, kw + 1; 16-31: kw + 2, kw + 3) over the
    // points lane % 16 + 16 j, j = 0 .. 3, in this order
    double g[2] = {0.0, 0.0};
    double rt[4][2 * J];  // depths 2 lane + 64 j, + 1
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 2 * J; j++)
            rt[i][j] = 0.0;

    for (int n0 = nb; n0 < ne; n0 += TILE) {
        __syncthreads();
        if (two) {
#pragma unroll 4
            for (int r = warp; r < TILE; r += FT / 32)
#pragma unroll
                for (int j = 0; j < J; j++) {
                    const int d = 2 * lane + 64 * j;
                    float2 v = make_float2(0.f, 0.f);
                    if (n0 + r < ne && d < D)
                        v = *(const float2 *) &a.T[(size_t) (n0 + r) * D + d];
                    *(float2 *) &Ts[r * ld + d] = v;
                }
        } else {
#pragma unroll 2
            for (int r = warp; r < TILE; r += FT / 32)
#pragma unroll
                for (int j = 0; j < 2 * J; j++) {
                    const int d = lane + 32 * j;
                    Ts[r * ld + d] = (n0 + r < ne && d < D) ? a.T[(size_t) (n0 + r) * D + d] : 0.f;
                }
        }
        if (threadIdx.x < TILE) {
            const int n = n0 + threadIdx.x;
            const double2 cs = n < ne ? a.colstat[n] : make_double2(0.0, 0.0);
            const Pair l = split(cs.y);
            pc[threadIdx.x] = make_float4((float) cs.x, l.h, l.l, (float) (n < ne ? a.tt[n] : 0.0));
        }
        __syncthreads();
        float acc[4][2];
#pragma unroll
        for (int i = 0; i < 4; i++)
            acc[i][0] = acc[i][1] = 0.f;
#pragma unroll 2
        for (int d = 0; d < D4; d += 4) {
            const float4 t0 = *(const float4 *) &Ts[lane * ld + d], t1 = *(const float4 *) &Ts[(lane + 32) * ld + d];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float4 y = *(const float4 *) &Ys[(4 * warp + i) * ld + d];
                acc[i][0] = __fmaf_rn(y.x, t0.x, acc[i][0]);
                acc[i][0] = __fmaf_rn(y.y, t0.y, acc[i][0]);
                acc[i][0] = __fmaf_rn(y.z, t0.z, acc[i][0]);
                acc[i][0] = __fmaf_rn(y.w, t0.w, acc[i][0]);
                acc[i][1] = __fmaf_rn(y.x, t1.x, acc[i][1]);
                acc[i][1] = __fmaf_rn(y.y, t1.y, acc[i][1]);
                acc[i][1] = __fmaf_rn(y.z, t1.z, acc[i][1]);
                acc[i][1] = __fmaf_rn(y.w, t1.w, acc[i][1]);
            }
        }
        // (float) (-c (d - d_min) - ln s) of the eight pairs
        float r[4][2], dd[4][2];
        bool ok = true;
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const float4 p = pc[lane + 32 * e];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                dd[i][e] = __fadd_rn(__fmaf_rn(-2.f, acc[i][e], yf[i]), p.w);
                r[i][e] = pass2_argument(c, dd[i][e], p.x, p.y, p.z, ok);
            }
        }
        if (!ok) {
            asm volatile("");  // the FP64 instructions stay behind the branch
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int n = n0 + lane + 32 * e;
                const double2 cs = n < ne ? a.colstat[n] : make_double2(0.0, 0.0);
#pragma unroll
                for (int i = 0; i < 4; i++)
                    r[i][e] = (float) fma(-a.c, (double) dd[i][e] - cs.x, -cs.y);
            }
        }
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const int nl = lane + 32 * e;
            const bool zero_column = isnan(pc[nl].y);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                float w = dd[i][e] > cut ? 0.f : expf(r[i][e]);
                w = zero_column ? invK : w;
                r[i][e] = n0 + nl < ne && kw + i < a.K ? w : 0.f;
            }
            *(float4 *) &Rs[nl * RS + 8 * warp] = make_float4(r[0][e], r[0][e], r[1][e], r[1][e]);
            *(float4 *) &Rs[nl * RS + 8 * warp + 4] = make_float4(r[2][e], r[2][e], r[3][e], r[3][e]);
        }
        {
            const bool up = lane & 16;
#pragma unroll
            for (int i = 0; i < 2; i++) {
                // own points n, n + 32; the partner's are n +- 16, +- 16 + 32
                const float p0 = __shfl_xor_sync(0xffffffffu, up ? r[i][0] : r[2 + i][0], 16);
                const float p1 = __shfl_xor_sync(0xffffffffu, up ? r[i][1] : r[2 + i][1], 16);
                const float m0 = up ? r[2 + i][0] : r[i][0], m1 = up ? r[2 + i][1] : r[i][1];
                g[i] += widen(up ? p0 : m0);
                g[i] += widen(up ? m0 : p0);
                g[i] += widen(up ? p1 : m1);
                g[i] += widen(up ? m1 : p1);
            }
        }
        __syncwarp();
        f2 loc[4][J];
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < J; j++)
                loc[i][j].v = 0ull;
#pragma unroll 4
        for (int n = 0; n < TILE; n++) {
            const ulonglong2 ra = *(const ulonglong2 *) &Rs[n * RS + 8 * warp];
            const ulonglong2 rb = *(const ulonglong2 *) &Rs[n * RS + 8 * warp + 4];
            const f2 rv[4] = {{ra.x}, {ra.y}, {rb.x}, {rb.y}};
#pragma unroll
            for (int j = 0; j < J; j++) {
                const f2 tv = {*(const uint64_t *) &Ts[n * ld + 2 * lane + 64 * j]};
#pragma unroll
                for (int i = 0; i < 4; i++)
                    loc[i][j] = f2_fma(rv[i], tv, loc[i][j]);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < J; j++) {
                rt[i][2 * j] += widen(f2_lo(loc[i][j]));
                rt[i][2 * j + 1] += widen(f2_hi(loc[i][j]));
            }
    }

    // the 16 point lanes of a centre, as the generic kernel's tree
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int o = 8; o > 0; o >>= 1)
            g[i] += __shfl_xor_sync(0xffffffffu, g[i], o);
    double *Gp = a.Gpart + (size_t) split_i * a.K;
    double *RTp = a.RTpart + (size_t) split_i * a.K * D;
    if ((lane & 15) == 0)
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int k = kw + (lane ? 2 : 0) + i;
            if (k < a.K)
                Gp[k] = g[i];
        }
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 2 * J; j++) {
            const int d = 2 * lane + 64 * (j >> 1) + (j & 1);
            if (kw + i < a.K && d < D)
                RTp[(size_t) (kw + i) * D + d] = rt[i][j];
        }
}

namespace {

using P1Kernel = void (*)(Pass1Args<float>, Pair, Pair);
using P2Kernel = void (*)(Pass2Args<float>, Pair, float);

struct Kernels {
    P1Kernel p1;
    P2Kernel p2;
    int ld1, ld2;
};

template <int J>
constexpr Kernels kernels_of()
{
    constexpr int J2 = (J + 1) / 2;
    return Kernels{pass1_f32_kernel<J>, pass2_f32_kernel<J2>, row_stride<J>() + 2 * half_stride<J>(), row_stride<2 * J2>()};
}

const Kernels KERNELS[8] = {kernels_of<1>(), kernels_of<2>(), kernels_of<3>(), kernels_of<4>(),
                            kernels_of<5>(), kernels_of<6>(), kernels_of<7>(), kernels_of<8>()};

int depth_class(int D, const Kernels **k)
{
    if (D < 1 || D > 256) {
        set_error(DGTM_ENOTSUP, "D = %d exceeds the CUDA-core form's limit of 256", D);
        return DGTM_ENOTSUP;
    }
    *k = &KERNELS[ceil_div(D, 32) - 1];
    return DGTM_OK;
}

}  // namespace

int launch_pass1_f32(const Pass1Args<float> &a, cudaStream_t s)
{
    const Kernels *k = nullptr;
    const int rc = depth_class(a.D, &k);
    if (rc != DGTM_OK)
        return rc;
    const size_t smem = sizeof(float) * ((size_t) TILE * k->ld1 + TILE);
    DGTM_CUDA_TRY(cudaFuncSetAttribute(k->p1, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem));
    k->p1<<<ceil_div(a.N, TILE), FT, smem, s>>>(a, split(a.c1), split(a.c2));
    DGTM_CUDA_TRY(cudaGetLastError());
    return DGTM_OK;
}

// Device code is loaded kernel by kernel on first use: this loads pass 1 of every D.
int load_pass1_f32()
{
    for (const Kernels &k : KERNELS) {
        cudaFuncAttributes attr;
        DGTM_CUDA_TRY(cudaFuncGetAttributes(&attr, (const void *) k.p1));
        const size_t smem = sizeof(float) * ((size_t) TILE * k.ld1 + TILE);
        DGTM_CUDA_TRY(cudaFuncSetAttribute(k.p1, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem));
    }
    return DGTM_OK;
}

int launch_pass2_f32(const Pass2Args<float> &a, int nsplit, cudaStream_t s)
{
    const Kernels *k = nullptr;
    const int rc = depth_class(a.D, &k);
    if (rc != DGTM_OK)
        return rc;
    const size_t smem = sizeof(float) * ((size_t) (TILE + P2C) * k->ld2 + TILE * (2 * P2C + 4)) + sizeof(float4) * TILE;
    // d > dcut for an FP32 d: d above the largest FP32 value not above dcut
    float cut = (float) a.dcut;
    if ((double) cut > a.dcut)
        cut = nextafterf(cut, -INFINITY);
    DGTM_CUDA_TRY(cudaFuncSetAttribute(k->p2, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem));
    k->p2<<<dim3(ceil_div(a.K, P2C), nsplit), FT, smem, s>>>(a, split(a.c), cut);
    DGTM_CUDA_TRY(cudaGetLastError());
    return DGTM_OK;
}

}  // namespace dgtm
