// oz.cu -- FP64-accurate matrix products on the tensor cores (tcgen05 + TMA +
// TMEM, sm_103a) by exact digit slices.
//
// GB300's FP64 pipe does 2 FMA per clock per SM (0.63 TFMA/s measured on the
// whole GPU), its BF16 tensor pipe 4096.  Each FP64 operand value is therefore
// written as a 56-bit integer on its row's (or the matrix's) power-of-two grid
// and cut into eight balanced base-128 digits, |d| <= 64, exact in BF16 (the
// error-free splitting of Ozaki, Ogita, Oishi and Rump, "Error-free
// transformations of matrix multiplication by using fast routines of matrix
// multiplication and its applications", Numer. Algorithms 59, 2012).  Products
// of digits i and j carry the weight of level l = i + j, so one FP32
// accumulator per level holds them all:
//     C = sum_l 128^(14 - l) S_l,  S_l = sum_{i + j = l} sum_k a_i[k] b_j[k],
// |S_l| <= (l + 1) 512 4096 <= 2^24 over 512 elements of k: an exact FP32
// integer whatever the order.  Levels 0 .. 7 are kept (36 of the 64 digit
// products); what is dropped is below 2^-58 of the operands' largest products
// per term, under the rounding of an FP64 multiply-add chain.  The levels are
// combined in 96-bit integers every 512 elements; FP64 comes back only once per
// item of a sum.
//
// oz_gemm_kernel: persistent, one CTA per SM (TMEM: 8 levels x 64 columns = all
// 512).  Tile 128 (A rows, TMEM lanes) x 64 (B rows).  Per 64-deep panel the
// eight B planes (64 KB, double-buffered) stay while the A planes stream
// through a ring of 16 KB slots; A plane i multiplies B planes 0 .. 7 - i in one
// or two instructions, because consecutive planes of B are consecutive rows in
// shared memory and their levels i .. 7 consecutive column blocks in TMEM
// (N up to 256: the tensor pipe's full rate, where an N = 64 instruction per
// digit pair is bound by shared-memory reads).  Per panel 36 x 128 clocks of
// MMA against 192 KB of loads.
#include "common.cuh"
#include "kernels.cuh"
#include "oz.cuh"
#include "oz_slice.cuh"
#include "sm100.cuh"

#include <math.h>
#include <new>
#include <vector>

namespace dgtm {

int make_tmap_bf16(CUtensorMap *map, const void *ptr, uint64_t rows, uint64_t cols, uint64_t ld,
                   uint32_t box_rows, uint32_t box_cols);

using namespace sm100;

namespace {

constexpr int DRAIN_WARPS = 16;
constexpr int OZ_THREADS = 64 + 32 * DRAIN_WARPS;  // warp 0 TMA, warp 1 MMA, then the drain
constexpr int TM = 128, TN = 64; // tile
constexpr int PANEL = 64;
constexpr int SB = oz::DIGITS;   // planes of B, levels
constexpr int A_SLOT = TM * 128;           // one A plane of one panel: 16 KB
constexpr int B_PLANE = TN * 128;          // 8 KB
constexpr int B_BUF = SB * B_PLANE;        // 64 KB
constexpr int A_SLOTS = 5;
constexpr int SEG = 8;                     // panels per exact segment (512 elements)
constexpr int COLS = TN / (DRAIN_WARPS / 4);  // columns of a drain warp
constexpr size_t OZ_SMEM = 1024 + 2 * (size_t) B_BUF + A_SLOTS * (size_t) A_SLOT + 256 + DRAIN_WARPS * COLS * 16;

struct OzParams {
    int panels, b_panel0, a_rows, b_rows, a_tile0, b_row0, mtiles, ntiles, nitems, splits, item_panels;
    const int *tiles;
    double *sums;
    int64_t *out;
    size_t ldm;
    int mrows, ncols;
    const OzUnit *units;
    const oz::Centre *cen;
    const int *skip;
    int *status;
};

__device__ __forceinline__ void oz_item(const OzParams &p, int it, int &mt, int &nt, int &p0, int &p1)
{
    const int t = it / p.splits, sp = it - t * p.splits;
    if (p.tiles) {
        const int v = p.tiles[t];
        mt = v >> 16;
        nt = v & 0xFFFF;
    } else {
        mt = t / p.ntiles;
        nt = t - mt * p.ntiles;
    }
    p0 = sp * p.item_panels;
    p1 = min(p.panels, p0 + p.item_panels);
}

// One element's levels v[0], v[4], .., v[28] as hi 2^28 + lo; the four pairs of
// levels are exact in 32 bits.  NARROW: every |S_l| is at most 2^22, so
// 1.5 2^23 + S_l has the integer in its low bits; a conversion instruction runs
// at an eighth of the adder's rate.
template <bool NARROW>
__device__ __forceinline__ void level_pairs(const uint32_t *v, int64_t &hi, int64_t &lo)
{
    int q[4];
#pragma unroll
    for (int h = 0; h < 4; h++) {
        const float a = __uint_as_float(v[8 * h]), b = __uint_as_float(v[8 * h + 4]);
        if (NARROW) {
            const uint32_t x = __float_as_uint(__fadd_rn(a, 12582912.f));
            const uint32_t y = __float_as_uint(__fadd_rn(b, 12582912.f));
            q[h] = (int) (x * 128u + (y - 0x4B400000u * 129u));
        } else {
            q[h] = __float2int_rz(a) * 128 + __float2int_rz(b);
        }
    }
    hi = (int64_t) q[0] * 16384 + q[1];
    lo = (int64_t) q[2] * 16384 + q[3];
}

template <int SA, bool SUM, bool NARROW>
__global__ void __launch_bounds__(OZ_THREADS, 1) oz_gemm_kernel(const __grid_constant__ CUtensorMap tmA,
                                                               const __grid_constant__ CUtensorMap tmB,
                                                               const OzParams p)
{
    if (p.skip && *p.skip)
        return;
    extern __shared__ unsigned char smem_raw[];
    unsigned char *sm = (unsigned char *) (((uintptr_t) smem_raw + 1023) & ~(uintptr_t) 1023);
    unsigned char *Bst = sm, *Ast = sm + 2 * B_BUF;
    uint64_t *bars = (uint64_t *) (Ast + A_SLOTS * A_SLOT);
    uint64_t *a_full = bars, *a_empty = bars + A_SLOTS;
    uint64_t *b_full = bars + 2 * A_SLOTS, *b_empty = b_full + 2;
    uint64_t *acc_full = b_full + 4, *acc_empty = acc_full + 1, *drain = acc_full + 2;
    uint32_t *tmem_sh = (uint32_t *) (drain + 1);
    int4 *cols_sh = (int4 *) ((unsigned char *) bars + 256);  // COLS centres of each drain warp
    __shared__ int failed;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        failed = 0;
        for (int i = 0; i < A_SLOTS; i++) {
            mbar_init(&a_full[i], 1);
            mbar_init(&a_empty[i], 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(&b_full[i], 1);
            mbar_init(&b_empty[i], 1);
        }
        mbar_init(acc_full, 1);
        mbar_init(acc_empty, 32 * DRAIN_WARPS);
        mbar_init(drain, 1);
        fence_barrier_init();
    }
    if (warp == 0) {
        tmem_alloc(tmem_sh, 512);
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_sh, 0);

    if (warp == 0 && lane == 0) {
        // ---------------- producer ----------------
        prefetch_tmap(&tmA);
        prefetch_tmap(&tmB);
        int as = 0, na = 0, nb = 0;
        uint32_t aph = 0;
        bool ok = true;
        for (int it = blockIdx.x; ok && it < p.nitems; it += gridDim.x) {
            int mt, nt, p0, p1;
            oz_item(p, it, mt, nt, p0, p1);
            for (int pn = p0; ok && pn < p1; pn++, nb++) {
                const int b = nb & 1;
                if (nb >= 2 && !mbar_wait(&b_empty[b], (uint32_t) (((nb >> 1) & 1) ^ 1), p.status, 71)) {
                    ok = false;
                    break;
                }
                mbar_expect_tx(&b_full[b], (uint32_t) B_BUF);
#pragma unroll
                for (int j = 0; j < SB; j++)
                    tma_load_2d(Bst + b * B_BUF + j * B_PLANE, &tmB, &b_full[b], PANEL * (pn + p.b_panel0),
                                j * p.b_rows + p.b_row0 + nt * TN);
                for (int i = 0; i < SA; i++, na++) {
                    if (na >= A_SLOTS && !mbar_wait(&a_empty[as], aph ^ 1u, p.status, 72)) {
                        ok = false;
                        break;
                    }
                    mbar_expect_tx(&a_full[as], (uint32_t) A_SLOT);
                    tma_load_2d(Ast + as * A_SLOT, &tmA, &a_full[as], PANEL * pn,
                                i * p.a_rows + (p.a_tile0 + mt) * TM);
                    if (++as == A_SLOTS) {
                        as = 0;
                        aph ^= 1u;
                    }
                }
            }
        }
        if (!ok)
            failed = 1;
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        const uint64_t adesc0 = sdesc_sw128(smem_u32(Ast), 16, 1024);
        const uint64_t bdesc0 = sdesc_sw128(smem_u32(Bst), 16, 1024);
        int as = 0, nb = 0, nseg = 0;
        uint32_t aph = 0;
        bool ok = true;
        for (int it = blockIdx.x; ok && it < p.nitems; it += gridDim.x) {
            int mt, nt, p0, p1;
            oz_item(p, it, mt, nt, p0, p1);
            for (int pn = p0; ok && pn < p1; pn++, nb++) {
                const int in_seg = (pn - p0) % SEG;
                if (in_seg == 0 && nseg > 0 &&
                    !mbar_wait_w(acc_empty, (uint32_t) ((nseg - 1) & 1), p.status, 73)) {
                    ok = false;
                    break;
                }
                const int b = nb & 1;
                if (!mbar_wait_w(&b_full[b], (uint32_t) ((nb >> 1) & 1), p.status, 74)) {
                    ok = false;
                    break;
                }
                const uint64_t bd = bdesc0 + (uint64_t) ((b * B_BUF) >> 4);
#pragma unroll
                for (int i = 0; i < SA; i++) {
                    if (!mbar_wait_w(&a_full[as], aph, p.status, 75)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint64_t ad = adesc0 + (uint64_t) ((as * A_SLOT) >> 4);
#pragma unroll
                    for (int ks = 0; ks < 4; ks++) {
                        const int first = SB - i < 4 ? SB - i : 4;  // B planes of the first instruction
                        mma_ss_w(tmem + (uint32_t) (i * TN), ad + 2 * ks, bd + 2 * ks,
                                 idesc_bf16(TM, TN * first, 0, 0),
                                 (in_seg || i || ks) ? 1u : 0u);
                        if (SB - i > 4)
                            mma_ss_w(tmem + (uint32_t) ((i + 4) * TN), ad + 2 * ks,
                                     bd + (uint64_t) ((4 * B_PLANE) >> 4) + 2 * ks,
                                     idesc_bf16(TM, TN * (SB - i - 4), 0, 0),
                                     (in_seg || i || ks) ? 1u : 0u);
                    }
                    mma_commit_w(&a_empty[as]);
                    if (++as == A_SLOTS) {
                        as = 0;
                        aph ^= 1u;
                    }
                }
                if (!ok)
                    break;
                mma_commit_w(&b_empty[b]);
                if (in_seg == SEG - 1 || pn == p1 - 1) {
                    mma_commit_w(acc_full);
                    nseg++;
                }
            }
        }
        if (!ok)
            failed = 1;
    } else if (warp >= 2) {
        // ---------------- drain: levels to 64-bit integers ----------------
        const int q = warp & 3, h = (warp - 2) >> 2;  // lane quarter, 16 of the columns
        const uint32_t lane_base = tmem + ((uint32_t) (q * 32) << 16) + (uint32_t) (16 * h);
        const int row = q * 32 + lane;
        int nseg = 0;
        bool ok = true;
        for (int it = blockIdx.x; ok && it < p.nitems; it += gridDim.x) {
            int mt, nt, p0, p1;
            oz_item(p, it, mt, nt, p0, p1);
            // sums over all segments of an item: exact, in 96 bits (rounded once at its end;
            // a unit that a whole contraction of full terms fits is too coarse for a centre
            // whose R lies on few points: 2^-49 of the grids at 5000 points put critical
            // temperatures 1e-12 off)
            oz::Sum96 acc[SUM ? 16 : 1];
            if constexpr (SUM) {
#pragma unroll
                for (int c = 0; c < 16; c++)
                    acc[c] = oz::Sum96{0, 0, 0};
            }
            // Distances: this warp's centres by way of shared memory, |y|^2 / 2 on one
            // exponent (half_square).  Where that serves all 32 points (near_group: hardly
            // ever not) an element costs two shifts by constants of its row and one by its
            // centre's, else oz::level.  With the centres from global memory and level()
            // for all, a chunk of 1e7 products took 59 us instead of 42.
            OzUnit un{0, 0};
            bool near = true;
            int rh = 0;
            int4 *cols = cols_sh + (warp - 2) * COLS;
            if constexpr (!SUM) {
                un = p.units[min(mt * TM + row, p.mrows - 1)];
                const oz::Centre c = p.cen[min(nt * TN + 16 * h + (lane & 15), p.ncols - 1)];
                int top = c.yx;
#pragma unroll
                for (int o = 8; o > 0; o >>= 1)
                    top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
                const int64_t hs = oz::half_square(c, top);
                __syncwarp();
                if (lane < COLS)
                    cols[lane] = make_int4((int) hs, (int) (hs >> 32), c.f, 0);
                __syncwarp();
                near = __all_sync(0xffffffffu, oz::near_group(top, un.u));
                rh = un.u - top + 10;
            }
            for (int pn = p0; pn < p1; pn += SEG, nseg++) {
                if (!mbar_wait(acc_full, (uint32_t) (nseg & 1), p.status, 76)) {
                    ok = false;
                    break;
                }
                __syncwarp();
                tc_fence_after();
                // four columns a batch; the accumulators are free once the last one is read
                auto fetch = [&](int cb, uint32_t *v) {
#pragma unroll
                    for (int l = 0; l < SB; l++)
                        tmem_ld4p(lane_base + (uint32_t) (l * TN + 4 * cb), v + 4 * l);
                    tmem_ld_wait();
                    if (cb == 3) {
                        tc_fence_before();
                        mbar_arrive(acc_empty);
                    }
                };
                // units 2^-61 (sa = 8): 8 bits down; sa = 1: exact in 2^-55
                auto product = [&](const uint32_t *v) {
                    int64_t hi, lo;
                    level_pairs<NARROW>(v, hi, lo);
                    return SA == 1 ? hi * 268435456 + lo : hi * 1048576 + ((lo + 128) >> 8);
                };
                const int m = mt * TM + row, n0 = nt * TN + 16 * h;
                int64_t *out = SUM ? nullptr : p.out + (size_t) n0 * p.ldm + m;
                if constexpr (SUM) {
#pragma unroll
                    for (int cb = 0; cb < 4; cb++) {
                        uint32_t v[4 * SB];
                        fetch(cb, v);
#pragma unroll
                        for (int c = 0; c < 4; c++) {
                            int64_t hi, lo;
                            level_pairs<NARROW>(v + c, hi, lo);
                            oz::add96(acc[4 * cb + c], hi, lo);
                        }
                    }
                } else if (near) {
#pragma unroll
                    for (int cb = 0; cb < 4; cb++) {
                        uint32_t v[4 * SB];
                        fetch(cb, v);
#pragma unroll
                        for (int c = 0; c < 4; c++) {
                            const int j = 4 * cb + c;
                            const int4 y = cols[j];
                            const int64_t hs = (int64_t) (uint32_t) y.x | ((int64_t) y.y << 32);
                            const int64_t x = oz::shifted(product(v + c), un.p + y.z - un.u) - oz::sar(hs, rh);
                            if (m < p.mrows && n0 + j < p.ncols)
                                out[(size_t) j * p.ldm] = x;
                        }
                    }
                } else {
#pragma unroll 1
                    for (int cb = 0; cb < 4; cb++) {
                        uint32_t v[4 * SB];
                        fetch(cb, v);
#pragma unroll
                        for (int c = 0; c < 4; c++) {
                            const int j = 4 * cb + c;
                            const int64_t x = oz::level(product(v + c), p.cen[min(n0 + j, p.ncols - 1)], un.p, un.u);
                            if (m < p.mrows && n0 + j < p.ncols)
                                out[(size_t) j * p.ldm] = x;
                        }
                    }
                }
            }
            if constexpr (SUM) {
                if (ok) {
                    double *dst = p.sums + (size_t) it * (TM * TN) + (size_t) (16 * h) * TM + row;
#pragma unroll
                    for (int c = 0; c < 16; c++)
                        dst[(size_t) c * TM] = oz::to_double96(acc[c]);
                }
            }
        }
        if (!ok)
            failed = 1;
    }
    __syncthreads();
    if (failed && warp == 1) {
        mma_commit_w(drain);
        mbar_wait_w(drain, 0, p.status, 77, 100000000ull);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0)
        tmem_dealloc(tmem, 512);
}

__host__ __device__ constexpr int rup(int a, int b) { return (a + b - 1) / b * b; }

}  // namespace

// Splits of the contraction: whole panels an item, the count that gives the
// shortest schedule of equal items on `sms` CTAs (36 x 128 clocks of MMA a panel,
// about 5000 clocks to fill the pipeline and drain the accumulator, 60 an item to
// write its sums and read them back).
int oz_item_panels(int ntile, int panels, int sms)
{
    int per = 1;
    double best = 1e300;
    for (int c = 1; c <= panels; c++) {
        const double items = (double) ntile * ceil_div(panels, c);
        const double cost = ceil(items / sms) * (c * 4608.0 + 5000.0) + 60.0 * items;
        if (cost < best) {
            best = cost;
            per = c;
        }
    }
    return per;
}

int launch_oz_gemm(const OzGemm &g, int sms, int *status, cudaStream_t s)
{
    CUtensorMap tmA, tmB;
    const uint64_t lda = (uint64_t) g.a_ld, ldb = (uint64_t) g.b_ld;
    int rc = make_tmap_bf16(&tmA, g.A, (uint64_t) g.sa * g.a_rows, lda, lda, TM, PANEL);
    if (rc == DGTM_OK)
        rc = make_tmap_bf16(&tmB, g.B, (uint64_t) SB * g.b_rows, ldb, ldb, TN, PANEL);
    if (rc != DGTM_OK)
        return rc;
    OzParams p{};
    p.panels = g.panels;
    p.b_panel0 = g.b_panel0;
    p.a_rows = g.a_rows;
    p.b_rows = g.b_rows;
    p.a_tile0 = g.a_tile0;
    p.b_row0 = g.b_row0;
    p.mtiles = g.mtiles;
    p.ntiles = g.ntiles;
    p.item_panels = g.sums ? g.item_panels : g.panels;
    p.splits = ceil_div(g.panels, p.item_panels);
    p.nitems = (g.tiles ? g.ntile : g.mtiles * g.ntiles) * p.splits;
    p.tiles = g.tiles;
    p.sums = g.sums;
    p.out = g.out;
    p.ldm = g.ldm;
    p.mrows = g.mrows;
    p.ncols = g.ncols;
    p.units = g.units;
    p.cen = g.cen;
    p.skip = g.skip;
    p.status = status;
    using Kernel = void (*)(const CUtensorMap, const CUtensorMap, const OzParams);
    // |S_l| <= (l + 1) 64 panels 4096: at most 2^22 for two panels, and for 0/1 data
    const Kernel k = g.sums       ? (Kernel) oz_gemm_kernel<8, true, false>
                     : g.sa == 1  ? (Kernel) oz_gemm_kernel<1, false, true>
                     : g.panels <= 2 ? (Kernel) oz_gemm_kernel<8, false, true>
                                     : (Kernel) oz_gemm_kernel<8, false, false>;
    DGTM_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) OZ_SMEM));
    k<<<p.nitems < sms ? p.nitems : sms, OZ_THREADS, OZ_SMEM, s>>>(tmA, tmB, p);
    DGTM_CUDA_TRY(cudaGetLastError());
    return DGTM_OK;
}

// ---------------------------------------------------------------------------
// the M-step's normal equations
// ---------------------------------------------------------------------------
struct OzAB {
    int K = 0, M1 = 0, D = 0, sms = 0;
    int Kp = 0, panels = 0, Mp = 0, Ap = 0, Wp = 0;  // Ap: columns of diag(G) FI, padded to 64
    int ntile = 0, splits = 0, item_panels = 0;
    __nv_bfloat16 *Fp = nullptr, *Wpl = nullptr;
    unsigned long long *fbits = nullptr, *wbits = nullptr;
    double *part = nullptr;
    int *tiles = nullptr;
    int *wide = nullptr;  // G spans too much for the columns' grids: form_ab's chain does it
};

namespace {

// A column of diag(G) FI is on the grid of its largest value, and what a basis function
// loses is 2^-56 of that times its own largest value.  Where G is far smaller in the reach
// of one basis function than elsewhere, the terms that determine its weights are as far
// below the grid.  The line is a factor of 2^4 between max G times the function's maximum
// and the maximum of their product.  Against long double, at K = 1600 to 8000, M1 = 65 and
// 82, bases of condition 3e4 to 1e14, G falling over 0 to 12 decades: the centres' error is
// 0.03 to 1.1 times the multiply-add chain's up to there (0.5 in the middle), 2 at 2^6,
// 5 at 2^8, 30 at 2^13, 1000 at 2^20.
__global__ void __launch_bounds__(256) ozab_wide_kernel(const unsigned long long *__restrict__ fbits,
                                                        const unsigned long long *__restrict__ wbits, int M1,
                                                        int gcol, int *__restrict__ wide)
{
    const double g = oz::bits_double(wbits[gcol]);
    int w = 0;
    for (int m = threadIdx.x; m < M1; m += 256)
        w |= !(oz::bits_double(fbits[m]) * g <= 16.0 * oz::bits_double(wbits[m]));
    w = __syncthreads_or(w);
    if (threadIdx.x == 0)
        *wide = w;
}

// A and B from the tiles' split sums; a column with a non-finite value gives NaN.
__global__ void __launch_bounds__(256) ozab_reduce_kernel(const double *__restrict__ part,
                                                          const int *__restrict__ tiles, int splits,
                                                          int M1, int D, int Ap,
                                                          const unsigned long long *__restrict__ fbits,
                                                          const unsigned long long *__restrict__ wbits,
                                                          double *__restrict__ A, double *__restrict__ B,
                                                          int *__restrict__ flag, const int *__restrict__ wide)
{
    if (*wide)
        return;
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x < 3)
        flag[threadIdx.x] = 0;
    const int t = blockIdx.x, v = tiles[t], mt = v >> 16, nt = v & 0xFFFF;
    for (int e = blockIdx.y * 256 + threadIdx.x; e < TM * TN; e += 256 * gridDim.y) {
        const int m = mt * TM + (e & (TM - 1)), c = nt * TN + (e >> 7);
        const bool isA = c < Ap;
        const int j = isA ? c : c - Ap;
        if (m >= M1 || (isA ? (j >= M1 || j < m) : j >= D))
            continue;
        double sum = 0.0;
        for (int sp = 0; sp < splits; sp++)
            sum += part[((size_t) t * splits + sp) * (TM * TN) + e];
        const unsigned long long fb = fbits[m], wb = wbits[isA ? j : M1 + j];
        double r = scalbn(sum, oz::exponent_of(fb) + oz::exponent_of(wb) - OZ_SUM_BITS);
        if (fb >= oz::INF_BITS || wb >= oz::INF_BITS)
            r = NAN;
        if (isA) {
            A[(size_t) m * M1 + j] = r;
            A[(size_t) j * M1 + m] = r;
        } else {
            B[(size_t) m * D + j] = r;
        }
    }
}

}  // namespace

// Measured, the whole solve phase by slices against by the chain: 198 us against 215 at
// K = 4000, M1 = 50, D = 75 and 196 against 260 at K = 8000, M1 = 50, D = 25 (2.0e7, the
// line: below it the slices' six launches have little left to win), 398 against 582 at
// K = 8000, M1 = 65, D = 166 (1.0e8).
bool ozab_wanted(int K, int M1, int D)
{
    return K <= (1 << 26) && (double) K * M1 * (0.5 * M1 + D) >= 2e7;
}

void ozab_destroy(OzAB *st)
{
    if (!st)
        return;
    void *ptrs[] = {st->Fp, st->Wpl, st->fbits, st->wbits, st->part, st->tiles, st->wide};
    for (void *p : ptrs)
        if (p)
            cudaFree(p);
    delete st;
}

int ozab_create(OzAB **out, int K, int M1, int D, int sms, cudaStream_t s)
{
    *out = nullptr;
    OzAB *st = new (std::nothrow) OzAB();
    if (!st) {
        set_error(DGTM_ENOMEM, "host allocation failed");
        return DGTM_ENOMEM;
    }
    st->K = K;
    st->M1 = M1;
    st->D = D;
    st->sms = sms;
    st->Kp = rup(K, PANEL);
    st->panels = st->Kp / PANEL;
    st->Mp = rup(M1, TM);
    st->Ap = rup(M1, TN);
    st->Wp = st->Ap + rup(D, TN);
    // the tiles that reach the upper triangle of A, and all of B's
    std::vector<int> tiles;
    for (int mt = 0; mt < st->Mp / TM; mt++)
        for (int nt = 0; nt < st->Wp / TN; nt++)
            if (nt * TN >= st->Ap || nt * TN + TN - 1 >= mt * TM)
                tiles.push_back(mt << 16 | nt);
    st->ntile = (int) tiles.size();
    const int per = oz_item_panels(st->ntile, st->panels, sms);
    st->item_panels = per;
    st->splits = ceil_div(st->panels, per);
    cudaError_t e = cudaMalloc((void **) &st->Fp, sizeof(__nv_bfloat16) * oz::DIGITS * (size_t) st->Mp * st->Kp);
    if (e == cudaSuccess)
        e = cudaMalloc((void **) &st->Wpl, sizeof(__nv_bfloat16) * oz::DIGITS * (size_t) st->Wp * st->Kp);
    if (e == cudaSuccess)
        e = cudaMalloc((void **) &st->fbits, sizeof(unsigned long long) * M1);
    if (e == cudaSuccess)
        e = cudaMalloc((void **) &st->wbits, sizeof(unsigned long long) * (M1 + D + 1));
    if (e == cudaSuccess)
        e = cudaMalloc((void **) &st->part, sizeof(double) * TM * TN * (size_t) st->ntile * st->splits);
    if (e == cudaSuccess)
        e = cudaMalloc((void **) &st->wide, sizeof(int));
    if (e == cudaSuccess)
        e = cudaMalloc((void **) &st->tiles, sizeof(int) * tiles.size());
    // on the stream of their readers; from pageable memory the call returns once the
    // list is staged
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(st->tiles, tiles.data(), sizeof(int) * tiles.size(), cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) {
        const int code = e == cudaErrorMemoryAllocation ? DGTM_ENOMEM : DGTM_ECUDA;
        cudaGetLastError();
        set_error(code, "ozab_create: %s", cudaGetErrorString(e));
        ozab_destroy(st);
        return code;
    }
    *out = st;
    return DGTM_OK;
}

// FI's digit planes, once per basis; the padding rows of both operands are zero
int ozab_basis(OzAB *st, const double *FI, cudaStream_t s)
{
    const int K = st->K, M1 = st->M1;
    DGTM_CUDA_TRY(cudaMemsetAsync(st->Fp, 0, sizeof(__nv_bfloat16) * oz::DIGITS * (size_t) st->Mp * st->Kp, s));
    DGTM_CUDA_TRY(cudaMemsetAsync(st->Wpl, 0, sizeof(__nv_bfloat16) * oz::DIGITS * (size_t) st->Wp * st->Kp, s));
    DGTM_CUDA_TRY(cudaMemsetAsync(st->fbits, 0, sizeof(unsigned long long) * M1, s));
    const OzSource src{nullptr, FI, nullptr, M1, M1, 0};
    oz_colmax_kernel<<<dim3(ceil_div(K, 128), ceil_div(M1, 32)), 256, 0, s>>>(src, K, M1, 128, st->fbits);
    DGTM_CUDA_TRY(cudaGetLastError());
    oz_slice_t_kernel<<<dim3(st->panels, ceil_div(M1, 32)), 256, 0, s>>>(src, K, M1, st->Mp, st->Kp,
                                                                        st->fbits, st->Fp, nullptr, nullptr);
    DGTM_CUDA_TRY(cudaGetLastError());
    return DGTM_OK;
}

int ozab_form(OzAB *st, const double *FI, const double *G, const double *RT, double *A, double *B, double *scratch,
              int *flag, int *nlaunch, cudaStream_t s)
{
    const int K = st->K, M1 = st->M1, D = st->D, W = M1 + D + 1;
    DGTM_CUDA_TRY(cudaMemsetAsync(st->wbits, 0, sizeof(unsigned long long) * W, s));
    // diag(G) FI at rows 0 .. M1 of the planes, RT at rows Ap ..; and G's own maximum
    const OzSource both{G, FI, RT, M1, M1, D};
    oz_colmax_kernel<<<dim3(ceil_div(K, 128), ceil_div(W, 32)), 256, 0, s>>>(both, K, W, 128, st->wbits);
    DGTM_CUDA_TRY(cudaGetLastError());
    // every launch below looks at wide: the slices do nothing where it is set, the chain
    // where it is not
    ozab_wide_kernel<<<1, 256, 0, s>>>(st->fbits, st->wbits, M1, W - 1, st->wide);
    DGTM_CUDA_TRY(cudaGetLastError());
    const OzSource left{G, FI, nullptr, M1, M1, 0}, right{nullptr, RT, nullptr, D, D, 0};
    oz_slice_t_kernel<<<dim3(st->panels, ceil_div(M1, 32)), 256, 0, s>>>(left, K, M1, st->Wp, st->Kp,
                                                                        st->wbits, st->Wpl, nullptr, st->wide);
    DGTM_CUDA_TRY(cudaGetLastError());
    oz_slice_t_kernel<<<dim3(st->panels, ceil_div(D, 32)), 256, 0, s>>>(
        right, K, D, st->Wp, st->Kp, st->wbits + M1, st->Wpl + (size_t) st->Ap * st->Kp, nullptr,
        st->wide);
    DGTM_CUDA_TRY(cudaGetLastError());
    OzGemm g;
    g.A = st->Fp;
    g.B = st->Wpl;
    g.a_rows = st->Mp;
    g.b_rows = st->Wp;
    g.panels = st->panels;
    g.a_ld = g.b_ld = st->Kp;
    g.mtiles = st->Mp / TM;
    g.ntiles = st->Wp / TN;
    g.tiles = st->tiles;
    g.ntile = st->ntile;
    g.sums = st->part;
    g.item_panels = st->item_panels;
    g.skip = st->wide;
    int rc = launch_oz_gemm(g, st->sms, flag + 3, s);
    if (rc != DGTM_OK)
        return rc;
    ozab_reduce_kernel<<<dim3(st->ntile, 32), 256, 0, s>>>(st->part, st->tiles, st->splits, M1, D, st->Ap,
                                                          st->fbits, st->wbits, A, B, flag, st->wide);
    DGTM_CUDA_TRY(cudaGetLastError());
    if ((rc = launch_form_ab(FI, G, RT, K, M1, D, A, B, scratch, flag, s, st->wide)) != DGTM_OK)
        return rc;
    if (nlaunch)
        *nlaunch = 8;
    return DGTM_OK;
}

}  // namespace dgtm
