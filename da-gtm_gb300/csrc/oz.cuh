// oz.cuh -- FP64-accurate products on the tensor cores by digit slices (oz.cu).
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "ozfix.cuh"

namespace dgtm {

// a point's unit 2^u and p (oz::level)
struct OzUnit {
    int p, u;
};

// One product C[m][n] = sum_k A[m][k] B[n][k] over digit planes: A has sa planes
// (8, or 1 for values that are small integers themselves) of a_rows x a_ld BF16, B has
// 8 planes of b_rows x b_ld; row lengths a multiple of 8.  The contraction runs over
// `panels` panels of 64, from panel 0 of A and panel b_panel0 of B; columns past a row's
// end count as zero.  Rows of a last tile past a_rows or b_rows are the next plane's:
// what they give is finite and not read.
struct OzGemm {
    const __nv_bfloat16 *A = nullptr, *B = nullptr;
    int sa = 8;
    int a_rows = 0, b_rows = 0;
    int panels = 0;        // 64-deep panels of the contraction
    int a_ld = 0, b_ld = 0, b_panel0 = 0;
    int a_tile0 = 0;       // first 128-row tile of A
    int b_row0 = 0;        // first row of B (tiles of 64 from there)
    int mtiles = 0, ntiles = 0;
    const int *tiles = nullptr;  // (mt << 16 | nt) of each tile, or null: all mtiles x ntiles
    int ntile = 0;               // entries of tiles
    // sums (not null): an item is one tile over `item_panels` panels; it leaves 64 x 128
    // doubles (column, row), each an exact sum rounded once, in units of 2^-OZ_SUM_BITS of
    // the operands' 2^e, at sums + item 8192, item = tile * splits + split
    double *sums = nullptr;
    int item_panels = 0;
    // distances (sums == null, panels <= 4): out[n ldm + m] = oz::level of the sum, which
    // is in units of 2^-53 (sa = 8) or 2^-55 (sa = 1) of the operands' 2^e, for m < mrows,
    // n < ncols; units of A's rows from a_tile0, centres of B's rows from b_row0
    int64_t *out = nullptr;
    size_t ldm = 0;
    int mrows = 0, ncols = 0;
    const OzUnit *units = nullptr;
    const oz::Centre *cen = nullptr;
    const int *skip = nullptr;  // device, may be null: nothing is done where it is set
};

constexpr int OZ_SUM_BITS = 61;
int oz_item_panels(int ntile, int panels, int sms);
int launch_oz_gemm(const OzGemm &g, int sms, int *status, cudaStream_t s);

// A = FI^T diag(G) FI and B = FI^T RT by digit slices; FI's planes are kept.
struct OzAB;
int ozab_create(OzAB **out, int K, int M1, int D, int sms, cudaStream_t s);
int ozab_basis(OzAB *st, const double *FI, cudaStream_t s);
void ozab_destroy(OzAB *st);
// flag: [0..2] set to 0 (as launch_form_ab does), [3] the bounded waits' status word.
// scratch: form_ab_scratch_doubles, for the multiply-add chain that takes over where G
// spans too much for the columns' grids
int ozab_form(OzAB *st, const double *FI, const double *G, const double *RT, double *A, double *B, double *scratch,
              int *flag, int *nlaunch, cudaStream_t s);
// whether the digit-slice product is the faster one at this size
bool ozab_wanted(int K, int M1, int D);

// The E-step, responsibility pass and map from digit-slice distances
// (oz_estep.cu).
struct OzE;
struct OzEArgs {
    const double *T64, *tt;  // N x D, N
    int N, D, K, sms;
    // 0/1 data already in BF16 (rows_pad a multiple of 128, ld = 64 panels; columns
    // past D meet zeros), or null: eight digit planes of T64 are made
    const __nv_bfloat16 *Tb;
    int Tb_rows, Tb_ld;
    bool mstep;              // with what the responsibility pass needs
    int *status;             // device: the bounded waits' status word
};
bool oze_wanted(int N, int D, int K);
// *out stays null (and the call succeeds) where the data have a non-finite value or, for
// the responsibility pass, a column that does not fit one grid
int oze_create(OzE **out, const OzEArgs &a, cudaStream_t s);
void oze_destroy(OzE *st);
int oze_estep_blocks(const OzE *st);
// sums: the two totals of part
int oze_estep(OzE *st, const double *Y, const double *yy, double c1, double c2, int isDA,
              double2 *colstat, double *part, double dcut, double *sums, int *nlaunch, cudaStream_t s);
int oze_mstep_pass(OzE *st, double c, double *G, double *RT, int *nlaunch, cudaStream_t s);
// The parts other products with R are made of.  oze_refer: the centres' planes and
// the points' references (kept when they are those of the last oze_estep; c1 = beta / 2,
// c the exponents' factor);
// oze_chunks: how many chunks, and their points; oze_r_digits: R (or R^2) of the
// centres k0 .. k0 + kb over a chunk as eight planes of prows x (points rounded
// up to 64), and the integer exponents of their grids: a sum of the
// product with B counts 2^(5 - nmin[k]) of B's grid.  products: form
// the chunk's distances first (they stay until the next chunk's).
int oze_refer(OzE *st, const double *Y, const double *yy, const double2 *colstat, double c1, double c, double dcut,
              cudaStream_t s);
int oze_chunks(const OzE *st, int *points);
int oze_r_digits(OzE *st, int ch, int k0, int kb, double c, bool squares, bool products, int prows,
                 __nv_bfloat16 *planes, int *nmin, cudaStream_t s);
// R of the centres k0 .. k0 + nk and the points n0 .. n0 + nn (nk x nn)
int oze_r_block(OzE *st, const double *Y, const double *yy, const double2 *colstat, double c1, double c, double dcut,
                int k0, int nk, int n0, int nn, double *R, cudaStream_t s);
// M = R^T X from a context's column statistics
int oze_map(OzE *st, const double *Y, const double *yy, const double2 *colstat, double c1, double c,
            const double *X, int L, double *M, cudaStream_t s);

// The AUTO schedule's scatter in FP64 accuracy as digit-slice products of R and
// R^2 with pair features (oz_ctemp.cu): out and gsum as launch_ctemp_batch;
// spread[k]: what the expansion about the data's mean and the features' grids cost, as a
// factor of 2^-53 (see there).  DGTM_ENOMEM (nothing done) if not even 128 centres fit the budget.
int oz_ctemp(OzE *st, const double *T64, const double *Y, const double *yy, const double2 *colstat, int N,
             int D, int K, int sms, double c1, double c, double dcut, const double *gg_dev, double lim_scale,
             size_t budget, double *gsum_dev, double *out_dev, double *spread_dev, int *status,
             cudaStream_t s);

}  // namespace dgtm
