// oz.cuh -- FP64-accurate products on the tensor cores by digit slices (oz.cu).
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "ozfix.cuh"

namespace dgtm {

// One product C[m][n] = sum_k A[m][k] B[n][k] over digit planes: A has sa planes
// (8, or 1 for values that are small integers themselves) of a_rows x ld BF16,
// B has 8 planes of b_rows x ld; ld = 64 panels; a_rows a multiple of 128,
// b_rows of 64.
struct OzGemm {
    const __nv_bfloat16 *A = nullptr, *B = nullptr;
    int sa = 8;
    int a_rows = 0, b_rows = 0;
    int panels = 0;        // 64-deep panels of the contraction
    int a_tile0 = 0;       // first 128-row tile of A
    int mtiles = 0, ntiles = 0;
    const int *tiles = nullptr;  // (mt << 16 | nt) of each tile, or null: all mtiles x ntiles
    int ntile = 0;               // entries of tiles
    // sums (out64 != null): an item is one tile over `item_panels` panels; it leaves
    // 64 x 128 integers (column, row) in units of 2^(-53 + oz_sum_ext(panels)) of
    // the operands' 2^e at out64 + item 8192, item = tile * splits + split; the
    // integers of all splits can be added
    int64_t *out64 = nullptr;
    int item_panels = 0;
    // distances (out64 == null, panels <= 4): out[n ldm + m] = sum >> shift in units of
    // 2^-53 (sa = 8) or 2^-55 (sa = 1) of the operands' 2^e, for m < mrows, n < ncols
    int64_t *out = nullptr;
    size_t ldm = 0;
    int mrows = 0, ncols = 0;
    const int *shift = nullptr;  // device: further right shift (see oz.cu)
};

int oz_sum_ext(int panels);
int launch_oz_gemm(const OzGemm &g, int sms, int *status, cudaStream_t s);

// A = FI^T diag(G) FI and B = FI^T RT by digit slices; FI's planes are kept.
struct OzAB;
int ozab_create(OzAB **out, int K, int M1, int D, int sms);
int ozab_basis(OzAB *st, const double *FI, cudaStream_t s);
void ozab_destroy(OzAB *st);
int ozab_form(OzAB *st, const double *FI, const double *G, const double *RT, double *A, double *B,
              int *status, int *nlaunch, cudaStream_t s);
// whether the digit-slice product is the faster one at this size
bool ozab_wanted(int K, int M1, int D);

}  // namespace dgtm
