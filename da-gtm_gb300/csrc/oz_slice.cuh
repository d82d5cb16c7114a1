// oz_slice.cuh -- kernels that cut FP64 matrices into the digit planes of the
// digit-slice products (oz.cu).  Bound by memory: 8 bytes in, 16 out a value.
#pragma once

#include "ozfix.cuh"
#include "sm100.cuh"

#include <cuda_bf16.h>

namespace dgtm {
namespace {

// The digits of two values as BF16 pairs, w[i] = (digit i of a, digit i of b):
// a field f becomes the float 2^23 + f by its bits, f - 64 by one subtraction, and
// its upper half is the BF16, since eight bits hold it.
__device__ __forceinline__ void digit_pairs(int64_t a, int64_t b, uint32_t (&w)[oz::DIGITS])
{
    const uint64_t ua = (uint64_t) a + oz::digit_bias(), ub = (uint64_t) b + oz::digit_bias();
#pragma unroll
    for (int i = 0; i < oz::DIGITS; i++) {
        const float x = __fsub_rn(__uint_as_float(oz::digit_field(ua, i) | 0x4B000000u), 8388672.f);
        const float y = __fsub_rn(__uint_as_float(oz::digit_field(ub, i) | 0x4B000000u), 8388672.f);
        w[i] = __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632);
    }
}

// Column c of the source: c < c1: G[k] X1[k][c] (G may be null), else X2[k][c - c1], then
// G[k] (X2 null: 1).
struct OzSource {
    const double *G, *X1, *X2;
    int c1, ld1, ld2;
    __device__ __forceinline__ double at(int k, int c) const
    {
        if (c < c1) {
            const double v = X1[(size_t) k * ld1 + c];
            return G ? G[k] * v : v;
        }
        return !X2 ? 1.0 : c - c1 < ld2 ? X2[(size_t) k * ld2 + (c - c1)] : G[k];
    }
};

// bits[c] = max(bits[c], the largest |value| of column c over the block's rows)
static __global__ void __launch_bounds__(256) oz_colmax_kernel(OzSource src, int rows, int cols, int rows_per,
                                                        unsigned long long *__restrict__ bits)
{
    __shared__ unsigned long long red[8][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int c = blockIdx.y * 32 + lane;
    const int k0 = blockIdx.x * rows_per, k1 = min(rows, k0 + rows_per);
    unsigned long long m = 0ull;
    if (c < cols)
        for (int k = k0 + w; k < k1; k += 8) {
            const unsigned long long b = oz::double_bits(src.at(k, c)) & oz::ABS_MASK;
            m = b > m ? b : m;
        }
    red[w][lane] = m;
    __syncthreads();
    if (w == 0 && c < cols) {
        for (int i = 1; i < 8; i++)
            m = red[i][lane] > m ? red[i][lane] : m;
        atomicMax(&bits[c], m);
    }
}

// planes[i][c][k] = digit i of column c of the source on the column's grid:
// the transposed operand (contraction over the source's rows), zero past rows
// and cols.  low (may be null): low[c] += how many values of column c are short of bits on
// its grid.  skip (may be null): nothing is done where *skip is set.  Block: 64 rows x 32
// columns.
static __global__ void __launch_bounds__(256) oz_slice_t_kernel(OzSource src, int rows, int cols, int prows,
                                                         int ld, const unsigned long long *__restrict__ bits,
                                                         __nv_bfloat16 *__restrict__ planes,
                                                         unsigned *__restrict__ low, const int *__restrict__ skip)
{
    if (skip && *skip)
        return;
    __shared__ int64_t qs[32][65];
    __shared__ unsigned few[8][32];
    const int k0 = blockIdx.x * 64, c0 = blockIdx.y * 32;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int c = c0 + lane;
    const int e = c < cols ? oz::exponent_of(bits[c]) : 0;
    unsigned n = 0;
#pragma unroll
    for (int r = w; r < 64; r += 8) {
        const int k = k0 + r;
        const double v = (k < rows && c < cols) ? src.at(k, c) : 0.0;
        qs[lane][r] = oz::to_fixed(v, e);
        n += oz::short_of_bits(v, e);
    }
    few[w][lane] = n;
    __syncthreads();
    if (low && w == 0 && c < cols) {
        for (int i = 1; i < 8; i++)
            n += few[i][lane];
        if (n)
            atomicAdd(&low[c], n);
    }
#pragma unroll
    for (int cc = w; cc < 32; cc += 8) {
        if (c0 + cc >= prows)
            break;
        uint32_t v[oz::DIGITS];
        digit_pairs(qs[cc][2 * lane], qs[cc][2 * lane + 1], v);
        uint32_t *dst = (uint32_t *) (planes + (size_t) (c0 + cc) * ld + k0) + lane;
        const size_t plane = (size_t) prows * ld / 2;
#pragma unroll
        for (int i = 0; i < oz::DIGITS; i++)
            dst[(size_t) i * plane] = v[i];
    }
}

}  // namespace
}  // namespace dgtm
