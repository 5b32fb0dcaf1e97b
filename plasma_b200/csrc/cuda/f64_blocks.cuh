// f64_blocks.cuh -- 32 x 32 FP64 blocks in shared memory and the triangular
// solve of 8-row strips on DMMA, shared by the diagonal-tile factor
// (potrf_diag.cu) and the panel solve (trsm_f64.cu).
//
// Blocks are column-major, 32 x 32 without padding; the row index of column
// c is XORed with 4 ((c + c/4) mod 4).  That keeps the DMMA operand reads
// (four consecutive or four even columns x 8 rows a warp) and the accumulator
// accesses free of bank conflicts, and pairs of rows adjacent.
#pragma once
#include "common.cuh"

namespace {

constexpr int F64_BLK = 32 * 32;              // elements per block

__device__ __forceinline__ int pd_at(int c, int r)
{
    return c * 32 + (r ^ (4 * ((c + (c >> 2)) & 3)));
}

// FP64 MMA of 8 x 8 x 4.  Lane = 4 g + t holds a (g, t), b (k = t, n = g) and
// the accumulator (g, 2t), (g, 2t+1).  The small shape: a strip of 8 rows
// halves the latency of every dependent step against 16 x 8 x 8, at the same
// rate.
__device__ __forceinline__ void dmma_8x8x4(double (&c)[2], double a, double b)
{
    asm volatile(
        "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
        : "+d"(c[0]), "+d"(c[1]) : "d"(a), "d"(b));
}

// A strip of 8 rows x 8 columns lives in a warp's registers as such an
// accumulator.  It serves unchanged as the A operand of the next product
// when the K index is taken in the order 2t, then 2t+1: the B operands of
// columns 8q .. 8q+7 are then B(8q + 2t, g) and B(8q + 2t + 1, g).
__device__ __forceinline__ void strip_mma(double (&d)[2], const double (&x)[2], double sign,
                                          double b0, double b1)
{
    dmma_8x8x4(d, sign * x[0], b0);
    dmma_8x8x4(d, sign * x[1], b1);
}

// The inverse of the 8 x 8 lower-triangular block whose entry (i, q) is
// l(i, q) and whose diagonal has the reciprocals r(i): column j of it.
template <typename L, typename R>
__device__ __forceinline__ void inv8_column(int j, L l, R r, double (&w)[8])
{
#pragma unroll
    for (int i = 0; i < 8; i++) {
        double s = i == j ? 1.0 : 0.0;
#pragma unroll
        for (int q = 0; q < i; q++) s = fma(-l(i, q), w[q], s);
        w[i] = i >= j ? s * r(i) : 0.0;
    }
}

// Y L^T = X for 8 rows and the 32 columns of a diagonal block, in place:
// y[q] = columns 8q .. 8q+7.  D: the block (pd_at layout); W8: the inverses
// of its 8 x 8 diagonal blocks, entry (i, j) of block q at
// W8[(8 q + j) * 8 + i].  Only 8 x 8 blocks are inverted, so the result
// differs from plain substitution by no more than their condition, and the
// solve runs at the pace of four dependent pairs of products.
__device__ __forceinline__ void strip_solve32(double (&y)[4][2], const double *D,
                                              const double *W8)
{
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        double x[2] = {0.0, 0.0};
        strip_mma(x, y[q], 1.0, W8[(8 * q + 2 * t) * 8 + g], W8[(8 * q + 2 * t + 1) * 8 + g]);
#pragma unroll
        for (int f = q + 1; f < 4; f++)
            strip_mma(y[f], x, -1.0, D[pd_at(8 * q + 2 * t, 8 * f + g)],
                      D[pd_at(8 * q + 2 * t + 1, 8 * f + g)]);
        y[q][0] = x[0];
        y[q][1] = x[1];
    }
}

}  // namespace
