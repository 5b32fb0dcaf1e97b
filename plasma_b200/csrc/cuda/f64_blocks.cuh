// f64_blocks.cuh -- 32 x 32 blocks in shared memory, their Cholesky factor by
// one warp and the triangular solve of strips of rows on the tensor cores,
// shared by the diagonal-tile factor (potrf_diag.cu), the panel solve
// (trsm_f64.cu) and the batched kernel (batched.cu, FP64 and FP32).
//
// Blocks are column-major, 32 x 32 without padding; the row index of column
// c is XORed with 4 ((c + c/4) mod 4).  That keeps the DMMA operand reads
// (four consecutive or four even columns x 8 rows a warp) and the accumulator
// accesses free of bank conflicts, and pairs of rows adjacent.
#pragma once
#include "common.cuh"
#include "mma.cuh"

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
__device__ __forceinline__ void strip_mma(double (&d)[2], const double (&x)[2], double b0,
                                          double b1)
{
    dmma_8x8x4(d, x[0], b0);
    dmma_8x8x4(d, x[1], b1);
}

// The inverse of the 8 x 8 lower-triangular block whose entry (i, q) is
// l(i, q) and whose diagonal has the reciprocals r(i): column j of it.
template <typename T, typename L, typename R>
__device__ __forceinline__ void inv8_column(int j, L l, R r, T (&w)[8])
{
#pragma unroll
    for (int i = 0; i < 8; i++) {
        T s = i == j ? T(1) : T(0);
#pragma unroll
        for (int q = 0; q < i; q++) s = fma(-l(i, q), w[q], s);
        w[i] = i >= j ? s * r(i) : T(0);
    }
}

// Y L^T = X - S for 8 rows and the 32 columns of a diagonal block, in place:
// y[q] = columns 8q .. 8q+7 of X, then of Y; s[q] those of S, what solved
// columns to the left owe (destroyed).  D: the block (pd_at layout); W8: the
// inverses of its 8 x 8 diagonal blocks, entry (i, j) of block q at
// W8[(8 q + j) * 8 + i].  Only 8 x 8 blocks are inverted, so the result
// differs from plain substitution by no more than their condition, and the
// solve runs at the pace of four dependent pairs of products.  The products
// are summed apart from X, which takes one rounding: added to X one by one,
// each would round at the size of X (order 300 in tiles of 128, entries below
// the diagonal: 3.3 u against 2.6 u for a well-conditioned Gram matrix).
__device__ __forceinline__ void strip_solve32(double (&y)[4][2], double (&s)[4][2],
                                              const double *D, const double *W8)
{
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        double x[2] = {0.0, 0.0};
#pragma unroll
        for (int e = 0; e < 2; e++) y[q][e] -= s[q][e];
        strip_mma(x, y[q], W8[(8 * q + 2 * t) * 8 + g], W8[(8 * q + 2 * t + 1) * 8 + g]);
#pragma unroll
        for (int f = q + 1; f < 4; f++)
            strip_mma(s[f], x, D[pd_at(8 * q + 2 * t, 8 * f + g)],
                      D[pd_at(8 * q + 2 * t + 1, 8 * f + g)]);
        y[q][0] = x[0];
        y[q][1] = x[1];
    }
}

// 1/sqrt(d) for normal d away from the ends of the range, as mathematics gives
// it: with r near 1/sqrt(d) and e = 1 - d r^2, 1/sqrt(d) = r (1 - e)^(-1/2),
// by the binomial series r (1 + e/2 + 3/8 e^2 + ...).  From the hardware's
// approximation, an instruction with its e below 2^-19, the terms written leave
// 5/16 e^3 < 2^-58 (a step of Householder's method, of third order); the
// roundings of d r and of the result remain, so the error is at most one unit
// in the last place, CUDA's bound for rsqrt().  rsqrt() itself has a slow path
// for the ends of the range (blocks that need it take blk_factor_any); this
// has no branch, so the compiler can run a column's updates between its
// dependent steps.
__device__ __forceinline__ double blk_rsqrt(double d)
{
    double r;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
    const double e = fma(-d * r, r, 1.0);
    return fma(r * e, fma(0.375, e, 0.5), r);
}

// FP32: the hardware's e is below 2^-21 and the series stops at e/2 (Newton's
// step), which leaves 3/8 e^2 < 2^-43; the same bound
__device__ __forceinline__ float blk_rsqrt(float d)
{
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    return fma(0.5f * r, fma(-d * r, r, 1.f), r);
}

// well inside the normal range
__device__ __forceinline__ bool blk_plain(double d) { return d > 1e-280 && d < 1e280; }
__device__ __forceinline__ bool blk_plain(float d) { return d > 1e-30f && d < 1e30f; }

template <typename T> struct Vec2;
template <> struct Vec2<double> { using type = double2; };
template <> struct Vec2<float> { using type = float2; };

// NB x NB Cholesky (NB = 16 or 32) of the block at S by one warp, in place
// (zero above the diagonal on exit), and the inverses of its 8 x 8 diagonal
// blocks to W8.  Eight columns at a time: every lane factors the 8 x 8
// diagonal block for itself, in registers, so a pivot waits for its
// reciprocal square root, one multiplication and one multiply-add, and no
// lane waits for another; its own row and (lanes 0-7) a row of the identity,
// which becomes a column of the inverse, are eliminated in the gaps.  The
// tensor cores update the columns to the right (SPLIT as mma8).  The loop
// over the column groups is kept rolled: unrolled, a block is 1500
// instructions that run once, and fetching them beside the other warps' code
// made a step 12500 clocks where 4300 were its latency.
// False, with S partly overwritten, when a pivot is not well inside the
// normal range (not positive, NaN, tiny or huge).
template <typename T, int SPLIT, int NB>
__device__ __forceinline__ bool blk_factor(T *S, T *W8)
{
    using V2 = typename Vec2<T>::type;
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    bool fine = true;
#pragma unroll 1
    for (int o = 0; o < NB; o += 8) {
        T a[8][8], v[8], u[8];           // a[j][i]: column j, row i >= j
        T dd = T(1), rr = T(1);
#pragma unroll
        for (int j = 0; j < 8; j++)
#pragma unroll
            for (int i = j & ~1; i < 8; i += 2) {
                const V2 x = *reinterpret_cast<const V2 *>(S + pd_at(o + j, o + i));
                a[j][i] = x.x;
                a[j][i + 1] = x.y;
            }
#pragma unroll
        for (int j = 0; j < 8; j++) {
            v[j] = S[pd_at(o + j, lane)];
            u[j] = lane == j ? T(1) : T(0);
        }
        // every lane has read the diagonal block before its rows are written
        __syncwarp();
#pragma unroll
        for (int c = 0; c < 8; c++) {
            const T d = a[c][c];
            fine = fine && blk_plain(d);
            const T r = blk_rsqrt(d);
#pragma unroll
            for (int i = c + 1; i < 8; i++) a[c][i] *= r;
            v[c] *= r;
            u[c] *= r;
#pragma unroll
            for (int j = c + 1; j < 8; j++) {
#pragma unroll
                for (int i = j; i < 8; i++) a[j][i] = fma(-a[c][j], a[c][i], a[j][i]);
                v[j] = fma(-v[c], a[c][j], v[j]);
                u[j] = fma(-u[c], a[c][j], u[j]);
            }
            S[pd_at(o + c, lane)] = lane > o + c ? v[c] : T(0);
            if (lane == o + c) {
                dd = d;
                rr = r;
            }
        }
        // the diagonal: sqrt(d), one Newton step on d r
        if ((unsigned)(lane - o) < 8u) {
            const T s = dd * rr;
            S[pd_at(lane, lane)] = fma(T(0.5) * rr, fma(-s, s, dd), s);
        }
        if (lane < 8) {
#pragma unroll
            for (int i = 0; i < 8; i++) W8[(o + lane) * 8 + i] = u[i];
        }
        __syncwarp();
#pragma unroll
        for (int f = 1; f < NB / 8; f++)
#pragma unroll
            for (int h = 0; h < NB / 16; h++) {
                if (8 * f <= o || 16 * h + 15 < 8 * f) continue;
                const int r0 = 16 * h;
                const T af[4] = {S[pd_at(o + t, r0 + g)], S[pd_at(o + t, r0 + g + 8)],
                                 S[pd_at(o + t + 4, r0 + g)], S[pd_at(o + t + 4, r0 + g + 8)]};
                const T bf[2] = {S[pd_at(o + t, 8 * f + g)], S[pd_at(o + t + 4, 8 * f + g)]};
                T acc[4], old[4];
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    old[e] = S[pd_at(8 * f + 2 * t + (e & 1), r0 + g + 8 * (e >> 1))];
                    acc[e] = T(0);
                }
                mma8<SPLIT>(acc, af, bf);
#pragma unroll
                for (int e = 0; e < 4; e++)
                    S[pd_at(8 * f + 2 * t + (e & 1), r0 + g + 8 * (e >> 1))] = old[e] - acc[e];
            }
        __syncwarp();
    }
    return fine;
}

// The same for any pivots, from the copy of the block at O; returns the
// first bad column + 1 (LAPACK's test), or 0.
template <typename T, int NB>
__device__ __noinline__ int blk_factor_any(T *S, T *W8, const T *O, T *rdiag)
{
    const int lane = threadIdx.x & 31;
    int bad = 0;
    for (int c = 0; c < NB; c++) S[pd_at(c, lane)] = O[pd_at(c, lane)];
    __syncwarp();
    for (int c = 0; c < NB; c++) {
        const T d = S[pd_at(c, c)];
        const bool ok = d > T(0);
        if (!ok && bad == 0) bad = c + 1;
        const T sd = ok ? sqrt(d) : T(1), r = T(1) / sd;
        const T l = lane == c ? sd : lane > c ? S[pd_at(c, lane)] * r : T(0);
        __syncwarp();
        S[pd_at(c, lane)] = l;
        if (lane == c) rdiag[c] = r;
        __syncwarp();
        for (int c2 = c + 1; c2 <= lane && c2 < NB; c2++)
            S[pd_at(c2, lane)] = fma(-l, S[pd_at(c, c2)], S[pd_at(c2, lane)]);
        __syncwarp();
    }
    const int o = lane & ~7;
    T w[8];
    inv8_column(lane & 7, [&](int i, int q) { return S[pd_at(o + q, o + i)]; },
                [&](int i) { return rdiag[o + i]; }, w);
#pragma unroll
    for (int i = 0; i < 8; i++)
        if (lane < NB) W8[lane * 8 + i] = w[i];
    return bad;
}

// Strips of 16 rows x 8 columns on m16n8k8 (mma8: DMMA, or split TF32), for
// kernels with many strips per warp: accumulator x[0] (g, 2t), x[1] (g, 2t+1),
// x[2] (g+8, 2t), x[3] (g+8, 2t+1), again the next A operand as it stands.
// d <- x B, formed from zero: the tensor cores truncate what they add to an
// FP32 accumulator, so products are not added to larger values there.
template <typename T, int SPLIT>
__device__ __forceinline__ void strip16_product(T (&d)[4], const T (&x)[4], T b0, T b1)
{
    const T a[4] = {x[0], x[2], x[1], x[3]};
    const T b[2] = {b0, b1};
#pragma unroll
    for (int e = 0; e < 4; e++) d[e] = T(0);
    mma8<SPLIT>(d, a, b);
}

// y <- y - x B
template <typename T, int SPLIT>
__device__ __forceinline__ void strip16_subtract(T (&y)[4], const T (&x)[4], T b0, T b1)
{
    T d[4];
    strip16_product<T, SPLIT>(d, x, b0, b1);
#pragma unroll
    for (int e = 0; e < 4; e++) y[e] -= d[e];
}

// d <- x B for a triangular B (an inverse in W8) whose diagonal entries of this
// lane's columns are w0 = B(2t, 2t) and w1 = B(2t+1, 2t+1).  FP32: the tensor
// cores truncate a sum at its own size, which here is the result's, and all
// in one direction; the diagonal's terms, the largest in general, stay out of
// it and are added rounded.
template <typename T, int SPLIT>
__device__ __forceinline__ void strip16_inverse(T (&d)[4], const T (&x)[4], T b0, T b1, T w0,
                                                T w1)
{
    if (sizeof(T) == 8) {
        strip16_product<T, SPLIT>(d, x, b0, b1);
        return;
    }
    const int g = (threadIdx.x >> 2) & 7, t = threadIdx.x & 3;
    strip16_product<T, SPLIT>(d, x, g == 2 * t ? T(0) : b0, g == 2 * t + 1 ? T(0) : b1);
#pragma unroll
    for (int e = 0; e < 4; e++) d[e] = fma(x[e], e & 1 ? w1 : w0, d[e]);
}

// strip_solve32 for 16 rows and NB columns
template <typename T, int SPLIT, int NB>
__device__ __forceinline__ void strip16_solve(T (&y)[NB / 8][4], const T *D, const T *W8)
{
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int q = 0; q < NB / 8; q++) {
        T x[4];
        const T *w = W8 + 64 * q;
        strip16_inverse<T, SPLIT>(x, y[q], w[16 * t + g], w[16 * t + 8 + g], w[18 * t],
                                  w[18 * t + 9]);
#pragma unroll
        for (int f = q + 1; f < NB / 8; f++)
            strip16_subtract<T, SPLIT>(y[f], x, D[pd_at(8 * q + 2 * t, 8 * f + g)],
                                       D[pd_at(8 * q + 2 * t + 1, 8 * f + g)]);
#pragma unroll
        for (int e = 0; e < 4; e++) y[q][e] = x[e];
    }
}

}  // namespace
