// batched.cu -- thousands of independent SPD systems of uneven size in one
// persistent launch: Cholesky factor (potrf), solve (potrs, one right-hand
// side) and their adjoints.  No reference counterpart (PLASMA factors one
// matrix at a time); the per-matrix algorithm is the reference's blocked
// right-looking Cholesky (compute/pzpotrf.c:37-80 at the scale of one CTA).
//
// Layout: matrix i is column-major n_i x n_i (ld = n_i) at A + off_a[i];
// its right-hand side / solution at B + off_b[i].  A plan (host side) sorts
// the matrices by decreasing size (longest processing time first) and picks
// the block width NB of each size bucket from a measured table.
//
// Persistent CTAs of 256 threads (one per SM in FP64, two in FP32, whose
// panels are half the size) take the next matrix from an atomic counter until
// the list is exhausted, so large and small matrices balance across SMs.  Per
// matrix, for each block column j0:
//   (a) one warp factors the NB x NB diagonal block (blk_factor: eight
//       columns at a time in registers; LAPACK's info on a non-positive or
//       NaN pivot, and the matrix is abandoned);
//   (b) the rows below solve x D^T = a in strips of 16 on the tensor cores
//       (strip16_solve); the panel is kept in shared memory;
//   (c) the trailing lower triangle is updated, A22 -= P P^T, with DMMA
//       (FP64) or the three-product TF32 split (FP32, FP32-accurate), C read
//       and written in global memory (L2): the next diagonal block first, an
//       8-column piece per warp, then warp 0 factors it while the other warps
//       update the rest in tasks of 16 x 32 from a counter.  The other warp
//       of warp 0's scheduler waits for the factor before it joins: FP64
//       tensor work on the same scheduler doubles the time of a pivot.
// 4096 systems, n in [16, 512], FP64 factor and solve: 8.1 ms a call with the
// diagonal blocks factored and inverted by one warp, 6.6 ms in this form; the
// FP32 gradient of 1024 systems 15.4 -> 5.3 ms.
// The solve follows in the same CTA while the factor is in L2: forward by
// block (diagonal block by one warp, the rows below by all threads),
// backward by block (column dot products by warps, then the diagonal block).
#include "common.cuh"
#include "mma.cuh"
#include "f64_blocks.cuh"

#include <stdlib.h>
#include <string.h>

namespace {

constexpr int BT = 256;               // threads per CTA
constexpr int NMAX = 512;             // largest matrix of the batched path
constexpr int NBMAXB = 32;            // largest block width

template <typename T> constexpr int ps_ld() { return NBMAXB + Pad<T>::v; }
// shared memory: panel [NMAX][ps_ld], three blocks of 32 x 33 (two diagonal
// blocks in turn and the copy of the one being factored; the adjoints use
// them with a stride of 33), two sets of 8 x 8 inverses, a vector of NMAX, 32
// reciprocal pivots
constexpr int BLK_ELEMS = NBMAXB * (NBMAXB + 1);
template <typename T> constexpr int batched_smem()
{
    return (NMAX * ps_ld<T>() + 3 * BLK_ELEMS + 2 * 8 * NBMAXB + NMAX + NBMAXB) * (int)sizeof(T);
}
template <typename T> constexpr int batched_ctas() { return sizeof(T) == 4 ? 2 : 1; }

template <int V> struct IntC { static constexpr int value = V; };

enum { OP_POSV = 0, OP_POTRF = 1, OP_POTRS = 2, OP_POTRF_ADJ = 3, OP_POTRS_ADJ = 4 };

struct BatchArgs {
    int batch;
    const int *n;               // [batch]
    const long long *off_a;     // [batch] element offsets of the matrices
    const long long *off_b;     // [batch] element offsets of the vectors
    const int *order;           // processing order (largest first)
    const unsigned char *nbsel; // [batch] block width of each matrix (16 or 32)
    void *A;                    // matrices (the factor for solves and adjoints)
    void *B;                    // right-hand sides / solutions (X for the adjoint)
    void *C;                    // Xbar -> Bbar (potrs adjoint)
    void *D;                    // Lbar (adjoints)
    int *info;                  // [batch] (factorisations)
    int *counter;               // zeroed before the launch
    int op;
};

// ------------------------------------------------------------------ factor
// y <- D^-1 y for the right-hand side entries ys[0 .. jb-1] by one warp, with
// the inverses of D's 8 x 8 diagonal blocks: lane i holds y_i.
template <typename T, int NB>
__device__ __forceinline__ void forward_block(T *ys, int jb, const T *D, const T *W8)
{
    const int lane = threadIdx.x & 31;
    T y = lane < jb ? ys[lane] : T(0);
#pragma unroll
    for (int q = 0; q < NB / 8; q++) {
        const int i = lane - 8 * q;
        T x[8], nv = T(0);
#pragma unroll
        for (int k = 0; k < 8; k++) x[k] = __shfl_sync(0xffffffffu, y, 8 * q + k);
#pragma unroll
        for (int k = 0; k < 8; k++) nv = fma(W8[(8 * q + k) * 8 + (i & 7)], x[k], nv);
        if (i >= 0 && i < 8) y = nv;
#pragma unroll
        for (int k = 0; k < 8; k++) x[k] = __shfl_sync(0xffffffffu, y, 8 * q + k);
        if (i >= 8) {
#pragma unroll
            for (int k = 0; k < 8; k++) y = fma(-D[pd_at(8 * q + k, lane)], x[k], y);
        }
    }
    if (lane < jb) ys[lane] = y;
}

// See the header.  With ys (posv: the right-hand side in shared memory) the
// forward sweep L y = b runs along, y_j from the diagonal block by the last
// warp and the rows below from the panel, so the solve afterwards is the
// backward sweep alone.  task: a counter in shared memory.
template <typename T, int SPLIT, int NB>
__device__ int factor_one(T *A, int n, T *Ps, T *D0, T *D1, T *Dn, T *W8, T *rdiag, int *flag,
                          int *task, T *ys)
{
    constexpr int PLD = ps_ld<T>();
    constexpr int WARPS = BT / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    // warp 0: the block at D, of which Dn holds a copy
    auto factor = [&](T *D, T *W) {
        int bad = 0;
        if (!__all_sync(0xffffffffu, blk_factor<T, SPLIT, NB>(D, W)))
            bad = blk_factor_any<T, NB>(D, W, Dn, rdiag);
        if (lane == 0) *flag = bad;
    };
    // the first diagonal block, padded with the identity
    for (int e = tid; e < NB * 32; e += BT) {
        const int r = e % 32, c = e / 32;
        const T v = r < min(NB, n) && c < n ? (r >= c ? A[(size_t)c * n + r] : T(0))
                                            : (r == c ? T(1) : T(0));
        D0[pd_at(c, r)] = v;
        Dn[pd_at(c, r)] = v;
    }
    __syncthreads();
    if (warp == 0) factor(D0, W8);
    __syncthreads();
    for (int j0 = 0, cur = 0; j0 < n; j0 += NB, cur ^= 1) {
        const int jb = min(NB, n - j0);
        const int m2 = n - j0 - jb;
        const int bad = *flag;
        if (bad) return j0 + bad;
        const T *D = cur ? D1 : D0;
        const T *W = W8 + cur * 8 * NBMAXB;
        T *Dnext = cur ? D0 : D1, *Wnext = W8 + (cur ^ 1) * 8 * NBMAXB;
        if (tid == 0) *task = 0;
        if (ys != nullptr && warp == WARPS - 1) forward_block<T, NB>(ys + j0, jb, D, W);
        for (int e = tid; e < jb * 32; e += BT) {
            const int r = e % 32, c = e / 32;
            if (r >= c && r < jb) A[(size_t)(j0 + c) * n + j0 + r] = D[pd_at(c, r)];
        }
        // (b) the panel below (there is one only below a full diagonal
        // block), to A and to Ps
        {
            T *A21 = A + (size_t)j0 * n + (j0 + jb);
            for (int r0 = warp * 16; r0 < m2; r0 += 16 * WARPS) {
                T y[NB / 8][4];
#pragma unroll
                for (int q = 0; q < NB / 8; q++)
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        const int r = r0 + g + 8 * (e >> 1), c = 8 * q + 2 * t + (e & 1);
                        y[q][e] = r < m2 ? A21[(size_t)c * n + r] : T(0);
                    }
                strip16_solve<T, SPLIT, NB>(y, D, W);
#pragma unroll
                for (int q = 0; q < NB / 8; q++)
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        const int r = r0 + g + 8 * (e >> 1), c = 8 * q + 2 * t + (e & 1);
                        if (r < m2) {
                            A21[(size_t)c * n + r] = y[q][e];
                            Ps[r * PLD + c] = y[q][e];
                        }
                    }
            }
        }
        __syncthreads();
        if (m2 == 0) break;
        T *C = A + (size_t)(j0 + jb) * n + (j0 + jb);   // A22(0,0)
        // C(r0 .. r0+15, c0 .. c0+8 NF-1) - P P^T, handed to put(r, c, value)
        auto block = [&](int r0, int c0, auto nf, auto put) {
            constexpr int NF = decltype(nf)::value;
            T cv[NF][4], acc[NF][4];
            const int ra = r0 + g;
#pragma unroll
            for (int f = 0; f < NF; f++)
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int r = ra + 8 * (e >> 1), c = c0 + 8 * f + 2 * t + (e & 1);
                    cv[f][e] = r < m2 && c < m2 && r >= c ? C[(size_t)c * n + r] : T(0);
                    acc[f][e] = T(0);
                }
#pragma unroll
            for (int k8 = 0; k8 < NB; k8 += 8) {
                T bf[NF][2], af[4];
#pragma unroll
                for (int f = 0; f < NF; f++) {
                    const int cr = c0 + 8 * f + g;
                    bf[f][0] = cr < m2 ? Ps[cr * PLD + k8 + t] : T(0);
                    bf[f][1] = cr < m2 ? Ps[cr * PLD + k8 + t + 4] : T(0);
                }
                af[0] = ra < m2 ? Ps[ra * PLD + k8 + t] : T(0);
                af[1] = ra + 8 < m2 ? Ps[(ra + 8) * PLD + k8 + t] : T(0);
                af[2] = ra < m2 ? Ps[ra * PLD + k8 + t + 4] : T(0);
                af[3] = ra + 8 < m2 ? Ps[(ra + 8) * PLD + k8 + t + 4] : T(0);
#pragma unroll
                for (int f = 0; f < NF; f++) mma8<SPLIT>(acc[f], af, bf[f]);
            }
#pragma unroll
            for (int f = 0; f < NF; f++)
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int r = ra + 8 * (e >> 1), c = c0 + 8 * f + 2 * t + (e & 1);
                    put(r, c, cv[f][e] - acc[f][e]);
                }
        };
        // (c) the next diagonal block, an 8-column piece per warp, padded
        {
            const int jn = min(NB, m2);
            if (warp < NB / 16 * (NB / 8))
                block(16 * (warp / (NB / 8)), 8 * (warp % (NB / 8)), IntC<1>{},
                      [&](int r, int c, T v) {
                          v = r < jn && c < jn ? (r >= c ? v : T(0)) : (r == c ? T(1) : T(0));
                          Dnext[pd_at(c, r)] = v;
                          Dn[pd_at(c, r)] = v;
                      });
        }
        __syncthreads();
        if (warp == 0) {
            factor(Dnext, Wnext);
        } else if (ys != nullptr) {
            // y_below -= P y_j
            for (int r = tid - 32; r < m2; r += BT - 32) {
                T s0 = T(0), s1 = T(0);
#pragma unroll
                for (int c = 0; c < NB; c += 2) {
                    s0 += Ps[r * PLD + c] * ys[j0 + c];
                    s1 += Ps[r * PLD + c + 1] * ys[j0 + c + 1];
                }
                ys[j0 + jb + r] -= s0 + s1;
            }
        }
        if ((warp & 3) == 0) asm volatile("bar.sync 1, %0;" :: "n"(BT / 4) : "memory");
        // the rest of the lower triangle: blocks (bi, bj) of 16 x 32, bi >=
        // 2 bj, column by column, without the NB / 16 of the diagonal block
        const int nrb = (m2 + 15) / 16;
        for (;;) {
            int q = 0;
            if (lane == 0) q = atomicAdd(task, 1);
            q = __shfl_sync(0xffffffffu, q, 0) + NB / 16;
            int bj = 0;
            while (2 * bj < nrb && q >= nrb - 2 * bj) { q -= nrb - 2 * bj; bj++; }
            if (2 * bj >= nrb) break;
            block(16 * (2 * bj + q), 32 * bj, IntC<4>{}, [&](int r, int c, T v) {
                if (r < m2 && c < m2 && r >= c) C[(size_t)c * n + r] = v;
            });
        }
        __syncthreads();
    }
    return 0;
}

// ------------------------------------------------------------------- solve
// b <- A^-1 b with the factor L in the lower triangle of A (n x n, ld n).
// Each 32 x 32 diagonal block is first staged in shared memory (one parallel
// load), so the warp's substitution reads shared memory only.
template <typename T>
__device__ void solve_one(const T *A, int n, T *b, T *Ys, T *Db, T *Dr, bool forward_done = false)
{
    constexpr int NB = 32, DLD = NB + 1;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (!forward_done)
        for (int i = tid; i < n; i += BT) Ys[i] = b[i];
    // forward: L y = b (unless the factorization ran it: Ys holds y)
    for (int j0 = 0; j0 < n && !forward_done; j0 += NB) {
        const int jb = min(NB, n - j0);
        for (int e = tid; e < NB * NB; e += BT) {
            const int r = e % NB, c = e / NB;
            Db[c * DLD + r] = (r < jb && c < jb && r >= c) ? A[(size_t)(j0 + c) * n + j0 + r] : T(0);
        }
        if (tid < jb) Dr[tid] = T(1) / A[(size_t)(j0 + tid) * n + j0 + tid];
        __syncthreads();
        if (warp == 0) {
            T y = lane < jb ? Ys[j0 + lane] : T(0);
            for (int c = 0; c < jb; c++) {
                if (lane == c) y = y * Dr[c];
                const T yc = __shfl_sync(0xffffffffu, y, c);
                if (lane > c && lane < jb) y -= Db[c * DLD + lane] * yc;
            }
            if (lane < jb) Ys[j0 + lane] = y;
        }
        __syncthreads();
        for (int r = j0 + jb + tid; r < n; r += BT) {
            T s = Ys[r];
#pragma unroll 8
            for (int c = 0; c < jb; c++) s -= A[(size_t)(j0 + c) * n + r] * Ys[j0 + c];
            Ys[r] = s;
        }
        __syncthreads();
    }
    // backward: L^T x = y
    for (int j0 = ((n - 1) / NB) * NB; j0 >= 0; j0 -= NB) {
        const int jb = min(NB, n - j0);
        for (int e = tid; e < NB * NB; e += BT) {
            const int r = e % NB, c = e / NB;
            Db[c * DLD + r] = (r < jb && c < jb && r >= c) ? A[(size_t)(j0 + c) * n + j0 + r] : T(0);
        }
        if (tid < jb) Dr[tid] = T(1) / A[(size_t)(j0 + tid) * n + j0 + tid];
        // a warp takes its four columns of the block at once (their loads
        // overlap)
        {
            constexpr int NC = NB / (BT / 32);
            T s[NC];
#pragma unroll
            for (int q = 0; q < NC; q++) s[q] = T(0);
#pragma unroll 4
            for (int i = j0 + jb + lane; i < n; i += 32) {
                const T y = Ys[i];
#pragma unroll
                for (int q = 0; q < NC; q++) {
                    const int c = warp + q * (BT / 32);
                    if (c < jb) s[q] += A[(size_t)(j0 + c) * n + i] * y;
                }
            }
#pragma unroll
            for (int q = 0; q < NC; q++)
#pragma unroll
                for (int off = 16; off > 0; off >>= 1)
                    s[q] += __shfl_xor_sync(0xffffffffu, s[q], off);
            if (lane < NC && warp + lane * (BT / 32) < jb) {
                T v = s[0];
#pragma unroll
                for (int q = 1; q < NC; q++) v = lane == q ? s[q] : v;
                Ys[j0 + warp + lane * (BT / 32)] -= v;
            }
        }
        __syncthreads();
        if (warp == 0) {
            T x = lane < jb ? Ys[j0 + lane] : T(0);
            for (int c = jb - 1; c >= 0; c--) {
                if (lane == c) x = x * Dr[c];
                const T xc = __shfl_sync(0xffffffffu, x, c);
                if (lane < c) x -= Db[lane * DLD + c] * xc;
            }
            if (lane < jb) Ys[j0 + lane] = x;
        }
        __syncthreads();
    }
    for (int i = tid; i < n; i += BT) b[i] = Ys[i];
    __syncthreads();
}

// ------------------------------------------------------------ potrs adjoint
// xbar <- A^-1 xbar (= bbar); Lbar -= tril(bbar (L^T x)^T + x (L^T bbar)^T)
template <typename T>
__device__ void solve_adjoint_one(const T *Lf, int n, const T *x, T *xbar, T *Lbar, T *Ys,
                                  T *U, T *Db, T *Dr)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    solve_one<T>(Lf, n, xbar, Ys, Db, Dr);         // Ys keeps bbar
    T *u1 = U, *u2 = U + NMAX;                     // L^T x, L^T bbar
    for (int c = warp; c < n; c += BT / 32) {
        T s1 = T(0), s2 = T(0);
        for (int r = c + lane; r < n; r += 32) {
            const T l = Lf[(size_t)c * n + r];
            s1 += l * x[r];
            s2 += l * Ys[r];
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            s1 += __shfl_xor_sync(0xffffffffu, s1, off);
            s2 += __shfl_xor_sync(0xffffffffu, s2, off);
        }
        if (lane == 0) { u1[c] = s1; u2[c] = s2; }
    }
    __syncthreads();
    for (int c = warp; c < n; c += BT / 32)
        for (int r = c + lane; r < n; r += 32)
            Lbar[(size_t)c * n + r] -= Ys[r] * u1[c] + x[r] * u2[c];
    __syncthreads();
}

// ------------------------------------------------------------ potrf adjoint
// Blocked reverse mode of the Cholesky factor, walking block columns from the
// last to the first and recomputing from the factor L (lower triangle of Lf):
//   Cbar <- Cbar D^-1;  Bbar -= Cbar R;  Dbar <- tril(Dbar) - tril(Cbar^T C);
//   Dbar <- unblocked reverse of the diagonal block;
//   Rbar -= Cbar^T B + (Dbar + Dbar^T) R
// (R, D, B, C: the blocks left of, on, below-left of and below the diagonal
// block; bars the same blocks of Lbar).  The result Abar is lower triangular
// and the symmetric cotangent is (Abar + Abar^T)/2 with Abar's own diagonal,
// written into both triangles of Lbar at the end.
// FP32 sums leave the tensor cores every 8 terms (add_up): what these add to an
// accumulator is truncated, and the bias would grow with the length.
template <typename T>
__device__ __forceinline__ void add_up(T (&sum)[4], T (&acc)[4])
{
#pragma unroll
    for (int e = 0; e < 4; e++) {
        sum[e] += acc[e];
        acc[e] = T(0);
    }
}

// The products (the four block updates) run on the tensor cores (mma8): a
// thread per output entry made them 90% of the adjoint's time.  Warp 0 runs
// the unblocked reverse beside the update of Bbar by the others.
template <typename T, int SPLIT>
__device__ void factor_adjoint_one(const T *Lf, int n, T *Lb, T *Cs, T *Ds, T *Dbs, T *Dp, T *W8)
{
    constexpr int NB = 32, CLD = NB + 1;
    constexpr int WARPS = BT / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    for (int k = n; k > 0; k -= NB) {
        const int j = max(0, k - NB), jb = k - j, m2 = n - k;   // j > 0 only if jb = NB
        for (int e = tid; e < NB * NB; e += BT) {
            const int r = e % NB, c = e / NB;
            const bool in = r < jb && c < jb && r >= c;
            const T v = in ? Lf[(size_t)(j + c) * n + j + r] : T(0);
            Ds[c * CLD + r] = v;
            Dp[pd_at(c, r)] = r >= jb || c >= jb ? (r == c ? T(1) : T(0)) : v;
            Dbs[c * CLD + r] = in ? Lb[(size_t)(j + c) * n + j + r] : T(0);
        }
        __syncthreads();
        // (1) Cbar <- Cbar D^-1 in strips of 16 rows, with the inverses of D's
        // 8 x 8 diagonal blocks
        if (m2 > 0) {
            if (warp == 0) {
                const int o = lane & ~7;
                T w[8];
                inv8_column(lane & 7, [&](int i, int q) { return Dp[pd_at(o + q, o + i)]; },
                            [&](int i) { return T(1) / Dp[pd_at(o + i, o + i)]; }, w);
#pragma unroll
                for (int i = 0; i < 8; i++) W8[lane * 8 + i] = w[i];
            }
            __syncthreads();
            for (int r0 = 16 * warp; r0 < m2; r0 += 16 * WARPS) {
                T y[NB / 8][4];
#pragma unroll
                for (int q = 0; q < NB / 8; q++)
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        const int r = r0 + g + 8 * (e >> 1), c = 8 * q + 2 * t + (e & 1);
                        y[q][e] = r < m2 && c < jb ? Lb[(size_t)(j + c) * n + k + r] : T(0);
                    }
#pragma unroll
                for (int q = NB / 8 - 1; q >= 0; q--) {
                    T x[4];
                    const T *w = W8 + 64 * q;
                    strip16_inverse<T, SPLIT>(x, y[q], w[8 * g + 2 * t], w[8 * g + 2 * t + 1],
                                              w[18 * t], w[18 * t + 9]);
#pragma unroll
                    for (int f = 0; f < q; f++)
                        strip16_subtract<T, SPLIT>(y[f], x, Dp[pd_at(8 * f + g, 8 * q + 2 * t)],
                                                   Dp[pd_at(8 * f + g, 8 * q + 2 * t + 1)]);
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        const int r = r0 + g + 8 * (e >> 1), c = 8 * q + 2 * t + (e & 1);
                        if (r < m2) {
                            Cs[r * CLD + c] = x[e];
                            if (c < jb) Lb[(size_t)(j + c) * n + k + r] = x[e];
                        }
                    }
                }
            }
            __syncthreads();
            // (3) Dbar -= tril(Cbar^T C): a 16 x 8 piece per warp
            {
                const int i0 = 16 * (warp >> 2), c0 = 8 * (warp & 3);
                const T *Cc = Lf + (size_t)(j + min(c0 + g, jb - 1)) * n + k;
                T acc[4] = {T(0), T(0), T(0), T(0)}, sum[4] = {T(0), T(0), T(0), T(0)};
#pragma unroll 4
                for (int r = 0; r < m2; r += 8) {
                    const int ra = r + t, rb = ra + 4;
                    const T af[4] = {ra < m2 ? Cs[ra * CLD + i0 + g] : T(0),
                                     ra < m2 ? Cs[ra * CLD + i0 + g + 8] : T(0),
                                     rb < m2 ? Cs[rb * CLD + i0 + g] : T(0),
                                     rb < m2 ? Cs[rb * CLD + i0 + g + 8] : T(0)};
                    const T bf[2] = {ra < m2 ? Cc[ra] : T(0), rb < m2 ? Cc[rb] : T(0)};
                    mma8<SPLIT>(acc, af, bf);
                    if (sizeof(T) == 4) add_up<T>(sum, acc);
                }
                add_up<T>(sum, acc);
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int i = i0 + g + 8 * (e >> 1), c = c0 + 2 * t + (e & 1);
                    if (i >= c && i < jb && c < jb) Dbs[c * CLD + i] -= sum[e];
                }
            }
            __syncthreads();
        }
        // (2) Bbar -= Cbar R (rows k.., columns 0..j): per task 32 columns,
        // whose R stays in registers, and 64 rows; the warps beside warp 0
        if (warp > 0 && j > 0 && m2 > 0) {
            const int ncb = (j + 31) / 32, nrg = (m2 + 63) / 64;
            for (int task = warp - 1; task < ncb * nrg; task += WARPS - 1) {
                const int c0 = 32 * (task % ncb), rg = 64 * (task / ncb);
                T bf[4][NB / 8][2];
#pragma unroll
                for (int f = 0; f < 4; f++) {
                    const int col = c0 + 8 * f + g;
                    const T *Rc = Lf + (size_t)col * n + j;
#pragma unroll
                    for (int k8 = 0; k8 < NB; k8 += 8) {
                        bf[f][k8 / 8][0] = col < j ? Rc[k8 + t] : T(0);
                        bf[f][k8 / 8][1] = col < j ? Rc[k8 + t + 4] : T(0);
                    }
                }
                for (int r0 = rg; r0 < min(m2, rg + 64); r0 += 16) {
                    const int ra = r0 + g;
                    T acc[4][4];
#pragma unroll
                    for (int f = 0; f < 4; f++)
#pragma unroll
                        for (int e = 0; e < 4; e++) acc[f][e] = T(0);
#pragma unroll
                    for (int k8 = 0; k8 < NB; k8 += 8) {
                        const T af[4] = {ra < m2 ? Cs[ra * CLD + k8 + t] : T(0),
                                         ra + 8 < m2 ? Cs[(ra + 8) * CLD + k8 + t] : T(0),
                                         ra < m2 ? Cs[ra * CLD + k8 + t + 4] : T(0),
                                         ra + 8 < m2 ? Cs[(ra + 8) * CLD + k8 + t + 4] : T(0)};
#pragma unroll
                        for (int f = 0; f < 4; f++) {
                            if (sizeof(T) == 8) {
                                mma8<SPLIT>(acc[f], af, bf[f][k8 / 8]);
                            } else {
                                T d[4] = {T(0), T(0), T(0), T(0)};
                                mma8<SPLIT>(d, af, bf[f][k8 / 8]);
                                add_up<T>(acc[f], d);
                            }
                        }
                    }
#pragma unroll
                    for (int f = 0; f < 4; f++)
#pragma unroll
                        for (int e = 0; e < 4; e++) {
                            const int r = ra + 8 * (e >> 1), col = c0 + 8 * f + 2 * t + (e & 1);
                            if (r < m2 && col < j) Lb[(size_t)col * n + k + r] -= acc[f][e];
                        }
                }
            }
        }
        // (4) unblocked reverse on the diagonal block, one warp, lane = column
        if (warp == 0) {
            for (int jj = jb - 1; jj >= 0; jj--) {
                const T djj = Ds[jj * CLD + jj];
                T p = (lane > jj && lane < jb) ? Ds[jj * CLD + lane] * Dbs[jj * CLD + lane] : T(0);
#pragma unroll
                for (int off = 16; off > 0; off >>= 1) p += __shfl_xor_sync(0xffffffffu, p, off);
                if (lane == 0) Dbs[jj * CLD + jj] -= p / djj;
                __syncwarp();
                if (lane >= jj && lane < jb) Dbs[jj * CLD + lane] /= djj;
                __syncwarp();
                if (lane < jj) {
                    T s = T(0);
                    for (int r = jj; r < jb; r++) s += Dbs[jj * CLD + r] * Ds[lane * CLD + r];
                    Dbs[lane * CLD + jj] -= s;
                    const T ljc = Ds[lane * CLD + jj];
                    for (int r = jj + 1; r < jb; r++) Dbs[lane * CLD + r] -= Dbs[jj * CLD + r] * ljc;
                }
                __syncwarp();
                if (lane == 0) Dbs[jj * CLD + jj] *= T(0.5);
                __syncwarp();
            }
        }
        __syncthreads();
        // (5) Rbar -= Cbar^T B + (Dbar + Dbar^T) R (rows j..k, columns 0..j),
        // 16 columns per task
        for (int c0 = 16 * warp; c0 < j; c0 += 16 * WARPS) {
            T acc[2][2][4], sum[2][2][4];
#pragma unroll
            for (int h = 0; h < 2; h++)
#pragma unroll
                for (int f = 0; f < 2; f++)
#pragma unroll
                    for (int e = 0; e < 4; e++) acc[h][f][e] = sum[h][f][e] = T(0);
            auto add_all = [&]() {
#pragma unroll
                for (int h = 0; h < 2; h++)
#pragma unroll
                    for (int f = 0; f < 2; f++) add_up<T>(sum[h][f], acc[h][f]);
            };
            const T *Lc[2];
            bool cv[2];
#pragma unroll
            for (int f = 0; f < 2; f++) {
                cv[f] = c0 + 8 * f + g < j;
                Lc[f] = Lf + (size_t)min(c0 + 8 * f + g, j - 1) * n;
            }
#pragma unroll
            for (int k8 = 0; k8 < NB; k8 += 8) {
                T bf[2][2];
#pragma unroll
                for (int f = 0; f < 2; f++) {
                    bf[f][0] = cv[f] ? Lc[f][j + k8 + t] : T(0);
                    bf[f][1] = cv[f] ? Lc[f][j + k8 + t + 4] : T(0);
                }
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    T af[4];
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        const int i = 16 * h + g + 8 * (e & 1), c = k8 + t + 4 * (e >> 1);
                        af[e] = Dbs[c * CLD + i] + Dbs[i * CLD + c];
                    }
#pragma unroll
                    for (int f = 0; f < 2; f++) mma8<SPLIT>(acc[h][f], af, bf[f]);
                }
                if (sizeof(T) == 4) add_all();
            }
            if (sizeof(T) == 8) add_all();
#pragma unroll 2
            for (int r = 0; r < m2; r += 8) {
                const int ra = r + t, rb = ra + 4;
                T bf[2][2];
#pragma unroll
                for (int f = 0; f < 2; f++) {
                    bf[f][0] = cv[f] && ra < m2 ? Lc[f][k + ra] : T(0);
                    bf[f][1] = cv[f] && rb < m2 ? Lc[f][k + rb] : T(0);
                }
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int i = 16 * h + g;
                    const T af[4] = {ra < m2 ? Cs[ra * CLD + i] : T(0),
                                     ra < m2 ? Cs[ra * CLD + i + 8] : T(0),
                                     rb < m2 ? Cs[rb * CLD + i] : T(0),
                                     rb < m2 ? Cs[rb * CLD + i + 8] : T(0)};
#pragma unroll
                    for (int f = 0; f < 2; f++) mma8<SPLIT>(acc[h][f], af, bf[f]);
                }
                if (sizeof(T) == 4) add_all();
            }
            add_all();
#pragma unroll
            for (int h = 0; h < 2; h++)
#pragma unroll
                for (int f = 0; f < 2; f++)
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        const int i = 16 * h + g + 8 * (e >> 1), col = c0 + 8 * f + 2 * t + (e & 1);
                        if (col < j) Lb[(size_t)col * n + j + i] -= sum[h][f][e];
                    }
        }
        for (int e = tid; e < jb * jb; e += BT) {
            const int r = e % jb, c = e / jb;
            if (r >= c) Lb[(size_t)(j + c) * n + j + r] = Dbs[c * CLD + r];
        }
        __syncthreads();
    }
    // symmetric cotangent in both triangles
    for (size_t e = tid; e < (size_t)n * n; e += BT) {
        const int r = (int)(e % n), c = (int)(e / n);
        if (r > c) {
            const T v = T(0.5) * Lb[(size_t)c * n + r];
            Lb[(size_t)c * n + r] = v;
            Lb[(size_t)r * n + c] = v;
        }
    }
    __syncthreads();
}

// ------------------------------------------------------------------ kernel
template <typename T, int SPLIT>
__global__ void __launch_bounds__(BT, batched_ctas<T>())
k_batched(BatchArgs a)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *Ps = reinterpret_cast<T *>(smem_raw);        // [NMAX][ps_ld]
    T *Ds = Ps + NMAX * ps_ld<T>();                 // [32][33]
    T *D2 = Ds + BLK_ELEMS;                         // [32][33]
    T *Dn = D2 + BLK_ELEMS;                         // [32][33]
    T *W8 = Dn + BLK_ELEMS;                         // [2][32][8]
    T *Ys = W8 + 2 * 8 * NBMAXB;                    // [NMAX]
    T *rdiag = Ys + NMAX;                           // [32]
    __shared__ int idx_s, flag_s, task_s;
    const int tid = threadIdx.x;
    for (;;) {
        if (tid == 0) idx_s = atomicAdd(a.counter, 1);
        __syncthreads();
        const int idx = idx_s;
        __syncthreads();
        if (idx >= a.batch) break;
        const int m = a.order[idx];
        const int n = a.n[m];
        T *A = (T *)a.A + a.off_a[m];
        if (a.op == OP_POSV || a.op == OP_POTRF) {
            T *b = (T *)a.B + a.off_b[m];
            T *ys = nullptr;
            if (a.op == OP_POSV) {
                for (int i = tid; i < n; i += BT) Ys[i] = b[i];
                __syncthreads();
                ys = Ys;
            }
            const int info = a.nbsel[m] == 16
                                 ? factor_one<T, SPLIT, 16>(A, n, Ps, Ds, D2, Dn, W8, rdiag, &flag_s, &task_s, ys)
                                 : factor_one<T, SPLIT, 32>(A, n, Ps, Ds, D2, Dn, W8, rdiag, &flag_s, &task_s, ys);
            if (tid == 0) a.info[m] = info;
            __syncthreads();
            if (info == 0 && a.op == OP_POSV) solve_one<T>(A, n, b, Ys, D2, rdiag, true);
        } else if (a.op == OP_POTRS) {
            solve_one<T>(A, n, (T *)a.B + a.off_b[m], Ys, D2, rdiag);
        } else if (a.op == OP_POTRS_ADJ) {
            solve_adjoint_one<T>(A, n, (const T *)a.B + a.off_b[m], (T *)a.C + a.off_b[m],
                                 (T *)a.D + a.off_a[m], Ys, Ps, D2, rdiag);
        } else {
            factor_adjoint_one<T, SPLIT>(A, n, (T *)a.D + a.off_a[m], Ps, Ds, D2, Dn, W8);
        }
    }
}

template <typename T, int SPLIT>
void launch_batched(cudaStream_t s, const BatchArgs &a, int grid)
{
    static unsigned long long attr = 0;
    if (plasma_first_on_device(&attr)) {
        cudaFuncSetAttribute(k_batched<T, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             batched_smem<T>());
    }
    k_batched<T, SPLIT><<<grid, BT, batched_smem<T>(), s>>>(a);
}

}  // namespace

// ------------------------------------------------------------------- plans
struct plasma_batch_s {
    int batch;
    int precision;
    int *d_n;
    long long *d_off_a, *d_off_b;
    int *d_order;
    unsigned char *d_nbsel;
    int *d_counter;
    long long *h_off_a, *h_off_b;
    long long elems_a, elems_b;
    int device;
    int graph;                  // replay launches from cached CUDA graphs
    cudaGraphExec_t exec[5];    // one per operation
    void *g_ptr[5][5];          // the pointers each graph was captured with
};

static void batch_free(plasma_batch_t *p)
{
    if (p == NULL) return;
    for (int i = 0; i < 5; i++)
        if (p->exec[i]) cudaGraphExecDestroy(p->exec[i]);
    cudaFree(p->d_n);
    cudaFree(p->d_off_a);
    cudaFree(p->d_off_b);
    cudaFree(p->d_order);
    cudaFree(p->d_nbsel);
    cudaFree(p->d_counter);
    free(p->h_off_a);
    free(p->h_off_b);
    free(p);
}

extern "C" int plasma_batch_create(plasma_enum_t precision, int batch, const int *n,
                                   plasma_batch_t **plan)
{
    plasma_context_t *plasma = plasma_context_self();
    if (plasma == NULL) return PlasmaErrorNotInitialized;
    if (precision != PlasmaRealDouble && precision != PlasmaRealFloat) return -1;
    if (batch < 0) return -2;
    if (n == NULL && batch > 0) return -3;
    if (plan == NULL) return -4;
    for (int i = 0; i < batch; i++)
        if (n[i] < 0 || n[i] > NMAX) {
            plasma_error("plasma_batch_create: matrix orders must lie in [0, 512]");
            return -3;
        }
    if (plasma->device < 0) return PlasmaErrorEnvironment;
    plasma_batch_t *p = (plasma_batch_t *)calloc(1, sizeof(plasma_batch_t));
    if (p == NULL) return PlasmaErrorOutOfMemory;
    p->batch = batch;
    p->precision = precision;
    p->device = plasma->device;
    const int cnt = batch > 0 ? batch : 1;
    p->h_off_a = (long long *)malloc(sizeof(long long) * cnt);
    p->h_off_b = (long long *)malloc(sizeof(long long) * cnt);
    int *order = (int *)malloc(sizeof(int) * cnt);
    unsigned char *nbsel = (unsigned char *)malloc(cnt);
    if (!p->h_off_a || !p->h_off_b || !order || !nbsel) {
        free(order); free(nbsel); batch_free(p);
        return PlasmaErrorOutOfMemory;
    }
    // packed column-major matrices and vectors, each start 32-element aligned
    long long oa = 0, ob = 0;
    for (int i = 0; i < batch; i++) {
        p->h_off_a[i] = oa;
        p->h_off_b[i] = ob;
        oa += ((long long)n[i] * n[i] + 31) / 32 * 32;
        ob += ((long long)n[i] + 31) / 32 * 32;
        order[i] = i;
        nbsel[i] = (unsigned char)plasma_tuning_get_batched_nb(precision, n[i]);
    }
    p->elems_a = oa;
    p->elems_b = ob;
    // longest processing time first: decreasing n (stable)
    int *tmp = (int *)malloc(sizeof(int) * cnt);
    if (tmp == NULL) {
        free(order); free(nbsel); batch_free(p);
        return PlasmaErrorOutOfMemory;
    }
    {
        // counting sort by n, largest first
        int hist[NMAX + 2] = {0};
        for (int i = 0; i < batch; i++) hist[NMAX - n[i]]++;
        int acc = 0;
        for (int v = 0; v <= NMAX + 1; v++) { int c = hist[v]; hist[v] = acc; acc += c; }
        for (int i = 0; i < batch; i++) tmp[hist[NMAX - n[i]]++] = i;
        memcpy(order, tmp, sizeof(int) * cnt);
    }
    free(tmp);
    bool ok = cudaMalloc(&p->d_n, sizeof(int) * cnt) == cudaSuccess &&
              cudaMalloc(&p->d_off_a, sizeof(long long) * cnt) == cudaSuccess &&
              cudaMalloc(&p->d_off_b, sizeof(long long) * cnt) == cudaSuccess &&
              cudaMalloc(&p->d_order, sizeof(int) * cnt) == cudaSuccess &&
              cudaMalloc(&p->d_nbsel, cnt) == cudaSuccess &&
              cudaMalloc(&p->d_counter, sizeof(int)) == cudaSuccess;
    if (ok && batch > 0) {
        ok = cudaMemcpy(p->d_n, n, sizeof(int) * batch, cudaMemcpyHostToDevice) == cudaSuccess &&
             cudaMemcpy(p->d_off_a, p->h_off_a, sizeof(long long) * batch,
                        cudaMemcpyHostToDevice) == cudaSuccess &&
             cudaMemcpy(p->d_off_b, p->h_off_b, sizeof(long long) * batch,
                        cudaMemcpyHostToDevice) == cudaSuccess &&
             cudaMemcpy(p->d_order, order, sizeof(int) * batch, cudaMemcpyHostToDevice) ==
                 cudaSuccess &&
             cudaMemcpy(p->d_nbsel, nbsel, batch, cudaMemcpyHostToDevice) == cudaSuccess;
    }
    free(order);
    free(nbsel);
    if (!ok) {
        cudaGetLastError();
        batch_free(p);
        return PlasmaErrorOutOfMemory;
    }
    *plan = p;
    return PlasmaSuccess;
}

extern "C" void plasma_batch_destroy(plasma_batch_t *plan)
{
    if (plan) cudaDeviceSynchronize();
    batch_free(plan);
}

extern "C" long long plasma_batch_matrix_elems(const plasma_batch_t *plan)
{
    return plan ? plan->elems_a : 0;
}

extern "C" long long plasma_batch_vector_elems(const plasma_batch_t *plan)
{
    return plan ? plan->elems_b : 0;
}

extern "C" int plasma_batch_offsets(const plasma_batch_t *plan, long long *off_a,
                                    long long *off_b)
{
    if (plan == NULL) return -1;
    if (off_a) memcpy(off_a, plan->h_off_a, sizeof(long long) * plan->batch);
    if (off_b) memcpy(off_b, plan->h_off_b, sizeof(long long) * plan->batch);
    return PlasmaSuccess;
}

extern "C" int plasma_batch_set_graph(plasma_batch_t *plan, int on)
{
    if (plan == NULL) return -1;
    plan->graph = on != 0;
    return PlasmaSuccess;
}

// One batched operation: the counter reset and one persistent launch on the
// context stream, or the replay of the CUDA graph that holds both.
static int batch_run(plasma_batch_t *p, int prec, int op, void *A, void *B, void *C, void *D,
                     int *info)
{
    plasma_context_t *plasma = plasma_context_self();
    if (plasma == NULL) return PlasmaErrorNotInitialized;
    if (p == NULL) return -1;
    if (p->precision != prec) {
        plasma_error("batched call: precision differs from the plan's");
        return -1;
    }
    if (p->batch == 0) return PlasmaSuccess;
    if (A == NULL || ((op == OP_POSV || op == OP_POTRF) && info == NULL) ||
        ((op == OP_POSV || op == OP_POTRS || op == OP_POTRS_ADJ) && B == NULL) ||
        (op == OP_POTRS_ADJ && C == NULL) ||
        ((op == OP_POTRF_ADJ || op == OP_POTRS_ADJ) && D == NULL))
        return -2;
    BatchArgs a;
    a.batch = p->batch;
    a.n = p->d_n;
    a.off_a = p->d_off_a;
    a.off_b = p->d_off_b;
    a.order = p->d_order;
    a.nbsel = p->d_nbsel;
    a.A = A;
    a.B = B;
    a.C = C;
    a.D = D;
    a.info = info;
    a.counter = p->d_counter;
    a.op = op;
    int grid = plasma->num_sms *         // what an SM holds (registers, shared memory)
               (prec == PlasmaRealDouble ? batched_ctas<double>() : batched_ctas<float>());
    if (grid > p->batch) grid = p->batch;
    cudaStream_t s = plasma->stream;

    void *key[5] = {A, B, C, D, (void *)info};
    if (p->graph) {
        if (p->exec[op] == NULL || memcmp(p->g_ptr[op], key, sizeof(key)) != 0) {
            if (p->exec[op]) {
                cudaGraphExecDestroy(p->exec[op]);
                p->exec[op] = NULL;
            }
            cudaStream_t cap;
            if (cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking) != cudaSuccess)
                return PlasmaErrorEnvironment;
            cudaGraph_t g = NULL;
            cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal);
            cudaMemsetAsync(p->d_counter, 0, sizeof(int), cap);
            if (prec == PlasmaRealDouble) launch_batched<double, 1>(cap, a, grid);
            else launch_batched<float, 3>(cap, a, grid);
            cudaError_t rc = cudaStreamEndCapture(cap, &g);
            if (rc == cudaSuccess)
                rc = cudaGraphInstantiate(&p->exec[op], g, 0);
            if (g) cudaGraphDestroy(g);
            cudaStreamDestroy(cap);
            if (rc != cudaSuccess) {
                cudaGetLastError();
                p->exec[op] = NULL;
                return PlasmaErrorEnvironment;
            }
            memcpy(p->g_ptr[op], key, sizeof(key));
        }
        PLASMA_COUNT_LAUNCH();
        return cudaGraphLaunch(p->exec[op], s) == cudaSuccess ? PlasmaSuccess
                                                               : PlasmaErrorEnvironment;
    }
    cudaMemsetAsync(p->d_counter, 0, sizeof(int), s);
    PLASMA_COUNT_LAUNCH();
    if (prec == PlasmaRealDouble) launch_batched<double, 1>(s, a, grid);
    else launch_batched<float, 3>(s, a, grid);
    return PlasmaSuccess;
}

extern "C" int plasma_dposv_batched(plasma_batch_t *plan, double *A, double *B, int *info)
{ return batch_run(plan, PlasmaRealDouble, OP_POSV, A, B, NULL, NULL, info); }
extern "C" int plasma_sposv_batched(plasma_batch_t *plan, float *A, float *B, int *info)
{ return batch_run(plan, PlasmaRealFloat, OP_POSV, A, B, NULL, NULL, info); }
extern "C" int plasma_dpotrf_batched(plasma_batch_t *plan, double *A, int *info)
{ return batch_run(plan, PlasmaRealDouble, OP_POTRF, A, NULL, NULL, NULL, info); }
extern "C" int plasma_spotrf_batched(plasma_batch_t *plan, float *A, int *info)
{ return batch_run(plan, PlasmaRealFloat, OP_POTRF, A, NULL, NULL, NULL, info); }
extern "C" int plasma_dpotrs_batched(plasma_batch_t *plan, const double *L, double *B)
{ return batch_run(plan, PlasmaRealDouble, OP_POTRS, (void *)L, B, NULL, NULL, NULL); }
extern "C" int plasma_spotrs_batched(plasma_batch_t *plan, const float *L, float *B)
{ return batch_run(plan, PlasmaRealFloat, OP_POTRS, (void *)L, B, NULL, NULL, NULL); }
extern "C" int plasma_dpotrf_adjoint_batched(plasma_batch_t *plan, const double *L,
                                             double *Lbar)
{ return batch_run(plan, PlasmaRealDouble, OP_POTRF_ADJ, (void *)L, NULL, NULL, Lbar, NULL); }
extern "C" int plasma_spotrf_adjoint_batched(plasma_batch_t *plan, const float *L,
                                             float *Lbar)
{ return batch_run(plan, PlasmaRealFloat, OP_POTRF_ADJ, (void *)L, NULL, NULL, Lbar, NULL); }
extern "C" int plasma_dpotrs_adjoint_batched(plasma_batch_t *plan, const double *L,
                                             const double *X, double *Xbar, double *Lbar)
{ return batch_run(plan, PlasmaRealDouble, OP_POTRS_ADJ, (void *)L, (void *)X, Xbar, Lbar, NULL); }
extern "C" int plasma_spotrs_adjoint_batched(plasma_batch_t *plan, const float *L,
                                             const float *X, float *Xbar, float *Lbar)
{ return batch_run(plan, PlasmaRealFloat, OP_POTRS_ADJ, (void *)L, (void *)X, Xbar, Lbar, NULL); }
