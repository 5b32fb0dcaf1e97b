// potrf_diag.cu -- Cholesky of an FP64 diagonal tile (plasma_core_dpotrf on
// A(k,k), compute/pzpotrf.c:41-44): the head of every step's critical path.
//
// What bounds it: the chain of n pivots (each a reciprocal square root, a
// scaling and one fused update before the next pivot is known), then the
// n^3/6 multiply-adds of one SM's FP64 units (64 a clock).  So everything
// but that chain is taken off it:
//   * the tile is held in shared memory in 32 x 32 blocks.  A tile of order
//     <= 128 fits at once; a 256-wide one is taken in two phases of 128
//     columns (26 of its 36 blocks resident, 208 KB; the second phase reuses
//     the slots of the first phase's L11 and reads L21 where it lies);
//   * one warp factors a 32 x 32 diagonal block, eight columns at a time in
//     registers (blk_factor, f64_blocks.cuh);
//   * the rows below solve x L^T = a in strips of 8 rows on DMMA, with the
//     inverses of L's 8 x 8 diagonal blocks (a thread per row spends its time
//     on broadcast loads of L: 5300 clocks a step against 900-2700);
//   * of the trailing update only the next diagonal block is needed at once:
//     it is updated first, by all warps, and then warp 0 factors it while the
//     other warps update the rest on DMMA, in tasks from a counter.  The
//     warps of warp 0's scheduler join when the factor is done: a DMMA holds
//     the FP64 pipe for 64 clocks, and a pivot step's dependent DFMAs would
//     queue behind it (5700 clocks a block alone, 9200 with one DMMA warp on
//     the same scheduler).
// Measured beside the one-CTA left-looking kernel before it (16-column
// sub-panels, shuffles): order 128 61 -> 27 us, order 256 217 -> 78 us.
// Pivot test and info as LAPACK dpotrf: the first pivot that is not > 0, NaN
// included.
#include "common.cuh"
#include "f64_blocks.cuh"

namespace {

constexpr int PD_THREADS = 384;
constexpr int PD_WARPS = PD_THREADS / 32;
constexpr int PD_W = 128;                     // columns per phase
constexpr int PD_NMAX = 256;

// slot of block (I, J), J < 4, in a panel of Rb block rows
__host__ __device__ __forceinline__ int pd_slot(int I, int J, int Rb)
{
    return J * Rb - J * (J - 1) / 2 + (I - J);
}

// Rows r0 .. r0+7 of the block at X: x L^T = x, one warp
__device__ __forceinline__ void pd_solve_strip(double *X, const double *D, const double *W8,
                                               int r0)
{
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    double y[4][2], s[4][2];
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
        for (int e = 0; e < 2; e++) {
            y[q][e] = X[pd_at(8 * q + 2 * t + e, r0 + g)];
            s[q][e] = 0.0;
        }
    strip_solve32(y, s, D, W8);
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
        for (int e = 0; e < 2; e++) X[pd_at(8 * q + 2 * t + e, r0 + g)] = y[q][e];
}

// C(r0 .. r0+15, 8 c8 .. +8 NF-1) -= sum over kb of Xi(kb) Xj(kb)^T for the
// blocks of rows I and J of the panel, one warp
// (and a copy of the result to O when it is not null)
template <int NF>
__device__ __forceinline__ void pd_update(double *C, const double *S, int I, int J, int kb0,
                                          int kb1, int Rb, int r0, int c8, double *O = nullptr)
{
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    double acc[NF][4];
#pragma unroll
    for (int f = 0; f < NF; f++)
#pragma unroll
        for (int e = 0; e < 4; e++) acc[f][e] = 0.0;
    for (int kb = kb0; kb < kb1; kb++) {
        const double *a = S + pd_slot(I, kb, Rb) * F64_BLK;
        const double *b = S + pd_slot(J, kb, Rb) * F64_BLK;
#pragma unroll
        for (int k8 = 0; k8 < 32; k8 += 8) {
            const double af[4] = {a[pd_at(k8 + t, r0 + g)], a[pd_at(k8 + t, r0 + g + 8)],
                                  a[pd_at(k8 + t + 4, r0 + g)],
                                  a[pd_at(k8 + t + 4, r0 + g + 8)]};
#pragma unroll
            for (int f = 0; f < NF; f++) {
                const double bf[2] = {b[pd_at(k8 + t, 8 * (c8 + f) + g)],
                                      b[pd_at(k8 + t + 4, 8 * (c8 + f) + g)]};
                dmma_16x8x8(acc[f], af, bf);
            }
        }
    }
#pragma unroll
    for (int f = 0; f < NF; f++)
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int at = pd_at(8 * (c8 + f) + 2 * t + (e & 1), r0 + g + 8 * (e >> 1));
            const double v = C[at] - acc[f][e];
            C[at] = v;
            if (O != nullptr) O[at] = v;
        }
}

__global__ void __launch_bounds__(PD_THREADS, 1)
k_potrf_diag_f64(plasma_desc_t A, int k, int iinfo, plasma_devstat_t *st, int call)
{
    extern __shared__ __align__(16) double pd_smem[];
    __shared__ double rdiag[32], W8[32 * 8];
    __shared__ int bad_s;
    __shared__ int task_s[2 * PD_NMAX / 32];   // next task of every step
    // one answer for the whole block, as its warps wait for one another
    if (__syncthreads_or(plasma_failed(st))) return;
    double *T = (double *)plasma_tile_addr(A, k, k);
    const int ld = plasma_tile_mmain(A, k);
    const int n = plasma_tile_mview(A, k);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = (n + 31) / 32;              // block rows of the tile
    const int Rb = g;                         // block rows of the first panel
    double *O = pd_smem;                      // copy of the block being factored
    double *S = pd_smem + F64_BLK;             // the panel
    if (tid < 2 * PD_NMAX / 32) task_s[tid] = 0;
    int step = 0;

    for (int ph = 0; ph * PD_W < n; ph++) {
        const int o = ph * (PD_W / 32);       // first block row/column of the phase
        const int nc = min(PD_W / 32, g - o); // block columns
        // columns e0 .. e1-1, counted through the blocks (J, J), (J+1, J) ..
        // of block column J, by warps w of nw: 32 rows each
        auto each = [&](int J, int e0, int e1, int w, int nw, auto fn) {
            for (int e = e0 + w; e < e1; e += nw) {
                const int c = e & 31, I = J + (e >> 5);
                fn(S + pd_slot(I, J, Rb) * F64_BLK + pd_at(c, lane), 32 * (o + J) + c,
                   32 * (o + I) + lane);
            }
        };
        // identity past the matrix, so no step depends on its order
        auto in = [&](double *d, int col, int row) {
            if (row < n && col < n && row >= col) cp_async_8(d, T + (size_t)col * ld + row, true);
            else *d = row == col ? 1.0 : 0.0;
        };
        auto out = [&](const double *d, int col, int row) {
            if (row < n && row >= col) T[(size_t)col * ld + row] = *d;
        };
        // the first diagonal block, which is all that the first factor
        // needs; the others follow while it runs, or at once in the second
        // phase, whose blocks owe L21 L21^T (rows o + I of the panel)
        each(0, 0, 32, warp, PD_WARPS, in);
        if (ph == 0) each(0, 0, 32, warp, PD_WARPS, [&](double *d, int col, int row) {
            in(O + (d - S), col, row);
        });
        if (ph > 0) {
            each(0, 32, 32 * (g - o), warp, PD_WARPS, in);
            for (int J = 1; J < nc; J++) each(J, 0, 32 * (g - o - J), warp, PD_WARPS, in);
        }
        cp_async_commit();
        cp_async_wait<0>();
        __syncthreads();
        if (ph > 0) {
            if (warp < 8)
                pd_update<1>(S + pd_slot(0, 0, Rb) * F64_BLK, S, o, o, 0, o, Rb,
                             16 * (warp >> 2), warp & 3, O);
            __syncthreads();
        }
        for (int J = 0; J < nc; J++, step++) {
            // warp 0: the diagonal block; the others: what earlier columns
            // owe the blocks of this column and the ones to its right, in
            // 16-row halves taken from a counter
            if (warp == 0) {
                double *D = S + pd_slot(J, J, Rb) * F64_BLK;
                int bad = 0;
                if (!__all_sync(0xffffffffu, blk_factor<double, 1, 32>(D, W8)))
                    bad = blk_factor_any<double, 32>(D, W8, O, rdiag);
                if (lane == 0) bad_s = bad;
            } else if (step == 0) {
                each(0, 32, 32 * g, warp - 1, PD_WARPS - 1, in);
                for (int Jc = 1; Jc < nc; Jc++)
                    each(Jc, 0, 32 * (g - Jc), warp - 1, PD_WARPS - 1, in);
                cp_async_commit();
                cp_async_wait<0>();
            }
            if (step > 0) {
                // warps of warp 0's scheduler join once the factor is done
                if ((warp & 3) == 0)
                    asm volatile("bar.sync 1, %0;" :: "n"(PD_THREADS / 4) : "memory");
                const int per = g - o - J, m = nc - J;    // block rows, columns from J on
                const int total = 2 * (m * per - m * (m - 1) / 2 - 1);
                for (;;) {
                    int task = 0;
                    if (lane == 0) task = atomicAdd(&task_s[step], 1);
                    task = __shfl_sync(0xffffffffu, task, 0);
                    if (task >= total) break;
                    // block task/2 + 1 in column-major order from (J, J) on
                    int b = task / 2 + 1, q = 0;
                    while (b >= per - q) { b -= per - q; q++; }
                    const int Jc = J + q, I = Jc + b, h = task & 1;
                    double *C = S + pd_slot(I, Jc, Rb) * F64_BLK;
                    if (J > 0) pd_update<4>(C, S, I, Jc, J - 1, J, Rb, 16 * h, 0);
                    else pd_update<4>(C, S, o + I, o + Jc, 0, o, Rb, 16 * h, 0);
                }
                // and the finished column to its left goes home
                if (J > 0 && warp > 0)
                    each(J - 1, 0, 32 * (g - o - J + 1), warp - 1, PD_WARPS - 1, out);
            }
            __syncthreads();
            const int bad = bad_s;
            if (bad != 0) {
                if (tid == 0) plasma_fail(st, iinfo + 32 * (o + J) + bad, call);
                return;
            }
            // rows below the block
            for (int r = warp; r < 4 * (g - o - J - 1); r += PD_WARPS)
                pd_solve_strip(S + pd_slot(J + 1 + (r >> 2), J, Rb) * F64_BLK,
                               S + pd_slot(J, J, Rb) * F64_BLK, W8, 8 * (r & 3));
            __syncthreads();
            // the next diagonal block, a 16 x 8 piece per warp
            if (J + 1 < nc) {
                if (warp < 8)
                    pd_update<1>(S + pd_slot(J + 1, J + 1, Rb) * F64_BLK, S, J + 1, J + 1, J,
                                 J + 1, Rb, 16 * (warp >> 2), warp & 3, O);
                __syncthreads();
            }
        }
        each(nc - 1, 0, 32 * (g - o - nc + 1), warp, PD_WARPS, out);
        __syncthreads();
    }
}

constexpr int pd_smem_bytes(int g)
{
    return (1 + (g <= 4 ? g * (g + 1) / 2 : 4 * g - 6)) * F64_BLK * (int)sizeof(double);
}

}  // namespace

// FP64 lower tiles of order <= 256; 0 (nothing launched) for others.
extern "C" int plasma_cuda_potrf_diag_f64(cudaStream_t s, plasma_devstat_t *st, int call,
                                          plasma_desc_t A, int k, int iinfo)
{
    const int n = plasma_tile_mview(A, k);
    if (n > PD_NMAX) return 0;
    static unsigned long long attr = 0;
    if (plasma_first_on_device(&attr))
        cudaFuncSetAttribute(k_potrf_diag_f64, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             pd_smem_bytes(PD_NMAX / 32));
    k_potrf_diag_f64<<<1, PD_THREADS, pd_smem_bytes((n + 31) / 32), s>>>(A, k, iinfo, st, call);
    return 1;
}
