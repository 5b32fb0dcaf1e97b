// trsm_rows.cu -- FP64 one-launch triangular sweep for up to 16 right-hand
// sides (potrs, posv and the band solves with 2 <= nrhs <= 32; the reference
// runs them as the tile tasks of compute/pztrsm.c:113-177):
//   forward : X_u = W_u   (B_u - sum_{k<u} L(u,k) X_k)
//   backward: X_u = W_u^T (B_u - sum_{k>u} L(k,u)^T X_k)
// over blocks of 64 rows, W_u the inverses of k_trtri_64, tickets and ready
// flags as in trsv.cu.
//
// What bounds it: the factor is read once (n^2/2 x 8 bytes), and a block can
// only finish after the one before it; the last block alone walks n/64
// products of 64 x 64 x NR.  Those run on DMMA (8 x 8 x 4: eight warps, 8 rows
// each), and a ninth warp keeps them fed: it streams the operator blocks two
// products ahead through a ring of four 32 KB slots, and the solution blocks
// as their flags appear.  n = 8192, 16 columns: 0.70 ms a sweep, of which the
// chain of 128 blocks is most; 1.80 ms with a thread per row and broadcast
// loads of X (14 us a product).
//
// Blocks of L are copied as they are stored; the row index of stored column
// c is XORed with 4 (c mod 4), which serves the operand reads of both
// orientations without bank conflicts.
#include "common.cuh"
#include "sweep.cuh"
#include "tc.cuh"

namespace {

constexpr int RW_SB = 64;
constexpr int RW_CONS = 256;                  // eight consumer warps
constexpr int RW_THREADS = RW_CONS + 32;      // and the producer warp
constexpr int RW_RING = 4;
constexpr int RW_BLK = RW_SB * RW_SB;

template <int NR> constexpr int rw_smem()
{
    // ring of L, W, ring of X, the residual
    return ((RW_RING + 1) * RW_BLK + (RW_RING + 1) * RW_SB * NR) * (int)sizeof(double);
}

__device__ __forceinline__ int rw_at(int c, int r) { return c * RW_SB + (r ^ (4 * (c & 3))); }

__device__ __forceinline__ void rw_mma(double (&c)[2], double a, double b)
{
    asm volatile(
        "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
        : "+d"(c[0]), "+d"(c[1]) : "d"(a), "d"(b));
}

// 16 bytes, of which the first `bytes` are read and the rest become zero
__device__ __forceinline__ void cp_async_16_part(void *dst, const void *src, int bytes)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_u32(dst)),
                 "l"(src), "r"(bytes));
}

// this thread's copies so far arrive on the barrier when they are complete
__device__ __forceinline__ void cp_async_arrive(uint64_t *bar)
{
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

// One warp copies the stored block p (rows x cols valid, leading dimension
// ld) into S, zero outside.
__device__ __forceinline__ void rw_copy(double *S, const double *p, size_t ld, int rows, int cols,
                                        int ncol, int lane)
{
    if ((ld & 1) == 0 && ((uintptr_t)p & 15) == 0) {
        const int r = 2 * lane, nv = rows - r;
        const int bytes = nv >= 2 ? 16 : nv == 1 ? 8 : 0;
#pragma unroll 8
        for (int c = 0; c < ncol; c++) {
            const bool in = c < cols && bytes > 0;
            cp_async_16_part(S + rw_at(c, r), in ? p + c * ld + r : p, in ? bytes : 0);
        }
    } else {
#pragma unroll 4
        for (int c = 0; c < ncol; c++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int r = lane + 32 * h;
                const bool in = c < cols && r < rows;
                cp_async_8(S + rw_at(c, r), in ? p + c * ld + r : p, in);
            }
    }
}

// acc (rows 8w .. 8w+7, NR columns) += M X for one 64 x 64 operator block:
// M(i,c) is stored element (row i, col c), or (row c, col i) when TR
template <int NR, bool TR>
__device__ __forceinline__ void rw_product(double (&acc)[NR / 8][2], const double *M,
                                           const double *X, int w, int lane)
{
    const int g = lane >> 2, t = lane & 3;
#pragma unroll 4
    for (int k = 0; k < RW_SB; k += 4) {
        const double a = TR ? M[rw_at(8 * w + g, k + t)] : M[rw_at(k + t, 8 * w + g)];
#pragma unroll
        for (int j = 0; j < NR / 8; j++) rw_mma(acc[j], a, X[rw_at(8 * j + g, k + t)]);
    }
}

// acc += W X, or W^T X when TR, for the lower-triangular inverse W of a diagonal
// block: zero parts left out, and every sum ends with the diagonal entry's
// term, in general its largest.  Begun with it, the sum's other terms would
// each round at the size of the result (band of 300, two right-hand sides:
// 3.0 u from the exact solution against 2.4 u).
template <int NR, bool TR>
__device__ __forceinline__ void rw_diagonal(double (&acc)[NR / 8][2], const double *W,
                                            const double *X, int w, int lane)
{
    const int g = lane >> 2, t = lane & 3;
    const int steps = TR ? (RW_SB - 8 * w) / 4 : 2 * w + 2;
#pragma unroll 4
    for (int i = 0; i < steps; i++) {
        const int k = TR ? RW_SB - 4 - 4 * i : 4 * i;
        const double a = TR ? W[rw_at(8 * w + g, k + t)] : W[rw_at(k + t, 8 * w + g)];
#pragma unroll
        for (int j = 0; j < NR / 8; j++) rw_mma(acc[j], a, X[rw_at(8 * j + g, k + t)]);
    }
}

template <int NR>
__global__ void __launch_bounds__(RW_THREADS, 1)
k_trsm_rows_f64(plasma_desc_t A, int uplo, int backward, const double *W, plasma_desc_t B, int c0,
                int ncols, SweepSync *sy, int epoch, plasma_devstat_t *st)
{
    extern __shared__ __align__(16) double rw_sm[];
    double *Lr = rw_sm;                        // [RING][64 x 64]
    double *Ws = Lr + RW_RING * RW_BLK;
    double *Xr = Ws + RW_BLK;                  // [RING][NR columns of 64]
    double *Rs = Xr + RW_RING * RW_SB * NR;
    __shared__ uint64_t full_l[RW_RING], full_x[RW_RING], empty[RW_RING], full_w;
    __shared__ int blk_s;
    __shared__ volatile int abort_s;
    // one answer for the whole block: the ticket loop holds barriers
    if (__syncthreads_or(plasma_failed(st))) return;
    const int n = A.m;
    const int nblk = (n + RW_SB - 1) / RW_SB;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, t4 = lane & 3;
    const bool lower = uplo == PlasmaLower;
    const bool tr = lower == (backward != 0);  // operator read transposed
    if (tid == 0) {
        for (int i = 0; i < RW_RING; i++) {
            mbar_init(&full_l[i], 32);
            mbar_init(&full_x[i], 32);
            mbar_init(&empty[i], RW_CONS / 32);
        }
        mbar_init(&full_w, 32);
        abort_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }

    int step0 = 0;                             // products of earlier tickets
    for (int round = 0;; round++) {
        if (tid == 0) blk_s = atomicAdd(&sy->ticket, 1);
        __syncthreads();
        const int t = blk_s;
        if (t >= nblk || abort_s) break;
        const int u = backward ? nblk - 1 - t : t;
        const int rows = min(RW_SB, n - u * RW_SB);
        const int s0 = sweep_first(A, lower, t, RW_SB, backward != 0, nblk);
        const int np = t - s0;                 // products of this ticket

        if (warp == RW_CONS / 32) {
            // ---------------- producer
            rw_copy(Ws, W + (size_t)u * RW_BLK, RW_SB, RW_SB, RW_SB, RW_SB, lane);
            cp_async_arrive(&full_w);
            auto load_l = [&](int j) {         // operator of product j
                const int s = s0 + j, k = backward ? nblk - 1 - s : s;
                const int kr = min(RW_SB, n - k * RW_SB);
                const LBlock<double> b = backward ? lblock<double, RW_SB>(A, lower, k, u)
                                                  : lblock<double, RW_SB>(A, lower, u, k);
                // stored rows run along the logical row index iff si == 1
                const int li = backward ? kr : rows, lj = backward ? rows : kr;
                const int sl = (step0 + j) % RW_RING;
                rw_copy(Lr + sl * RW_BLK, b.p, b.si == 1 ? b.sj : b.si, b.si == 1 ? li : lj,
                        b.si == 1 ? lj : li, RW_SB, lane);
                cp_async_arrive(&full_l[sl]);
            };
            for (int j = 0; j < RW_RING - 2 && j < np; j++) load_l(j);
            int ready = 0;                     // products whose solution block is known ready
            bool ok = true;
            for (int j = 0; j < np && ok; j++) {
                if (j + RW_RING - 2 < np) {
                    // the slot of product j + RING - 2 was last read two
                    // products ago
                    const int q = step0 + j + RW_RING - 2;
                    if (q >= RW_RING)
                        ok = __all_sync(0xffffffffu, mbar_wait(&empty[q % RW_RING],
                                                               (q / RW_RING - 1) & 1, &abort_s));
                    if (!ok) break;
                    load_l(j + RW_RING - 2);
                }
                const long long t0 = clock64();
                while (ready <= j) {
                    // 32 flags at a time; the leading ones that are set
                    const int s = s0 + ready + lane, k = backward ? nblk - 1 - s : s;
                    const bool set = s < t && ld_acquire(&sy->flags[k]) == epoch;
                    const unsigned m = __ballot_sync(0xffffffffu, set);
                    ready += m == 0xffffffffu ? 32 : __ffs(~m) - 1;
                    if (ready > j) break;
                    const bool stop = ld_acquire(&sy->abort) != 0 || abort_s ||
                                      clock64() - t0 > 4000000000LL;
                    if (__any_sync(0xffffffffu, stop)) {
                        if (lane == 0) {
                            atomicExch(&sy->abort, 1);
                            abort_s = 1;
                        }
                        ok = false;
                        break;
                    }
                }
                if (!ok) break;
                // the flags were read by single lanes: order the copies of all
                // lanes after that (a vote does not)
                __syncwarp();
                const int s = s0 + j, k = backward ? nblk - 1 - s : s;
                const int kr = min(RW_SB, n - k * RW_SB);
                const int sl = (step0 + j) % RW_RING;
                double *xd = Xr + sl * RW_SB * NR;
                const int tc = c0 / B.nb;
                if ((c0 + ncols - 1) / B.nb == tc) {
                    rw_copy(xd, b_elem<double>(B, k * RW_SB, c0),
                            (size_t)plasma_tile_mmain(B, k * RW_SB / B.mb), kr, ncols, NR, lane);
                } else {
                    // columns of two column tiles
                    for (int c = 0; c < NR; c++)
                        for (int r = lane; r < RW_SB; r += 32) {
                            const bool in = c < ncols && r < kr;
                            cp_async_8(xd + rw_at(c, r),
                                       in ? b_elem<double>(B, k * RW_SB + r, c0 + c) : W, in);
                        }
                }
                cp_async_arrive(&full_x[sl]);
            }
        } else {
            // ---------------- consumers: rows 8 warp .. 8 warp + 7 of block u
            const int row = 8 * warp + g;
            double acc[NR / 8][2], rhs[NR / 8][2];
#pragma unroll
            for (int j = 0; j < NR / 8; j++)
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const int col = 8 * j + 2 * t4 + e;
                    acc[j][e] = 0.0;
                    rhs[j][e] = row < rows && col < ncols
                                    ? *b_elem<double>(B, u * RW_SB + row, c0 + col) : 0.0;
                }
            bool ok = true;
            for (int j = 0; j < np; j++) {
                const int q = step0 + j, sl = q % RW_RING;
                ok = __all_sync(0xffffffffu,
                                mbar_wait(&full_l[sl], (q / RW_RING) & 1, &abort_s) &&
                                    mbar_wait(&full_x[sl], (q / RW_RING) & 1, &abort_s));
                if (!ok) break;
                if (tr) rw_product<NR, true>(acc, Lr + sl * RW_BLK, Xr + sl * RW_SB * NR, warp, lane);
                else rw_product<NR, false>(acc, Lr + sl * RW_BLK, Xr + sl * RW_SB * NR, warp, lane);
                __syncwarp();
                if (lane == 0) mbar_arrive(&empty[sl]);
            }
            // the residual to shared memory, then the diagonal block
#pragma unroll
            for (int j = 0; j < NR / 8; j++)
#pragma unroll
                for (int e = 0; e < 2; e++)
                    Rs[rw_at(8 * j + 2 * t4 + e, row)] = rhs[j][e] - acc[j][e];
            if (ok)
                ok = __all_sync(0xffffffffu, mbar_wait(&full_w, round & 1, &abort_s));
            asm volatile("bar.sync 1, %0;" ::"n"(RW_CONS) : "memory");
#pragma unroll
            for (int j = 0; j < NR / 8; j++) acc[j][0] = acc[j][1] = 0.0;
            if (backward) rw_diagonal<NR, true>(acc, Ws, Rs, warp, lane);
            else rw_diagonal<NR, false>(acc, Ws, Rs, warp, lane);
            if (ok) {
#pragma unroll
                for (int j = 0; j < NR / 8; j++)
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        const int col = 8 * j + 2 * t4 + e;
                        if (row < rows && col < ncols)
                            *b_elem<double>(B, u * RW_SB + row, c0 + col) = acc[j][e];
                    }
            }
            __threadfence();
            asm volatile("bar.sync 1, %0;" ::"n"(RW_CONS) : "memory");
            if (tid == 0 && !abort_s) st_release(&sy->flags[u], epoch);
        }
        step0 += np;
        __syncthreads();                       // slots, Ws and blk_s are free
    }
    cp_async_wait<0>();
    if (abort_s && tid == 0) plasma_fail(st, PlasmaErrorInternal, 0);
}

template <int NR>
void launch_rows_f64(cudaStream_t s, plasma_devstat_t *st, int uplo, int backward,
                     const plasma_desc_t &A, const void *W, const plasma_desc_t &B, int c0,
                     int ncols, void *sync, int epoch, int grid)
{
    static unsigned long long attr = 0;
    if (plasma_first_on_device(&attr))
        cudaFuncSetAttribute(k_trsm_rows_f64<NR>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             rw_smem<NR>());
    k_trsm_rows_f64<NR><<<grid, RW_THREADS, rw_smem<NR>(), s>>>(
        A, uplo, backward, (const double *)W, B, c0, ncols, (SweepSync *)sync, epoch, st);
}

}  // namespace

// Columns c0 .. c0+ncols-1 (at most 16) of B; arguments as checked by
// plasma_cuda_trsm_rows, `sync` the SweepSync with a fresh ticket.
extern "C" void plasma_cuda_trsm_rows_f64(cudaStream_t s, plasma_devstat_t *st,
                                          plasma_enum_t uplo, int backward, plasma_desc_t A,
                                          const void *W, plasma_desc_t B, int c0, int ncols,
                                          void *sync, int epoch, int grid)
{
    if (ncols <= 8)
        launch_rows_f64<8>(s, st, uplo, backward, A, W, B, c0, ncols, sync, epoch, grid);
    else
        launch_rows_f64<16>(s, st, uplo, backward, A, W, B, c0, ncols, sync, epoch, grid);
}
