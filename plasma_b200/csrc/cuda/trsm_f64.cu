// trsm_f64.cu -- the panel solve of an FP64 Cholesky step,
//
//     X L_kk^T = A(m,k)   for the row tiles m in [mlo, mhi)
//
// (compute/pzpotrf.c:50-56, plasma_core_dtrsm Right, Lower, Trans, NonUnit).
//
// What bounds it: rows nb^2 / 2 multiply-adds on the FP64 tensor pipe (16 a
// clock and scheduler), and, when there are few rows, the chain through the
// columns.  A warp owns 8 rows and walks the 32-column blocks J left to
// right: Y_J = A_J - sum_{I<J} X_I L(J,I)^T, then the strip solve with the
// inverted 8 x 8 diagonal blocks of L(J,J) (f64_blocks.cuh).  A solved strip
// is the A operand of later products as it stands in registers; it is kept in
// shared memory in that form (one 16-byte read a lane and 8 columns).  The
// warps of a CTA share the blocks of L, which come through a ring of eight
// 8 KB slots, in the order (J, 0) .. (J, J), seven blocks ahead.  32 rows a
// CTA (one warp per scheduler) while that leaves every CTA an SM of its own,
// 64 rows above: two warps hide each other's latencies and halve the reads
// of L.
#include "common.cuh"
#include "f64_blocks.cuh"

namespace {

constexpr int TF_NBMAX = 256;
constexpr int TF_RING = 8;                    // blocks of L in flight

__host__ __device__ constexpr int tf_smem(int warps, int nb)
{
    // solved strips (fragments), ring, 8 x 8 inverses
    return (8 * warps * nb + TF_RING * F64_BLK + nb * 8) * (int)sizeof(double);
}

template <int WARPS>
__global__ void __launch_bounds__(32 * WARPS, 1)
k_trsm_f64(plasma_desc_t A, int k, int mlo, int vec, const plasma_devstat_t *st)
{
    constexpr int TF_THREADS = 32 * WARPS, TF_ROWS = 8 * WARPS;
    extern __shared__ __align__(16) double tf_sm[];
    if (plasma_failed(st)) return;
    const int nb = plasma_tile_mview(A, k);   // a multiple of 32
    const int nblk = nb / 32;
    double *Xf = tf_sm;                       // [warp][column / 8][lane][2]
    double *Lr = Xf + TF_ROWS * nb;           // ring
    double *W8 = Lr + TF_RING * F64_BLK;      // [nb][8]
    const int m = mlo + blockIdx.x;
    const int rows = plasma_tile_mview(A, m);
    const int r0 = blockIdx.y * TF_ROWS;
    if (r0 >= rows) return;
    const double *L = (const double *)plasma_tile_addr(A, k, k);
    const int ldl = plasma_tile_mmain(A, k);
    double *B = (double *)plasma_tile_addr(A, m, k);
    const int ldb = plasma_tile_mmain(A, m);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, t = lane & 3;
    const int total = nblk * (nblk + 1) / 2;

    // block number b of the order (J, 0) .. (J, J) into its ring slot
    int nj = 0, ni = 0;                       // the next block to request
    auto request = [&](int b) {
        if (b < total) {
            double *d = Lr + (b % TF_RING) * F64_BLK;
            const double *src = L + (size_t)(32 * ni) * ldl + 32 * nj;
            if (vec) {
#pragma unroll
                for (int e = tid; e < F64_BLK / 2; e += TF_THREADS) {
                    const int c = e >> 4, r = 2 * (e & 15);
                    cp_async_16(d + pd_at(c, r), src + (size_t)c * ldl + r, true);
                }
            } else {
#pragma unroll
                for (int e = tid; e < F64_BLK; e += TF_THREADS) {
                    const int c = e >> 5, r = e & 31;
                    cp_async_8(d + pd_at(c, r), src + (size_t)c * ldl + r, true);
                }
            }
            if (++ni > nj) { nj++; ni = 0; }
        }
        cp_async_commit();
    };
    for (int b = 0; b < TF_RING - 1; b++) request(b);

    // this warp's strip of A_J in accumulator form
    const int row = r0 + 8 * warp + g;
    auto fetch = [&](int J, double (&y)[4][2]) {
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
            for (int e = 0; e < 2; e++)
                y[q][e] = row < rows ? B[(size_t)(32 * J + 8 * q + 2 * t + e) * ldb + row] : 0.0;
    };
    double y[4][2], nx[4][2], sum[4][2];      // sum: X_{<J} L(J,<J)^T
    fetch(0, nx);

    // the inverses of the 8 x 8 diagonal blocks, a thread per column
    for (int c = tid; c < nb; c += TF_THREADS) {
        const int o = c & ~7;
        double l[8][8], rd[8], w[8];
#pragma unroll
        for (int q = 0; q < 8; q++)
#pragma unroll
            for (int i = q; i < 8; i++) l[i][q] = L[(size_t)(o + q) * ldl + o + i];
#pragma unroll
        for (int i = 0; i < 8; i++) rd[i] = 1.0 / l[i][i];
        inv8_column(c & 7, [&](int i, int q) { return l[i][q]; }, [&](int i) { return rd[i]; }, w);
#pragma unroll
        for (int i = 0; i < 8; i++) W8[c * 8 + i] = w[i];
    }

    double *xf = Xf + (size_t)warp * 8 * nb + lane * 2;
    int b = 0;
    for (int J = 0; J < nblk; J++) {
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
            for (int e = 0; e < 2; e++) {
                y[q][e] = nx[q][e];
                sum[q][e] = 0.0;
            }
        if (J + 1 < nblk) fetch(J + 1, nx);
        for (int I = 0; I <= J; I++, b++) {
            cp_async_wait<TF_RING - 2>();
            __syncthreads();                  // block b is in; block b-1 is read
            request(b + TF_RING - 1);         // into the slot of block b-1
            const double *D = Lr + (b % TF_RING) * F64_BLK;
            if (I == J) break;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const double2 x01 = *(const double2 *)(xf + (4 * I + q) * 64);
                const double x[2] = {x01.x, x01.y};
#pragma unroll
                for (int f = 0; f < 4; f++)
                    strip_mma(sum[f], x, D[pd_at(8 * q + 2 * t, 8 * f + g)],
                              D[pd_at(8 * q + 2 * t + 1, 8 * f + g)]);
            }
        }
        strip_solve32(y, sum, Lr + (b % TF_RING) * F64_BLK, W8 + 32 * J * 8);
        b++;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            if (J + 1 < nblk) *(double2 *)(xf + (4 * J + q) * 64) = make_double2(y[q][0], y[q][1]);
#pragma unroll
            for (int e = 0; e < 2; e++)
                if (row < rows) B[(size_t)(32 * J + 8 * q + 2 * t + e) * ldb + row] = y[q][e];
        }
    }
    cp_async_wait<0>();
}

template <int WARPS>
void launch_trsm_f64(cudaStream_t s, plasma_devstat_t *st, const plasma_desc_t &A, int k,
                     int mlo, int mhi, int nk)
{
    static unsigned long long attr = 0;
    if (plasma_first_on_device(&attr))
        cudaFuncSetAttribute(k_trsm_f64<WARPS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             tf_smem(WARPS, TF_NBMAX));
    // 16-byte copies of L's columns
    const int vec = plasma_tile_mmain(A, k) % 2 == 0 &&
                    ((uintptr_t)plasma_tile_addr(A, k, k) & 15) == 0;
    dim3 grid((unsigned)(mhi - mlo), (unsigned)ceil_div(A.mb, 8 * WARPS));
    k_trsm_f64<WARPS><<<grid, 32 * WARPS, tf_smem(WARPS, nk), s>>>(A, k, mlo, vec, st);
}

}  // namespace

// FP64 lower tiles of a multiple of 32 columns, at most 256; 0 (nothing
// launched) for others.
extern "C" int plasma_cuda_trsm_f64(cudaStream_t s, plasma_devstat_t *st, plasma_desc_t A,
                                    int k, int mlo, int mhi)
{
    const int nk = plasma_tile_mview(A, k);
    if (nk % 32 != 0 || nk == 0 || nk > TF_NBMAX) return 0;
    if ((long long)(mhi - mlo) * ceil_div(A.mb, 32) <= plasma_context_self()->num_sms)
        launch_trsm_f64<4>(s, st, A, k, mlo, mhi, nk);
    else
        launch_trsm_f64<8>(s, st, A, k, mlo, mhi, nk);
    return 1;
}
