// update_i8.cu -- trailing update of the FP64 Cholesky on the integer tensor
// cores (tcgen05 kind::i8):
//
//     C(m,n) -= A(m,k) A(n,k)^T,   k < n <= m,  C and A in FP64
//
// (compute/pzpotrf.c:57-77).  What bounds the DMMA form (update.cu) is the
// FP64 pipe, 64 multiply-adds a clock and SM; kind::i8 does 8192.  The
// product is split after Ozaki et al. (2012) in the integer form of Ootomo,
// Ozaki and Yokota (2024): every row of the panel is scaled by a power of
// two 2^e (its largest entry at most 127/128 of it) and written as a 55-bit
// fixed-point number, seven signed base-256 digits,
//
//     x = 2^(e-55) sum_p d_p 256^(6-p),   -128 <= d_p <= 127,
//
// and x y is formed from the 28 digit products with p + q <= 6.  Sums of one
// order t = p + q are exact in 32 bits (at most 7 x 256 x 2^14 < 2^31), the
// seven sums are joined exactly in 64-bit integers, and C takes one rounding
// of its own.
//
// Accuracy: the digits are relative to the largest entry of a row in the
// panel, which is what Cholesky's normwise backward error rests on (|L(i,k)| <=
// sqrt(A(i,i))).  Largest residual |A - L L^T| of an order of 3329 in units of
// 2^-53 sqrt(a_ii a_jj), here, with the DMMA update and with LAPACK: likelihood
// 3.3, 2.3, 2.3; rows scaled by up to 2^200 3.3, 4.1, 3.2; a first panel that
// holds most of every row 1.7, 7.8, 8.8; its entries falling over 16 decades
// within the rows 8.7, 10.3, 13.3.  What it does not have is the bound of a sum
// of rounded products entry by entry, n u |L| |L|^T: entries small against
// their row's largest lose low bits, and in the last of these matrices the
// least favourable entry is off by 1.6e14 u |L| |L|^T where the DMMA update is
// off by 16.  Tiles that are not 128 or 256 wide (PlasmaNb) take that one.  A
// row holding Inf or NaN makes its products NaN.
//
// k_panel_i8: digits of a panel, one CTA per 32 rows; global layout by units
// of 128 rows: [unit][K / 32][digit][8-row group][16-byte half][8 rows][16
// B], the no-swizzle K-major operand form, so that a stage of the row operand
// is one bulk copy of 28 KB (as fourteen of 2 KB their issue took longer than
// the stage's products).
//
// k_update_i8: one CTA per run of 128 x 64 blocks of C of one column block.
//   warp 0    : bulk copies -- the column block's digits (64 rows x K x 7,
//               112 KB) once per run, and the row block's digits through a
//               ring of 28 KB stages of 32 columns;
//   warp 1    : MMAs -- the seven sums lie side by side in tensor memory
//               (64 columns each), and so do the digits q of the column block
//               in shared memory: for digit p of the rows one product of
//               N = 64 (7 - p) columns adds to the sums p .. 6 at once (two
//               where that exceeds 256).  10 MMAs per 32 columns of K;
//   warps 2-9 : per block, read C while the products run, join the sums,
//               subtract and free tensor memory, store C.
// n = 8192, first bulk step (3422 blocks, two waves): 6.3 us a block and SM
// with no epilogue at all (the products are 3.9 us of tensor pipe at full
// rate; the rest is the wave's start and the hand-over of tensor memory, of
// which there is only one set); 9.4 us with C read after the products.
// Every wait is bounded (tc.cuh).
#include "common.cuh"
#include "tc.cuh"

namespace {

constexpr int I8_S = 7;                        // digits
constexpr int I8_M = 128, I8_N = 64;
constexpr int I8_KB = 32;                      // K per stage and MMA
constexpr int I8_UNIT = I8_S * 64 * I8_KB;     // 14 KB: 64 rows, 32 columns
constexpr int I8_STAGE = 2 * I8_UNIT;          // 128 rows
constexpr int I8_STAGES = 4;
constexpr int I8_THREADS = 320;
constexpr int I8_EPI_WARP0 = 2, I8_EPI_WARPS = 8;
constexpr int I8_NBMAX = 256;
constexpr int i8_smem(int nb) { return I8_STAGES * I8_STAGE + nb / I8_KB * I8_UNIT + 1024; }
static_assert(i8_smem(I8_NBMAX) <= 226 * 1024, "shared memory");

// scale[row] = 2^(e - 31)
__global__ void __launch_bounds__(256)
k_panel_i8(plasma_desc_t A, int k, signed char *dig, double *scale, const plasma_devstat_t *st)
{
    __shared__ double mx[8][32];
    if (plasma_failed(st)) return;
    const int nb = A.mb, nkb = nb / I8_KB;
    const int m = k + 1 + blockIdx.y, r0 = 32 * blockIdx.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row = r0 + lane, rows = plasma_tile_mview(A, m);
    const double *a = (const double *)plasma_tile_addr(A, m, k);
    const size_t ld = plasma_tile_mmain(A, m);
    // warp w: columns 32 w .. 32 w + 31 of the 32 rows
    double x[32];
    double big = 0.0;
    if (warp < nkb) {
#pragma unroll
        for (int c = 0; c < 32; c++) x[c] = row < rows ? a[(size_t)(32 * warp + c) * ld + row] : 0.0;
        // largest magnitude; NaN and Inf survive as bit patterns above it
        unsigned long long b = 0;
#pragma unroll
        for (int c = 0; c < 32; c++) {
            const unsigned long long v = __double_as_longlong(x[c]) & 0x7fffffffffffffffull;
            b = v > b ? v : b;
        }
        big = __longlong_as_double(b);
    }
    mx[warp][lane] = big;
    __syncthreads();
    if (warp >= nkb) return;
    unsigned long long b = 0;
    for (int w = 0; w < nkb; w++) {
        const unsigned long long v = __double_as_longlong(mx[w][lane]);
        b = v > b ? v : b;
    }
    const bool finite = b < 0x7ff0000000000000ull;
    int e = 0;
    if (b != 0 && finite) {
        const double f = frexp(__longlong_as_double(b), &e);
        if (f > 127.0 / 128.0) e++;
    }
    if (warp == 0)
        scale[(size_t)m * nb + row] = finite ? ldexp(1.0, e - 31) : __longlong_as_double(0x7ff8000000000000ll);
    // x 2^(55 - e) in two exact steps, each inside the range
    const int s = 55 - e, s1 = s / 2;
    const double f1 = __longlong_as_double((long long)(1023 + s1) << 52);
    const double f2 = __longlong_as_double((long long)(1023 + s - s1) << 52);
    signed char *u = dig + ((size_t)(m * (nb / 128) + row / 128) * nkb + warp) * I8_STAGE +
                     (row % 128) / 8 * 256 + (row % 8) * 16;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        uint32_t d[I8_S][4];
#pragma unroll
        for (int p = 0; p < I8_S; p++)
#pragma unroll
            for (int q = 0; q < 4; q++) d[p][q] = 0;
#pragma unroll
        for (int c = 0; c < 16; c++) {
            const double y = finite ? x[16 * h + c] * f1 * f2 : 0.0;
            // bytes 0 .. 5 biased by 128, byte 6 the leading digit
            const long long X = __double2ll_rn(y) + 0x0000808080808080ll;
            const uint32_t lo = (uint32_t)X ^ 0x80808080u, hi = (uint32_t)(X >> 32) ^ 0x8080u;
            const int sh = 8 * (c & 3);
            d[6][c >> 2] |= (lo & 255u) << sh;
            d[5][c >> 2] |= ((lo >> 8) & 255u) << sh;
            d[4][c >> 2] |= ((lo >> 16) & 255u) << sh;
            d[3][c >> 2] |= (lo >> 24) << sh;
            d[2][c >> 2] |= (hi & 255u) << sh;
            d[1][c >> 2] |= ((hi >> 8) & 255u) << sh;
            d[0][c >> 2] |= ((hi >> 16) & 255u) << sh;
        }
#pragma unroll
        for (int p = 0; p < I8_S; p++)
            *(uint4 *)(u + p * 4096 + h * 128) = make_uint4(d[p][0], d[p][1], d[p][2], d[p][3]);
    }
}

struct I8Args {
    plasma_desc_t A;
    const signed char *dig;
    const double *scale;
    int nlo, nhi;
    int nitems, ipc;
};

// Work items: 128 x 64 blocks, row half si and column block sj of tile (m, n).
// Those of one column block (n, sj) are adjacent, from the diagonal down; the
// block of a diagonal tile strictly above the diagonal (rows 0-127, columns
// from 128 on) is not an item.
struct I8Cursor {
    int m, n, si, sj, sm, sn, mt;

    __device__ __forceinline__ int top() const { return sj * I8_N >= I8_M ? 1 : 0; }
    __device__ __forceinline__ void start(const I8Args &g, int w)
    {
        sm = g.A.mb / I8_M;                    // 2 and 4 (nb = 256), or 1 and 2
        sn = g.A.mb / I8_N;
        mt = g.A.mt;
        for (n = g.nlo;; n++) {
            const int count = sn * sm * (mt - n) - sn / 2 * (sm - 1);
            if (w < count || n + 1 >= g.nhi) break;
            w -= count;
        }
        for (sj = 0; sj < sn - 1; sj++) {
            const int count = sm * (mt - n) - top();
            if (w < count) break;
            w -= count;
        }
        w += top();
        m = n + w / sm;
        si = w % sm;
    }
    __device__ __forceinline__ void next()
    {
        if (++si < sm) return;
        si = 0;
        if (++m < mt) return;
        if (++sj == sn) {
            sj = 0;
            n++;
        }
        m = n;
        si = top();
    }
    __device__ __forceinline__ bool last_of_column() const { return si == sm - 1 && m == mt - 1; }
};

__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *bar)
{
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
        ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}

// no swizzle, K-major: 16-byte halves of K 128 bytes apart, 8-row groups 256
__device__ __forceinline__ uint64_t i8_desc(const void *p) { return smem_desc(p, 128, 256, 0u); }

__device__ __forceinline__ void i8_mma(uint32_t d, uint64_t a, uint64_t b, int n, uint32_t acc)
{
    // S32 sums, signed A and B, both K-major, M = 128
    const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) |
                           ((uint32_t)(I8_M >> 4) << 24);
    const uint32_t z = 0;
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}"
        :: "r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc), "r"(z));
}

__device__ __forceinline__ void i8_commit(uint64_t *bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                 :: "r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, int (&r)[8])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
                   "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
}

__device__ __forceinline__ long long mad_wide(int a, int b, long long c)
{
    long long d;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
    return d;
}

// exact for |v| < 2^51
__device__ __forceinline__ double small_ll_to_double(long long v)
{
    return __longlong_as_double(v + 0x4338000000000000ll) - 6755399441055744.0;
}

__global__ void __launch_bounds__(I8_THREADS, 1)
k_update_i8(I8Args g, plasma_devstat_t *st)
{
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ uint64_t full_bar[I8_STAGES], empty_bar[I8_STAGES];
    __shared__ uint64_t bfull_bar[I8_NBMAX / I8_KB], bempty_bar, tfull_bar, tempty_bar;
    __shared__ uint32_t tmem_base_s;
    __shared__ volatile int abort_s;
    // one answer for the whole block, as its warps wait for one another
    if (__syncthreads_or(plasma_failed(st))) return;
    const int first = blockIdx.x * g.ipc;
    const int nit = min(g.ipc, g.nitems - first);
    if (nit <= 0) return;
    const int nb = g.A.mb, nkb = nb / I8_KB, units = nb / 128;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    unsigned char *ring = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char *resb = ring + I8_STAGES * I8_STAGE;
    if (tid == 0) {
        for (int s = 0; s < I8_STAGES; s++) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for (int kb = 0; kb < nkb; kb++) mbar_init(&bfull_bar[kb], 1);
        mbar_init(&bempty_bar, 1);
        mbar_init(&tfull_bar, 1);
        mbar_init(&tempty_bar, I8_EPI_WARPS);
        abort_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"(smem_u32(&tmem_base_s)), "r"(512u));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base_s;

    if (warp == 0 && lane == 0) {
        // ---------------- producer
        int it = 0, loads = 0;
        bool ok = true, load_b = true;
        I8Cursor c;
        c.start(g, first);
        for (int j = 0; j < nit && ok; j++, load_b = c.last_of_column(), c.next()) {
            const signed char *da = g.dig + (size_t)(c.m * units + c.si) * nkb * I8_STAGE;
            const signed char *db = g.dig + (size_t)(c.n * units + c.sj / 2) * nkb * I8_STAGE +
                                    c.sj % 2 * 2048;
            if (load_b) {
                // the products with the block held so far are complete
                if (loads > 0 && !mbar_wait(&bempty_bar, (loads - 1) & 1, &abort_s)) break;
                loads++;
            }
            for (int kb = 0; kb < nkb; kb++, it++) {
                const int s = it % I8_STAGES;
                if (it >= I8_STAGES &&
                    !mbar_wait(&empty_bar[s], ((it / I8_STAGES) - 1) & 1, &abort_s)) {
                    ok = false;
                    break;
                }
                if (load_b) {
                    mbar_expect_tx(&bfull_bar[kb], I8_UNIT);
#pragma unroll
                    for (int p = 0; p < I8_S; p++)
                        bulk_load(resb + kb * I8_UNIT + p * 2048,
                                  db + (size_t)kb * I8_STAGE + p * 4096, 2048, &bfull_bar[kb]);
                }
                mbar_expect_tx(&full_bar[s], I8_STAGE);
                bulk_load(ring + s * I8_STAGE, da + (size_t)kb * I8_STAGE, I8_STAGE, &full_bar[s]);
            }
        }
    } else if (warp == 1 && lane == 0) {
        // ---------------- MMA issuer
        int it = 0, loads = 0;
        bool ok = true, new_b = true;
        I8Cursor c;
        c.start(g, first);
        for (int j = 0; j < nit && ok; j++, new_b = c.last_of_column(), c.next()) {
            const bool last_b = c.last_of_column() && j + 1 < nit;
            if (new_b) loads++;
            if (j >= 1 && !mbar_wait(&tempty_bar, (j - 1) & 1, &abort_s)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (int kb = 0; kb < nkb; kb++, it++) {
                const int s = it % I8_STAGES;
                if (!mbar_wait(&full_bar[s], (it / I8_STAGES) & 1, &abort_s) ||
                    (new_b && !mbar_wait(&bfull_bar[kb], (loads - 1) & 1, &abort_s))) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const unsigned char *sa = ring + s * I8_STAGE, *sb = resb + kb * I8_UNIT;
                // digit 0 first: it reaches every sum, and clears them at kb = 0
#pragma unroll
                for (int p = 0; p < I8_S; p++) {
                    const uint64_t da = i8_desc(sa + p * 4096);
                    const int cols = I8_N * (I8_S - p);
                    const uint32_t acc = p > 0 || kb > 0 ? 1u : 0u;
                    i8_mma(tmem + I8_N * p, da, i8_desc(sb), cols < 256 ? cols : 256, acc);
                    if (cols > 256)
                        i8_mma(tmem + I8_N * p + 256, da, i8_desc(sb + 4 * 2048), cols - 256, acc);
                }
                i8_commit(&empty_bar[s]);
            }
            if (ok) i8_commit(&tfull_bar);
            if (ok && last_b) i8_commit(&bempty_bar);
        }
    } else if (warp >= I8_EPI_WARP0) {
        // ---------------- epilogue: rows 32 q .. +31 of the block, 32 columns
        const int q = warp & 3, c0 = 32 * ((warp - I8_EPI_WARP0) >> 2);
        const uint32_t lanes = (uint32_t)(32 * q) << 16;
        I8Cursor cur;
        cur.start(g, first);
        for (int j = 0; j < nit; j++, cur.next()) {
            const int m = cur.m, n = cur.n, si = cur.si, sj = cur.sj;
            const int row = si * I8_M + 32 * q + lane;
            const double sr = -g.scale[(size_t)m * nb + row];
            const int rows = plasma_tile_mview(g.A, m), cols = plasma_tile_mview(g.A, n);
            double *C = (double *)plasma_tile_addr(g.A, m, n) + row;
            const size_t ldc = plasma_tile_mmain(g.A, m);
            const int j0 = sj * I8_N + c0;
            const double *sc = g.scale + (size_t)n * nb + j0;
            // columns j0 .. jn-1 of this row are updated
            const int jn = row < rows ? min(cols, m == n ? row + 1 : cols) : 0;
            double c[32];
#pragma unroll
            for (int i = 0; i < 32; i++) c[i] = j0 + i < jn ? C[(size_t)(j0 + i) * ldc] : 0.0;
            const bool ok = __all_sync(0xffffffffu, mbar_wait(&tfull_bar, j & 1, &abort_s));
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (int cc = 0; cc < 32; cc += 8) {
                int t[I8_S][8];
#pragma unroll
                for (int o = 0; o < I8_S; o++)
                    tmem_ld8(tmem + lanes + (uint32_t)(I8_N * o + c0 + cc), t[o]);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    // sum over t of 2^(8 (6 - t)) times the sums, in two exact
                    // halves (the first pair fits 32 bits: at most 2^22 and 2^23)
                    const long long hi = mad_wide(t[0][i] * 256 + t[1][i], 65536,
                                                  mad_wide(t[2][i], 256, t[3][i]));
                    const long long lo = mad_wide(t[4][i], 65536, mad_wide(t[5][i], 256, t[6][i]));
                    const double P = fma(small_ll_to_double(hi), 16777216.0, small_ll_to_double(lo));
                    // C -= 2^(e_i + e_j - 62) P, the factor in two exact steps
                    c[cc + i] = fma(P * sr, __ldg(sc + cc + i), c[cc + i]);
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&tempty_bar);
#pragma unroll
            for (int i = 0; i < 32; i++)
                if (j0 + i < jn) C[(size_t)(j0 + i) * ldc] = c[i];
        }
    }
    // ---------------- teardown
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (abort_s) {
        if (tid == 0) {
            plasma_fail(st, PlasmaErrorInternal, 0);
            // a bounded time for issued MMAs and copies to land
            long long t0 = clock64();
            while (clock64() - t0 < 200000000LL) {}
        }
        __syncthreads();
    }
    if (warp == 1) {
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;"
                     :: "r"(tmem), "r"(512u));
    }
}

size_t i8_digit_bytes(const plasma_desc_t &A)
{
    return ((size_t)A.mt * A.mb * A.mb * I8_S + 1023) & ~(size_t)1023;
}

}  // namespace

// FP64 lower storage (general or packed), square tiles of 128 or 256 from
// the origin; the last tile row may be ragged.
extern "C" int plasma_cuda_update_i8_ok(plasma_desc_t A, plasma_enum_t uplo)
{
    return A.precision == PlasmaRealDouble && uplo == PlasmaLower &&
           (A.type == PlasmaGeneral || A.type == PlasmaLower) && A.mb == A.nb &&
           (A.mb == 128 || A.mb == 256) && A.i == 0 && A.j == 0;
}

// Bytes of one panel's digits and row scales.
extern "C" size_t plasma_cuda_panel_i8_bytes(plasma_desc_t A)
{
    return i8_digit_bytes(A) + (((size_t)A.mt * A.mb * sizeof(double) + 1023) & ~(size_t)1023);
}

// Digits and scales of the tiles A(m,k), m > k, into `panel` (1024-byte
// aligned, plasma_cuda_panel_i8_bytes).
extern "C" void plasma_cuda_panel_i8(cudaStream_t s, plasma_devstat_t *st, plasma_desc_t A, int k,
                                     void *panel)
{
    const int rows = A.mt - k - 1;
    if (rows <= 0) return;
    PLASMA_COUNT_LAUNCH();
    k_panel_i8<<<dim3(A.mb / 32, rows), 256, 0, s>>>(
        A, k, (signed char *)panel, (double *)((char *)panel + i8_digit_bytes(A)), st);
}

// Update of the tile columns [nlo, nhi) by panel k from its digits.
extern "C" void plasma_cuda_update_i8(cudaStream_t s, plasma_devstat_t *st, plasma_desc_t A, int k,
                                      int nlo, int nhi, const void *panel, int num_sms)
{
    if (nhi <= nlo) return;
    const int sm = A.mb / I8_M, sn = A.mb / I8_N;
    long long items = 0;
    double flops = 0.0, bytes = 0.0;
    for (int n = nlo; n < nhi; n++) {
        items += (long long)sn * sm * (A.mt - n) - sn / 2 * (sm - 1);
        const double cn = plasma_tile_mview(A, n), K = plasma_tile_nview(A, k);
        for (int m = n; m < A.mt; m++) {
            const double rm = plasma_tile_mview(A, m);
            flops += (m == n) ? cn * (cn + 1) * K : 2.0 * rm * cn * K;
            bytes += 8.0 * (m == n ? cn * (cn + 1) : 2.0 * rm * cn);
        }
    }
    if (items <= 0) return;
    I8Args g;
    g.A = A;
    g.dig = (const signed char *)panel;
    g.scale = (const double *)((const char *)panel + i8_digit_bytes(A));
    g.nlo = nlo;
    g.nhi = nhi;
    g.nitems = (int)items;
    // items per CTA (one CTA per SM): the smallest makespan of waves times
    // items plus half an item of fill and drain; at most 16, so that SMs come
    // free for the critical stream
    long long best = -1;
    g.ipc = 1;
    for (int ipc = 1; ipc <= 16; ipc++) {
        const long long ctas = (items + ipc - 1) / ipc;
        const long long cost = ((ctas + num_sms - 1) / num_sms) * (2 * ipc + 1);
        if (best < 0 || cost <= best) {
            best = cost;
            g.ipc = ipc;
        }
    }
    static unsigned long long attr = 0;
    if (plasma_first_on_device(&attr))
        cudaFuncSetAttribute(k_update_i8, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             i8_smem(I8_NBMAX));
    PLASMA_COUNT_LAUNCH();
    int prof = plasma_prof_begin(s);
    k_update_i8<<<(unsigned)((items + g.ipc - 1) / g.ipc), I8_THREADS, i8_smem(A.mb), s>>>(g, st);
    plasma_prof_end(prof, s, PLASMA_KCLASS_UPDATE, flops, bytes);
}
