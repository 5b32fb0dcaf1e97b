// sweep.cuh -- shared by the one-launch triangular sweeps (trsv.cu,
// trsm_rows.cu): the ticket and ready flags, the blocks of a tile factor, and
// the range of blocks that couple with a row block.
#pragma once
#include "common.cuh"

namespace {

struct SweepSync {
    int ticket;
    int abort;
    int flags[1];          // [nblk]
};

__device__ __forceinline__ int ld_acquire(const int *p)
{
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_release(int *p, int v)
{
    asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ bool wait_block(SweepSync *sy, int k, int epoch)
{
    long long t0 = clock64();
    while (ld_acquire(&sy->flags[k]) != epoch) {
        if (ld_acquire(&sy->abort)) return false;
        if (clock64() - t0 > 4000000000LL) {
            atomicExch(&sy->abort, 1);
            return false;
        }
        __nanosleep(32);
    }
    return true;
}

// Logical block (bi, bj) of L, SB x SB: element (i,j) at p[i*si + j*sj].
template <typename T>
struct LBlock {
    const T *p;
    int si, sj;
};

template <typename T, int SB>
__device__ __forceinline__ LBlock<T> lblock(const plasma_desc_t &A, bool lower,
                                            int bi, int bj)
{
    const int gi = bi * SB, gj = bj * SB;
    const int ti = gi / A.mb, tj = gj / A.mb;
    const int oi = gi % A.mb, oj = gj % A.mb;
    LBlock<T> b;
    if (lower) {
        const T *t = (const T *)plasma_tile_addr(A, ti, tj);
        int ld = plasma_tile_mmain(A, ti);
        b.p = t + (size_t)oj * ld + oi;
        b.si = 1;
        b.sj = ld;
    } else {
        const T *t = (const T *)plasma_tile_addr(A, tj, ti);
        int ld = plasma_tile_mmain(A, tj);
        b.p = t + (size_t)oi * ld + oj;
        b.si = ld;
        b.sj = 1;
    }
    return b;
}

template <typename T>
__device__ __forceinline__ T *b_elem(const plasma_desc_t &B, int row, int col)
{
    const int m = row / B.mb, r = row - m * B.mb;
    const int t = col / B.nb, c = col - t * B.nb;
    return (T *)plasma_tile_addr(B, m, t) + (size_t)c * plasma_tile_mmain(B, m) + r;
}

// Tickets t of a sweep run over the row blocks in sweep order (block t
// forward, nblk-1-t backward).  The first ticket whose block couples with
// that of ticket t: 0 for a full triangle; in a band, element (i,j) is zero
// for |i - j| > kd, so blocks of sb rows couple up to kd rows past their
// own.
__host__ __device__ __forceinline__ int sweep_first(const plasma_desc_t &A, bool lower, int t,
                                                    int sb, bool backward, int nblk)
{
    if (A.type != PlasmaGeneralBand) return 0;
    const int kd = lower ? A.kl : A.ku;
    if (!backward) {
        const int lo = t * sb - kd;                       // first row coupled
        return lo > 0 ? lo / sb : 0;
    }
    const int u = nblk - 1 - t, hi = (u * sb + sb - 1 + kd) / sb;   // last block coupled
    return hi < nblk ? nblk - 1 - hi : 0;
}

}  // namespace
