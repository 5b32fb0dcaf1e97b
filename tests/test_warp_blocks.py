"""Synchronisation inside a block, without a GPU: the one-warp block factors of
f64_blocks.cuh under every order in which the hardware may run a warp's lanes
between two warp barriers, and how kernels with warps in different roles read
the failure status.

Lanes of a warp need not advance together (independent thread scheduling), so
shared memory that one lane writes and another reads has to be separated by a
__syncwarp.  A GPU hides a missing one; here the routines, taken from the
header as they stand, run on the CPU with one coroutine per lane, and a lane
runs alone until its next warp-wide operation, in ascending, descending and
shuffled order.  The result must be LAPACK's for every order.
"""
import ctypes
import os
import re
import subprocess

import numpy as np
import pytest

from conftest import ROOT

HEADER = os.path.join(ROOT, "plasma_b200", "csrc", "cuda", "f64_blocks.cuh")

HARNESS = r"""
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <ucontext.h>
#include <vector>
#define __device__
#define __forceinline__ inline
#define __noinline__
struct double2 { double x, y; };
struct float2 { float x, y; };
static struct { int x; } threadIdx;
using std::fma;
using std::sqrt;

// --- 32 coroutines; a lane runs until it yields at a warp-wide operation
static ucontext_t main_ctx, lane_ctx[32];
static int order[32], cur, done;
static void (*body)();
static void yield_lane() { swapcontext(&lane_ctx[cur], &main_ctx); threadIdx.x = cur; }
static void entry() { threadIdx.x = cur; body(); done++; }
static void run_warp(void (*fn)(), unsigned seed, int how)
{
    static std::vector<char> stacks(32 * 65536);
    body = fn;
    done = 0;
    for (int i = 0; i < 32; i++) {
        getcontext(&lane_ctx[i]);
        lane_ctx[i].uc_stack.ss_sp = &stacks[i * 65536];
        lane_ctx[i].uc_stack.ss_size = 65536;
        lane_ctx[i].uc_link = &main_ctx;
        makecontext(&lane_ctx[i], entry, 0);
        order[i] = how == 1 ? 31 - i : i;
    }
    srand(seed);
    while (done < 32) {
        if (how == 2)
            for (int i = 31; i > 0; i--) {
                const int j = rand() % (i + 1), t = order[i];
                order[i] = order[j];
                order[j] = t;
            }
        const int before = done;
        for (int i = 0; i < 32; i++) {
            cur = order[i];
            swapcontext(&main_ctx, &lane_ctx[cur]);
        }
        if (done != before && done < 32) abort();      // lanes disagree on the barriers
    }
}
static void __syncwarp() { yield_lane(); }
template <typename T> T blk_rsqrt(T d) { return T(1) / sqrt(d); }

// D(16 x 8) += A(16 x 8) B(8 x 8), lane = 4 g + t
template <int SPLIT, typename T> void mma8(T (&c)[4], const T (&a)[4], const T (&b)[2])
{
    static T A[16][8], B[8][8];
    const int lane = threadIdx.x, g = lane >> 2, t = lane & 3;
    A[g][t] = a[0]; A[g + 8][t] = a[1]; A[g][t + 4] = a[2]; A[g + 8][t + 4] = a[3];
    B[t][g] = b[0]; B[t + 4][g] = b[1];
    yield_lane();
    for (int e = 0; e < 4; e++)
        for (int k = 0; k < 8; k++)
            c[e] += A[g + 8 * (e >> 1)][k] * B[k][2 * t + (e & 1)];
    yield_lane();
}

@CODE@

template <typename T, int NB> struct Case {
    static T S[32 * 32], O[32 * 32], W8[32 * 8], rdiag[32];
    static int bad, fine[32];
    static void fast() { const int l = threadIdx.x; fine[l] = blk_factor<T, 3, NB>(S, W8); }
    static void any() { const int r = blk_factor_any<T, NB>(S, W8, O, rdiag); bad = r; }
};
template <typename T, int NB> T Case<T, NB>::S[32 * 32];
template <typename T, int NB> T Case<T, NB>::O[32 * 32];
template <typename T, int NB> T Case<T, NB>::W8[32 * 8];
template <typename T, int NB> T Case<T, NB>::rdiag[32];
template <typename T, int NB> int Case<T, NB>::bad;
template <typename T, int NB> int Case<T, NB>::fine[32];

template <typename T, int NB> int factor(T *a, T *w8, int general, unsigned seed, int how)
{
    typedef Case<T, NB> C;
    for (int c = 0; c < NB; c++)
        for (int r = 0; r < 32; r++) C::S[pd_at(c, r)] = C::O[pd_at(c, r)] = a[c * 32 + r];
    run_warp(general ? C::any : C::fast, seed, how);
    for (int c = 0; c < NB; c++)
        for (int r = 0; r < 32; r++) a[c * 32 + r] = C::S[pd_at(c, r)];
    memcpy(w8, C::W8, sizeof C::W8);
    if (general) return C::bad;
    for (int l = 0; l < 32; l++) if (!C::fine[l]) return -1;
    return 0;
}
extern "C" int factor_d32(double *a, double *w, int g, unsigned s, int h) { return factor<double, 32>(a, w, g, s, h); }
extern "C" int factor_d16(double *a, double *w, int g, unsigned s, int h) { return factor<double, 16>(a, w, g, s, h); }
extern "C" int factor_f32(float *a, float *w, int g, unsigned s, int h) { return factor<float, 32>(a, w, g, s, h); }
extern "C" int factor_f16(float *a, float *w, int g, unsigned s, int h) { return factor<float, 16>(a, w, g, s, h); }
"""


def definition(text, start):
    """The definition that begins at `start`, to its closing brace."""
    at = text.index(start)
    i = text.index("{", at)
    depth = 0
    while True:
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        i += 1
        if depth == 0:
            return text[at:i] + (";" if text[i] == ";" else "") + "\n"


@pytest.fixture(scope="module")
def warp(tmp_path_factory):
    text = open(HEADER).read()
    code = "".join(definition(text, s) for s in (
        "__device__ __forceinline__ int pd_at(",
        "template <typename T, typename L, typename R>\n__device__ __forceinline__ void inv8_column(",
        "__device__ __forceinline__ bool blk_plain(double",
        "__device__ __forceinline__ bool blk_plain(float"))
    code += "".join(re.findall(r"template <.*> struct Vec2.*;\n", text))
    code += "".join(definition(text, s) for s in (
        "template <typename T, int SPLIT, int NB>\n__device__ __forceinline__ bool blk_factor(",
        "template <typename T, int NB>\n__device__ __noinline__ int blk_factor_any("))
    d = tmp_path_factory.mktemp("warp")
    src, lib = d / "warp.cpp", d / "libwarp.so"
    src.write_text(HARNESS.replace("@CODE@", code))
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-ffp-contract=off",
                    "-Wno-unknown-pragmas", "-o", str(lib), str(src)], check=True)
    return ctypes.CDLL(str(lib))


@pytest.mark.parametrize("how", [0, 1, 2])
@pytest.mark.parametrize("general", [0, 1])
@pytest.mark.parametrize("nb", [16, 32])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_lane_orders(warp, dtype, nb, general, how):
    rng = np.random.default_rng(nb)
    m = rng.standard_normal((nb, nb))
    a = m @ m.T / nb + np.eye(nb)
    s = np.eye(32)
    s[:nb, :nb] = np.tril(a)
    fn = getattr(warp, f"factor_{'d' if dtype == np.float64 else 'f'}{nb}")
    buf = np.ascontiguousarray(s.T[:nb].astype(dtype))      # columns of 32 rows
    w8 = np.zeros((32, 8), dtype)
    assert fn(buf.ctypes.data_as(ctypes.c_void_p), w8.ctypes.data_as(ctypes.c_void_p), general,
              7, how) == 0
    ref = np.linalg.cholesky(a)
    eps = np.finfo(dtype).eps
    # |A - L L^T| <= (n + 1) u |L| |L^T|, entries of A at most 3: a small
    # multiple of n eps
    assert np.abs(buf[:, :nb].T - ref).max() <= 4 * nb * eps
    # w8[8 q + j] = column j of the inverse of diagonal block q
    for q in range(nb // 8):
        inv = np.linalg.inv(ref[8 * q:8 * q + 8, 8 * q:8 * q + 8])
        assert np.abs(w8[8 * q:8 * q + 8].T - inv).max() <= 64 * nb * eps


def test_status_is_read_once_per_block():
    """The status word may change while a kernel starts: a pivot that fails on
    one stream does so beside updates on others.  Where the warps of a block
    wait for one another (mbarriers, named barriers), they must all follow one
    reading, or those that go on wait for those that left."""
    bare = re.compile(r"if \(plasma_failed\(st\)\) return;")
    roles = re.compile(r"mbar_wait|\"bar\.sync")
    wrong = []
    cuda = os.path.dirname(HEADER)
    for name in sorted(os.listdir(cuda)):
        if not name.endswith(".cu"):
            continue
        text = open(os.path.join(cuda, name)).read()
        for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\(", text):
            body = definition(text[m.start():], "__global__")
            if roles.search(body) and bare.search(body):
                wrong.append(f"{name}: {m.group(1)}")
    assert not wrong
