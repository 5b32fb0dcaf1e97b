"""The tile kernels of the Cholesky step at the sizes where they can go wrong:
edges of their blocks and phases, ragged orders, the ends of the number range,
and the row scales of the split half-precision update.  References are LAPACK
(numpy) in FP64 on the same inputs; bounds are the reference tester's 50 eps
(test/test_zpotrf.c:124-152) unless a test derives its own.
"""
import numpy as np
import pytest
import torch  # noqa: F401  (CUDA context)

import gen
import plasma_b200 as pb
from conftest import EPS, SEPS, TOL, factor_residual

pytestmark = pytest.mark.gpu
LO, UP = pb.PlasmaLower, pb.PlasmaUpper


@pytest.fixture(scope="module")
def L():
    lib = pb.lib()
    assert lib.plasma_init() == 0
    assert lib.plasma_set(pb.PlasmaTuning, pb.PlasmaDisabled) == 0
    yield lib
    lib.plasma_finalize()


def potrf(L, a, nb, dtype=np.float64, uplo=LO):
    assert L.plasma_set(pb.PlasmaNb, nb) == 0
    f = np.asfortranarray(a.astype(dtype))
    fn = L.plasma_dpotrf if dtype == np.float64 else L.plasma_spotrf
    return fn(uplo, f.shape[0], f.ctypes.data, f.shape[0]), f


# one diagonal tile: 32-column blocks, 8-column groups, the second phase of
# tiles wider than 128
@pytest.mark.parametrize("n", [1, 7, 8, 9, 31, 32, 33, 63, 65, 96, 127, 128, 129, 136, 160, 161,
                               191, 224, 255, 256])
def test_diagonal_tile(L, n):
    a = gen.likelihood(n, 1, seed=n)[0]
    info, f = potrf(L, a, 256)
    assert info == 0
    ref = np.linalg.cholesky(a)
    assert np.abs(np.tril(f) - ref).max() <= TOL * EPS * np.abs(ref).max()
    np.testing.assert_array_equal(np.triu(f, 1), np.triu(a, 1))


# a few tiles: panel solve (tile widths a multiple of 32, and others) and
# the two block sizes of the update (few and many blocks)
@pytest.mark.parametrize("n,nb", [(70, 32), (200, 32), (333, 96), (257, 128), (640, 160),
                                  (1000, 224), (769, 256), (1100, 48), (2305, 128)])
def test_tile_steps(L, n, nb):
    a = gen.likelihood(n, 1, seed=n + nb)[0]
    info, f = potrf(L, a, nb)
    assert info == 0
    assert factor_residual(np.tril(f), a) < TOL


# pivots far outside the normal range take the general block factor: a power
# of two scales the factor exactly
@pytest.mark.parametrize("e", [-1000, -960, -500, 500, 960, 1000])
@pytest.mark.parametrize("n", [40, 200])
def test_extreme_scales(L, n, e):
    a = gen.likelihood(n, 1, seed=5)[0]
    s = 2.0 ** e
    info, f = potrf(L, a * s, 256)
    assert info == 0
    ref = np.linalg.cholesky(a) * 2.0 ** (e // 2)
    assert np.abs(np.tril(f) - ref).max() <= TOL * EPS * np.abs(ref).max()


# LAPACK's info wherever the bad pivot lies (8-column groups, 32-column
# blocks, phases, tiles), for zero, negative and NaN pivots
@pytest.mark.parametrize("col", [0, 5, 8, 31, 32, 100, 127, 128, 170, 255, 256, 300])
@pytest.mark.parametrize("bad", [0.0, -1.0, np.nan])
def test_info(L, col, bad):
    a = gen.likelihood(320, 1, seed=9)[0]
    a[col, :] = 0.0
    a[:, col] = 0.0
    a[col, col] = bad
    for dtype in (np.float64, np.float32):
        info, _ = potrf(L, a, 256, dtype)
        assert info == col + 1


# The split half-precision update scales rows by powers of two: the factor of
# D A D (D a power of two per row) is D L, to the same relative accuracy as
# L itself, over most of FP32's exponent range.  The residual against
# 2^-24 sqrt(a_ii a_jj): measured 7.1, with one of the small products of the
# split left out above 90; for a heavy first panel, its entries falling within
# the rows or not, 10 to 29 and above 1100.
@pytest.mark.parametrize("n,nb", [(1024, 256), (768, 128)])
@pytest.mark.parametrize("spread", [0, 12, 55])
def test_fp32_row_scales(L, n, nb, spread):
    a = gen.likelihood(n, 1, seed=11)[0].astype(np.float32).astype(np.float64)
    check_split(L, a, nb, spread, 16.0)


@pytest.mark.parametrize("n,nb", [(1024, 256), (768, 128)])
@pytest.mark.parametrize("decades", [0, 4, 8])
def test_fp32_within_rows(L, n, nb, decades):
    a = heavy_panel(n, nb, decades, n).astype(np.float32).astype(np.float64)
    check_split(L, a, nb, 0, 64.0)


def check_split(L, a, nb, spread, limit):
    n = len(a)
    d = 2.0 ** np.random.default_rng(n + spread).integers(-spread, spread + 1, n)
    info, f = potrf(L, a * d[:, None] * d[None, :], nb, np.float32)
    assert info == 0
    low = np.tril(f).astype(np.float64) / d[:, None]
    err = np.abs(low @ low.T - a) / np.sqrt(np.outer(np.diag(a), np.diag(a)))
    assert err.max() <= limit * SEPS


# an indefinite matrix whose rows outgrow their scale fails where LAPACK does
def test_fp32_indefinite_info(L):
    n = 1024
    a = gen.likelihood(n, 1, seed=13)[0]
    a[700, :300] = a[:300, 700] = 1e6
    a[900, :300] = a[:300, 900] = 1e30
    for nb in (128, 256):
        info, _ = potrf(L, a, nb, np.float32)
        assert info == 701


# several right-hand sides through the one-launch sweeps: both column widths
# of the kernel, two launches, ragged orders (odd leading dimensions), both
# triangles; a backward-stable solve has a residual of order n eps
@pytest.mark.parametrize("nrhs", [2, 8, 9, 16, 17, 32])
@pytest.mark.parametrize("n,nb", [(64, 64), (129, 64), (515, 128), (1000, 256)])
def test_sweeps_many_rhs(L, n, nb, nrhs):
    assert L.plasma_set(pb.PlasmaNb, nb) == 0
    a, b = gen.likelihood(n, nrhs, seed=n + nrhs)
    for dtype, fn, eps in ((np.float64, L.plasma_dposv, EPS), (np.float32, L.plasma_sposv, SEPS)):
        for uplo in (LO, UP):
            f, x = np.asfortranarray(a.astype(dtype)), np.asfortranarray(b.astype(dtype))
            assert fn(uplo, n, nrhs, f.ctypes.data, n, x.ctypes.data, n) == 0
            r = np.abs(b - a @ x).sum(axis=1).max()
            scale = n * np.abs(a).sum(axis=1).max() * np.abs(x).sum(axis=1).max()
            assert r / scale < TOL * eps


# the same sweeps cut to a band, down to a diagonal matrix and up to a band
# wider than a block
@pytest.mark.parametrize("kd", [0, 1, 63, 64, 65, 200])
@pytest.mark.parametrize("nrhs", [1, 3, 20])
def test_band_sweeps(L, kd, nrhs):
    n, nb = 700, 128
    assert L.plasma_set(pb.PlasmaNb, nb) == 0
    a, lo, up, b = gen.band(n, kd, nrhs, seed=kd)
    for dtype, fn, eps in ((np.float64, L.plasma_dpbsv, EPS), (np.float32, L.plasma_spbsv, SEPS)):
        for uplo, ab in ((LO, lo), (UP, up)):
            f, x = np.asfortranarray(ab.astype(dtype)), np.asfortranarray(b.astype(dtype))
            assert fn(uplo, n, kd, nrhs, f.ctypes.data, kd + 1, x.ctypes.data, n) == 0
            r = np.abs(b - a @ x).sum(axis=1).max()
            scale = n * np.abs(a).sum(axis=1).max() * np.abs(x).sum(axis=1).max()
            assert r / scale < TOL * eps


# FP32 orders that are no multiple of the tile go through padded tiles; the
# other triangle and the columns past n stay as they were
@pytest.mark.parametrize("n,nb", [(1, 128), (127, 128), (300, 128), (257, 256), (700, 256)])
def test_fp32_ragged(L, n, nb):
    a = gen.likelihood(n, 1, seed=n)[0]
    for uplo in (LO, UP):
        info, f = potrf(L, a, nb, np.float32, uplo)
        assert info == 0
        tri, other = (np.tril, np.triu) if uplo == LO else (np.triu, np.tril)
        k = 1 if uplo == LO else -1
        low = tri(f).astype(np.float64)
        low = low if uplo == LO else low.T
        assert np.linalg.norm(low @ low.T - a) <= TOL * n * SEPS * np.linalg.norm(a)
        np.testing.assert_array_equal(other(f, k), other(a.astype(np.float32), k))


def heavy_panel(n, nb, decades, seed):
    """A whose factor has rows of norm about 1 in its first tile column and
    little beyond, so that the first update decides the residual; the entries
    of a row fall by `decades`, those of odd rows in the other direction."""
    rng = np.random.default_rng(seed)
    p = rng.standard_normal((n, nb))
    w = 10.0 ** (-decades * np.arange(nb) / nb)
    p *= np.where((np.arange(n) % 2 == 0)[:, None], w, w[::-1])
    p /= np.linalg.norm(p, axis=1)[:, None]
    a = p @ p.T
    a = (a + a.T) * 0.5
    a[np.diag_indices(n)] = 1.1
    return a


# FP64 steps with 3072 trailing rows or more update from integer digits: one
# and a few such steps, tile orders 128 and 256, a ragged last tile, and rows
# whose scales differ by up to 2^400.  The residual of 24 rows, in extended
# precision, against u sqrt(a_ii a_jj).  Measured 2.7 to 3.3 u for the
# likelihood's matrices (LAPACK the same), 1.4 to 1.7 for a heavy first panel
# (LAPACK 8.8), 5.4 to 9.8 with entries that fall within the rows (18).  Without
# the least of the 28 digit products the same residuals are above 20, 550 and
# 1600 u, without the next above 2000.
@pytest.mark.parametrize("n,nb,spread", [(3328, 256, 0), (3329, 256, 0), (3585, 128, 0),
                                         (3500, 256, 400)])
@pytest.mark.parametrize("uplo", [LO, UP])
def test_digit_update(L, n, nb, spread, uplo):
    a = gen.likelihood(n, 1, seed=n)[0]
    check_digits(L, a, nb, spread, uplo, 8.0)


@pytest.mark.parametrize("n,nb", [(3329, 256), (3585, 128)])
@pytest.mark.parametrize("decades,limit", [(0, 4.0), (8, 16.0), (16, 16.0)])
def test_digit_update_within_rows(L, n, nb, decades, limit):
    check_digits(L, heavy_panel(n, nb, decades, n), nb, 0, LO, limit)


def check_digits(L, a, nb, spread, uplo, limit):
    n = len(a)
    rng = np.random.default_rng(n)
    d = 2.0 ** rng.integers(-spread // 2, spread // 2 + 1, n)
    info, f = potrf(L, a * d[:, None] * d[None, :], nb, uplo=uplo)
    assert info == 0
    lf = (np.tril(f) if uplo == LO else np.triu(f).T) / d[:, None]
    rows = np.concatenate([[n - 1, n - 2], rng.integers(nb, n, 22)])
    lf = lf.astype(np.longdouble)
    r = a[rows].astype(np.longdouble)
    for c in range(0, n, 128):
        r -= lf[rows, c:c + 128] @ lf[:, c:c + 128].T
    s = np.sqrt(np.diag(a))
    err = np.abs(r) / (s[rows][:, None] * s[None, :])
    assert err[np.arange(n)[None, :] <= rows[:, None]].max() <= limit * 2.0 ** -53


@pytest.mark.parametrize("bad", [-1.0, np.nan])
@pytest.mark.parametrize("col", [100, 300, 3200])
def test_digit_update_info(L, col, bad):
    a = gen.likelihood(3400, 1, seed=9)[0]
    a[col, col] = bad
    info, _ = potrf(L, a, 256)
    assert info == col + 1


# the right-hand sides' kept tiles: larger and smaller systems in turn
def test_sizes_in_turn(L):
    assert L.plasma_set(pb.PlasmaNb, 64) == 0
    for n, nrhs in [(300, 3), (40, 1), (700, 70), (65, 2), (700, 71), (300, 3)]:
        a, b = gen.likelihood(n, nrhs, seed=n + nrhs)
        for dtype, eps, fn in ((np.float64, EPS, L.plasma_dposv), (np.float32, SEPS, L.plasma_sposv)):
            af, x = np.asfortranarray(a.astype(dtype)), np.asfortranarray(b.astype(dtype))
            assert fn(LO, n, nrhs, af.ctypes.data, n, x.ctypes.data, n) == 0
            r = np.abs(a @ x.astype(np.float64) - b).max()
            assert r <= TOL * eps * n * np.abs(a).sum(1).max() * np.abs(x).max()
