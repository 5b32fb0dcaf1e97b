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
# L itself, over most of FP32's exponent range.
@pytest.mark.parametrize("n,nb", [(1024, 256), (768, 128)])
@pytest.mark.parametrize("spread", [0, 12, 55])
def test_fp32_row_scales(L, n, nb, spread):
    rng = np.random.default_rng(n + spread)
    a = gen.likelihood(n, 1, seed=11)[0].astype(np.float32).astype(np.float64)
    d = 2.0 ** rng.integers(-spread, spread + 1, n)
    info, f = potrf(L, a * d[:, None] * d[None, :], nb, np.float32)
    assert info == 0
    low = np.tril(f).astype(np.float64) / d[:, None]
    # (i,j) of D A D = (D L)(D L)^T to n eps32 d_i d_j sqrt(a_ii a_jj)
    err = np.abs(low @ low.T - a) / np.sqrt(np.outer(np.diag(a), np.diag(a)))
    assert err.max() <= 4 * np.sqrt(n) * SEPS


# an indefinite matrix whose rows outgrow their scale fails where LAPACK does
def test_fp32_indefinite_info(L):
    n = 1024
    a = gen.likelihood(n, 1, seed=13)[0]
    a[700, :300] = a[:300, 700] = 1e6
    a[900, :300] = a[:300, 900] = 1e30
    for nb in (128, 256):
        info, _ = potrf(L, a, nb, np.float32)
        assert info == 701
