"""How far the factors, solutions and gradients are from the exact ones.

The residual tests elsewhere allow 50 eps; a sum taken in a worse order, or
truncated where it should round, stays far inside that.  Here the error itself
is measured, in units of the rounding unit u (2^-53, 2^-24), in the 2-norm over
all entries, against extended precision (FP64) or FP64 (FP32), on
well-conditioned inputs.  Rounded sums of a few hundred terms leave a few u.
Each limit lies between what the present order of the sums gives and what a
worse one gave; both are stated.
"""
import ctypes

import numpy as np
import pytest
import torch

import gen
import plasma_b200 as pb
from plasma_b200.batched import Batch

pytestmark = pytest.mark.gpu
U64, U32 = 2.0 ** -53, 2.0 ** -24
ld = np.longdouble


@pytest.fixture(scope="module")
def L():
    lib = pb.lib()
    assert lib.plasma_init() == 0
    assert lib.plasma_set(pb.PlasmaTuning, pb.PlasmaDisabled) == 0
    lib.plasma_set_stream(ctypes.c_void_p(1))
    yield lib
    lib.plasma_finalize()


def gram(n, seed, m=None):
    """G G^T / n + I, as the Gaussian likelihood has it."""
    g = np.random.default_rng(seed).standard_normal((n, n))
    a = g @ g.T / n + np.eye(n)
    return (a + a.T) * 0.5


def cholesky(a):
    a, n = a.astype(ld), len(a)
    low = np.zeros_like(a)
    for j in range(n):
        v = a[j:, j] - low[j:, :j] @ low[j, :j]
        low[j, j] = np.sqrt(v[0])
        low[j + 1:, j] = v[1:] / low[j, j]
    return low


def solve(low, b):
    x = b.astype(ld)
    n = len(low)
    for i in range(n):
        x[i] = (x[i] - low[i, :i] @ x[:i]) / low[i, i]
    for i in range(n - 1, -1, -1):
        x[i] = (x[i] - low[i + 1:, i] @ x[i + 1:]) / low[i, i]
    return x


def error(got, want, u):
    want = want.astype(ld)
    return float(np.sqrt(((got.astype(ld) - want) ** 2).sum() / (want ** 2).sum())) / u


def below(m):
    return m[np.tril_indices(len(m), -1)]


# The panel solve and the strips of a diagonal tile: products summed apart from
# the entries, 1.1 to 1.6 u; added to them one by one, 2.8 to 3.3 u.
@pytest.mark.parametrize("nb", [64, 128, 256])
@pytest.mark.parametrize("kind", ["gram", "dominant"])
def test_fp64_factor(L, nb, kind):
    n = 300
    assert L.plasma_set(pb.PlasmaNb, nb) == 0
    a = gram(n, nb) if kind == "gram" else gen.diag_dominant(n, 1, seed=nb)[0]
    f = a.copy(order="F")
    assert L.plasma_dpotrf(pb.PlasmaLower, n, f.ctypes.data, n) == 0
    low = cholesky(a)
    assert error(below(f), below(low), U64) <= 2.0
    assert error(np.diag(f), np.diag(low), U64) <= 1.0


# The one-launch sweeps with a few right-hand sides: sums that end with the
# diagonal's term 2.1 u, sums that begin with it 3.0.
@pytest.mark.parametrize("nrhs", [2, 8, 16])
def test_fp64_sweeps(L, nrhs):
    n, kd = 2000, 300
    assert L.plasma_set(pb.PlasmaNb, 128) == 0
    err = []
    for seed in range(2):
        a, lo, up, b = gen.band(n, kd, nrhs, seed=seed)
        f, x = lo.copy(order="F"), b.copy(order="F")
        assert L.plasma_dpbsv(pb.PlasmaLower, n, kd, nrhs, f.ctypes.data, kd + 1, x.ctypes.data,
                              n) == 0
        err.append(error(x, solve(cholesky(a), b), U64))
    assert np.mean(err) <= 2.5


# FP32 factors through the tensor-core update of (padded) tiles.  Two walks over
# K, the small products first: below the diagonal 3.1 u and the diagonal 1.5 u;
# one walk 4.9 and 1.9.
@pytest.mark.parametrize("n", [2048, 3001])
def test_fp32_factor(L, n):
    assert L.plasma_set(pb.PlasmaNb, 256) == 0
    g = torch.Generator(device="cuda").manual_seed(n)
    z = torch.randn(n, n, generator=g, device="cuda")
    a = z @ z.t() / n
    a = (a + a.t()) * 0.5
    a.diagonal().add_(1.0)
    f = a.clone()
    torch.cuda.synchronize()
    assert L.plasma_spotrf(pb.PlasmaLower, n, f.data_ptr(), n) == 0
    low = torch.linalg.cholesky(a.double())
    d = f.t().double() - low

    def norm(x):
        return x.norm().item()
    assert norm(d.tril(-1)) / norm(low.tril(-1)) / U32 <= 4.0
    assert norm(d.diagonal()) / norm(low.diagonal()) / U32 <= 1.7


# FP32 solves with many right-hand sides (tile inverses on the tensor cores,
# k_diag_mma): A^-1 from identity columns.  Sums that leave the tensor cores
# every 32 terms, the backward ones begun with the diagonal's, 12.3 and 16.8 u;
# every 8 terms and towards the diagonal, whose own terms are rounded, 6.9 and
# 12.1.
@pytest.mark.parametrize("n,nb,limit", [(1536, 128, 7.5), (1100, 256, 14.5)])
def test_fp32_many_rhs(L, n, nb, limit):
    assert L.plasma_set(pb.PlasmaNb, nb) == 0
    a = gram(n, n).astype(np.float32)
    f, x = a.copy(order="F"), np.eye(n, dtype=np.float32, order="F")
    assert L.plasma_sposv(pb.PlasmaLower, n, n, f.ctypes.data, n, x.ctypes.data, n) == 0
    low = np.tril(f).astype(np.float64)               # this call's own factor
    assert error(x, np.linalg.inv(low @ low.T), U32) <= limit


def test_fp32_batched(L):
    """Strips in blocks of 32 rows, orders 100 to 180.  The diagonal's terms of
    the products with 8 x 8 inverses rounded: factor below its diagonal 3.7 u,
    solution 14.3 u, gradient in A 27.7 u; summed on the tensor cores with the
    rest 4.7, 17.8 and 34.7."""
    rng = np.random.default_rng(3)
    sizes = rng.integers(100, 181, 48).astype(np.int32)
    plan = Batch(sizes, dtype=torch.float32)
    oa = np.concatenate([[0], np.cumsum((sizes.astype(np.int64) ** 2 + 31) // 32 * 32)])
    ob = np.concatenate([[0], np.cumsum((sizes.astype(np.int64) + 31) // 32 * 32)])
    A, Lb = np.zeros(oa[-1], np.float32), np.zeros(oa[-1], np.float32)
    B, Xb = np.zeros(ob[-1], np.float32), np.zeros(ob[-1], np.float32)
    for i, n in enumerate(sizes):
        g = rng.standard_normal((n, n))
        a = (g @ g.T / n + 0.1 * np.eye(n)).astype(np.float32)
        A[oa[i]:oa[i] + n * n] = ((a + a.T) / 2).ravel()
        Lb[oa[i]:oa[i] + n * n] = np.tril(rng.standard_normal((n, n))).T.ravel()
        B[ob[i]:ob[i] + n], Xb[ob[i]:ob[i] + n] = rng.standard_normal((2, n))
    d = {k: torch.from_numpy(v.copy()).cuda() for k, v in
         (("F", A), ("X", B), ("GA", Lb), ("GB", Xb))}
    info = plan.info_buffer()
    torch.cuda.synchronize()
    plan.potrf(d["F"], info)
    plan.potrs(d["F"], d["X"])
    plan.potrs_adjoint(d["F"], d["X"], d["GB"], d["GA"])
    plan.potrf_adjoint(d["F"], d["GA"])
    torch.cuda.synchronize()
    assert not info.any()
    h = {k: v.cpu().numpy() for k, v in d.items()}
    got, want = {k: [] for k in d}, {k: [] for k in d}
    for i, n in enumerate(sizes):
        def mat(v):
            return v[oa[i]:oa[i] + n * n].reshape(n, n).T.astype(np.float64)

        def vec(v):
            return v[ob[i]:ob[i] + n].astype(np.float64)
        low = np.linalg.cholesky(mat(A))
        inv = np.linalg.inv(low)
        x, gb = (inv.T @ (inv @ vec(v)) for v in (B, Xb))
        y = np.outer(gb, x)
        p = np.tril(low.T @ (mat(Lb) - np.tril((y + y.T) @ low)))
        p[np.arange(n), np.arange(n)] *= 0.5
        t = inv.T @ p @ inv
        for k, u, v in (("F", below(mat(h["F"])), below(low)), ("X", vec(h["X"]), x),
                        ("GB", vec(h["GB"]), gb), ("GA", mat(h["GA"]), (t + t.T) / 2)):
            got[k].append(np.ravel(u))
            want[k].append(np.ravel(v))
    err = {k: error(np.concatenate(got[k]), np.concatenate(want[k]), U32) for k in got}
    assert err["F"] <= 4.2 and err["X"] <= 16.5 and err["GB"] <= 17.0 and err["GA"] <= 31.0, err
