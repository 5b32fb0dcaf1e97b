"""The work that programs hand to plasma_b200, case by case, for timing.

Each case is one call (or one forward and backward pass) through the public
entry points: the C ABI through ``plasma_b200.lib()``, the batched plans of
``plasma_b200.batched`` and the autograd binding.  Sizes and input
distributions are those of the test generators and of bench.py: diagonally
dominant systems, prescribed spectra, the Gaussian likelihood, uneven batches,
band and general systems, from one tile up to n = 32768, with orders that are
no multiple of a tile among them.

Kinds of case:
  posv   plasma_?posv on device arrays: a Cholesky factor and the solve of a
         few right-hand sides, either triangle.  The routine overwrites A and
         B, so a pass copies both from the program's own arrays first, as a
         program that still needs its matrix does.
  mixed  plasma_dsposv (low-precision factor, FP64 refinement), on device or
         on ordinary host arrays; A and B are left as they are.
  nll    logdet(A) + tr(B^T A^-1 B) and its gradients in A and B (autograd).
  batch  thousands of uneven systems in one plan: "posv" solves them, "grad"
         factors, solves and runs both adjoints.
  pbsv   a band system in LAPACK band storage (plasma_dpbsv).
  gesv   plasma_dsgesv, the LU-based mixed-precision solve.
"""
import ctypes
import math

import numpy as np
import torch

import plasma_b200 as pb
from plasma_b200 import autograd as pba
from plasma_b200.batched import Batch

_LEGACY_STREAM = 1      # cudaStreamLegacy: orders the library with torch's work


# --------------------------------------------------------------------- cases
def listed():
    return [
        # one small system: the latency of a whole call on a few tiles
        {"name": "posv_f64_n300", "kind": "posv", "dtype": "f64", "n": 300, "nrhs": 1,
         "upper": False},
        # the parity configuration's size
        {"name": "posv_f64_n2048", "kind": "posv", "dtype": "f64", "n": 2048, "nrhs": 1,
         "upper": False},
        # the plain FP64 solver's smallest and middle benchmark size
        {"name": "posv_f64_n8192", "kind": "posv", "dtype": "f64", "n": 8192, "nrhs": 16,
         "upper": False},
        {"name": "posv_f64_n16384", "kind": "posv", "dtype": "f64", "n": 16384, "nrhs": 16,
         "upper": False},
        # single precision, a ragged order, the other triangle
        {"name": "posv_f32_n5003_upper", "kind": "posv", "dtype": "f32", "n": 5003, "nrhs": 3,
         "upper": True},
        # the mixed-precision benchmark, and a mid-sized ragged call on a C
        # program's own malloc'ed arrays
        {"name": "mixed_n32768", "kind": "mixed", "n": 32768, "nrhs": 1, "logk": 5,
         "host": False},
        {"name": "mixed_host_n4100", "kind": "mixed", "n": 4100, "nrhs": 1, "logk": 2,
         "host": True},
        # a Gaussian-process training step: likelihood and gradients
        {"name": "nll_f64_n4096", "kind": "nll", "dtype": "f64", "n": 4096, "nrhs": 8},
        # many small systems at once: solve, and solve with gradients
        {"name": "batch_posv_f64", "kind": "batch", "dtype": "f64", "count": 4096,
         "nmin": 16, "nmax": 512, "op": "posv"},
        {"name": "batch_grad_f32", "kind": "batch", "dtype": "f32", "count": 1024,
         "nmin": 16, "nmax": 512, "op": "grad"},
        # a long band system, and a general one
        {"name": "pbsv_n32768_kd1024", "kind": "pbsv", "n": 32768, "kd": 1024, "nrhs": 1},
        {"name": "gesv_n4096", "kind": "gesv", "n": 4096, "nrhs": 1},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["posv", "posv", "posv", "mixed", "mixed", "nll", "batch", "batch",
                       "pbsv", "gesv"])
    if kind == "posv":
        return {"kind": kind, "dtype": rng.choice(["f64", "f64", "f32"]),
                "n": _logint(rng, 200, 16384), "nrhs": rng.choice([1, 1, 2, 5, 16, 24]),
                "upper": rng.random() < 0.4}
    if kind == "mixed":
        host = rng.random() < 0.3
        return {"kind": kind, "n": _logint(rng, 400, 6000 if host else 24000),
                "nrhs": rng.choice([1, 1, 2]), "logk": rng.choice([1, 2, 3, 4, 5]),
                "host": host}
    if kind == "nll":
        return {"kind": kind, "dtype": rng.choice(["f64", "f64", "f32"]),
                "n": _logint(rng, 256, 6000), "nrhs": rng.choice([2, 4, 8, 17])}
    if kind == "batch":
        nmax = rng.choice([64, 200, 333, 512])
        return {"kind": kind, "dtype": rng.choice(["f64", "f32"]),
                "count": _logint(rng, 256, 4096), "nmin": rng.choice([1, 16]),
                "nmax": nmax, "op": rng.choice(["posv", "posv", "grad"])}
    if kind == "pbsv":
        n = _logint(rng, 2000, 32768)
        return {"kind": kind, "n": n, "kd": _logint(rng, 16, min(2048, n // 2)),
                "nrhs": rng.choice([1, 1, 2])}
    return {"kind": kind, "n": _logint(rng, 300, 6000), "nrhs": rng.choice([1, 1, 2])}


def _dtype(case):
    return torch.float32 if case.get("dtype") == "f32" else torch.float64


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


# -------------------------------------------------------------------- inputs
# Column-major arrays: a torch tensor of shape (columns, rows).

def _diag_dominant(n, nrhs, dtype, g):
    """sym(U[-0.5, 0.5]) + n I and U[-1, 1]."""
    a = torch.rand(n, n, generator=g, device="cuda", dtype=dtype) - 0.5
    for i in range(0, n, 2048):                    # mirror the triangle, in place
        j = min(i + 2048, n)
        a[i:j, j:] = a[j:, i:j].t()
        blk = torch.tril(a[i:j, i:j])
        a[i:j, i:j] = blk + torch.tril(blk, -1).t()
    a.diagonal().add_(float(n))
    b = torch.rand(nrhs, n, generator=g, device="cuda", dtype=dtype) * 2 - 1
    return a, b


def _hartley_rows(a):
    """The orthogonal, symmetric Hartley transform of every row, in place."""
    n = a.shape[1]
    step = max(1, (1 << 27) // n)
    for i in range(0, a.shape[0], step):
        f = torch.fft.rfft(a[i:i + step], dim=1)
        lo = f[:, :n // 2 + 1]
        full = lo.real - lo.imag
        tail = torch.conj(f[:, 1:(n + 1) // 2]).flip(1)
        a[i:i + step] = torch.cat([full, tail.real - tail.imag], 1) / math.sqrt(n)


def _spectrum(n, logk, g):
    """A = Q diag(lambda) Q^T, lambda log-spaced from 1 to 10^-logk in random
    order, Q = H S1 H S2 (Hartley transforms and random signs): dense and
    without structure, in O(n^2 log n)."""
    lam = torch.logspace(0.0, -float(logk), n, device="cuda", dtype=torch.float64)
    lam = lam[torch.randperm(n, generator=g, device="cuda")]
    a = torch.diag(lam)
    for _ in range(2):
        _hartley_rows(a)
        _transpose_(a)
        _hartley_rows(a)
        s = (torch.randint(0, 2, (n,), generator=g, device="cuda") * 2 - 1).double()
        a.mul_(s[:, None]).mul_(s[None, :])
    return _symmetrize_(a)


def _transpose_(a):
    for i in range(0, a.shape[0], 4096):
        a[i:i + 4096, i:i + 4096] = a[i:i + 4096, i:i + 4096].t().clone()
        t = a[i:i + 4096, i + 4096:].clone()
        a[i:i + 4096, i + 4096:] = a[i + 4096:, i:i + 4096].t()
        a[i + 4096:, i:i + 4096] = t.t()


def _symmetrize_(a):
    for i in range(0, a.shape[0], 4096):
        d = a[i:i + 4096, i:i + 4096]
        d.copy_((d + d.t()) * 0.5)
        a[i:i + 4096, i + 4096:] = a[i + 4096:, i:i + 4096].t()
    return a


def _mixed_inputs(case, seed):
    g = _gen(seed)
    n, nrhs = case["n"], case["nrhs"]
    a = _spectrum(n, case["logk"], g)
    x = torch.randn(nrhs, n, generator=g, device="cuda", dtype=torch.float64)
    return a, x @ a


def _likelihood_inputs(case, seed):
    """A = G G^T / n + I and B ~ N(0, 1)."""
    g = _gen(seed)
    n, dt = case["n"], _dtype(case)
    m = torch.randn(n, n, generator=g, device="cuda", dtype=dt)
    a = m @ m.t() / n
    a = (a + a.t()) * 0.5
    a.diagonal().add_(1.0)
    b = torch.randn(n, case["nrhs"], generator=g, device="cuda", dtype=dt)
    return a, b


def _batch_sizes(case):
    """The orders are the program's own and stay from batch to batch."""
    rng = np.random.default_rng(5)
    return rng.integers(case["nmin"], case["nmax"] + 1, case["count"]).astype(np.int32)


def _offsets(lengths):
    """Starts of the packed parts, each on a multiple of 32 elements, and the
    length of the whole (the layout of plasma_batch_offsets)."""
    padded = (lengths.astype(np.int64) + 31) // 32 * 32
    return np.concatenate([[0], np.cumsum(padded)])


def _groups(sizes):
    """Indices of the systems in groups of similar order."""
    order = np.argsort(sizes, kind="stable")
    return [order[i:i + 256] for i in range(0, len(order), 256)]


def _batch_inputs(case, seed):
    """Groups of padded systems (the packing of the plan is prepare's): per
    group (indices, A, b, Lbar, Xbar) with A = G G^T / n + 0.1 I, padded to
    the group's largest order by the identity."""
    g = _gen(seed)
    sizes = _batch_sizes(case)
    dt = _dtype(case)
    out = []
    for idx in _groups(sizes):
        k = torch.from_numpy(sizes[idx].astype(np.int64)).cuda()
        m = int(sizes[idx].max())
        inside = torch.arange(m, device="cuda")[None, :] < k[:, None]
        both = inside[:, :, None] & inside[:, None, :]
        z = torch.randn(len(idx), m, m, generator=g, device="cuda", dtype=torch.float64)
        z = torch.where(both, z, 0)
        a = z @ z.transpose(1, 2) / k[:, None, None]
        a.diagonal(dim1=1, dim2=2).add_(torch.where(inside, 0.1, 1.0))
        b, xb = (torch.where(inside, torch.randn(len(idx), m, generator=g, device="cuda",
                                                 dtype=torch.float64), 0) for _ in range(2))
        lb = torch.randn(len(idx), m, m, generator=g, device="cuda", dtype=torch.float64)
        lb = torch.where(both, lb, 0).tril()
        out.append((idx, a.to(dt), b.to(dt), lb.to(dt), xb.to(dt)))
    return sizes, out


def _pack(sizes, groups, which, vector):
    """Group arrays packed as a plan lays them out (column-major)."""
    off = _offsets(sizes if vector else sizes.astype(np.int64) ** 2)
    buf = torch.zeros(int(off[-1]), dtype=groups[0][1].dtype, device="cuda")
    for grp in groups:
        src = grp[which]
        for j, i in enumerate(grp[0]):
            n = int(sizes[i])
            if vector:
                buf[off[i]:off[i] + n] = src[j, :n]
            else:
                buf[off[i]:off[i] + n * n].view(n, n).copy_(src[j, :n, :n].t())
    return buf


def _band_inputs(case, seed):
    """LAPACK lower band storage (columns x (kd + 1)) of U[-0.5, 0.5] with
    2 kd + 1 added to the diagonal, and U[-1, 1]."""
    g = _gen(seed)
    n, kd = case["n"], case["kd"]
    ab = torch.rand(n, kd + 1, generator=g, device="cuda", dtype=torch.float64) - 0.5
    ab[:, 0] += 2 * kd + 1
    rows = torch.arange(n, device="cuda")[:, None] + torch.arange(kd + 1, device="cuda")
    ab[rows >= n] = 0
    b = torch.rand(case["nrhs"], n, generator=g, device="cuda", dtype=torch.float64) * 2 - 1
    return ab, b


def _general_inputs(case, seed):
    g = _gen(seed)
    n = case["n"]
    a = torch.rand(n, n, generator=g, device="cuda", dtype=torch.float64) - 0.5
    b = torch.rand(case["nrhs"], n, generator=g, device="cuda", dtype=torch.float64) * 2 - 1
    return a, b


# --------------------------------------------------------------- the program
def _library():
    L = pb.lib()
    rc = L.plasma_init()
    if rc not in (0, pb.PlasmaErrorNotInitialized):     # the latter: already up
        raise RuntimeError(f"plasma_init failed: {rc}")
    L.plasma_set_stream(ctypes.c_void_p(_LEGACY_STREAM))
    return L


def _ok(rc, what):
    if rc != 0:
        raise RuntimeError(f"{what} returned {rc}")


def prepare(case, seed):
    L = _library()
    kind = case["kind"]
    s = {"L": L, "case": case}
    if kind == "posv":
        s["A"], s["B"] = _diag_dominant(case["n"], case["nrhs"], _dtype(case), _gen(seed))
        s["F"], s["X"] = torch.empty_like(s["A"]), torch.empty_like(s["B"])
    elif kind == "mixed":
        a, b = _mixed_inputs(case, seed)
        if case["host"]:
            s["A"], s["B"] = a.cpu().numpy(), b.cpu().numpy()
            s["X"] = np.zeros_like(s["B"])
        else:
            s["A"], s["B"] = a, b
            s["X"] = torch.empty_like(b)
        s["iter"] = ctypes.c_int(0)
    elif kind == "nll":
        a, b = _likelihood_inputs(case, seed)
        s["A"], s["B"] = a.requires_grad_(True), b.requires_grad_(True)
    elif kind == "batch":
        sizes, groups = _batch_inputs(case, seed)
        plan = Batch(sizes, dtype=_dtype(case))
        if (int(_offsets(sizes.astype(np.int64) ** 2)[-1]) != plan.matrix_elems
                or int(_offsets(sizes)[-1]) != plan.vector_elems):
            raise RuntimeError("the plan's layout is another one")
        s["plan"] = plan
        s["A"] = _pack(sizes, groups, 1, False)
        s["B"] = _pack(sizes, groups, 2, True)
        s["F"], s["X"] = torch.empty_like(s["A"]), torch.empty_like(s["B"])
        s["info"] = plan.info_buffer()
        if case["op"] == "grad":
            s["Lbar"] = _pack(sizes, groups, 3, False)
            s["Xbar"] = _pack(sizes, groups, 4, True)
            s["GA"], s["GB"] = torch.empty_like(s["A"]), torch.empty_like(s["B"])
    elif kind == "pbsv":
        s["A"], s["B"] = _band_inputs(case, seed)
        s["F"], s["X"] = torch.empty_like(s["A"]), torch.empty_like(s["B"])
    else:
        s["A"], s["B"] = _general_inputs(case, seed)
        s["X"] = torch.empty_like(s["B"])
        s["ipiv"] = np.zeros(case["n"], dtype=np.int32)
        s["iter"] = ctypes.c_int(0)
    return s


def run(s):
    case, L = s["case"], s["L"]
    kind = case["kind"]
    if kind == "posv":
        n, nrhs = case["n"], case["nrhs"]
        s["F"].copy_(s["A"])
        s["X"].copy_(s["B"])
        fn = L.plasma_sposv if case["dtype"] == "f32" else L.plasma_dposv
        uplo = pb.PlasmaUpper if case["upper"] else pb.PlasmaLower
        _ok(fn(uplo, n, nrhs, s["F"].data_ptr(), n, s["X"].data_ptr(), n), "posv")
        return {"F": s["F"], "X": s["X"]}
    if kind == "mixed":
        n = case["n"]
        A, B, X = (pb.ptr(s[k]) for k in "ABX")
        _ok(L.plasma_dsposv(pb.PlasmaLower, n, case["nrhs"], A, n, B, n, X, n,
                            ctypes.byref(s["iter"])), "dsposv")
        return {"X": s["X"]}
    if kind == "nll":
        f = pba.gaussian_nll(s["A"], s["B"])
        gA, gB = torch.autograd.grad(f, (s["A"], s["B"]))
        return {"f": f.detach(), "gA": gA, "gB": gB}
    if kind == "batch":
        plan = s["plan"]
        s["F"].copy_(s["A"])
        s["X"].copy_(s["B"])
        if case["op"] == "posv":
            plan.posv(s["F"], s["X"], s["info"])
            return {"F": s["F"], "X": s["X"], "info": s["info"]}
        s["GA"].copy_(s["Lbar"])
        s["GB"].copy_(s["Xbar"])
        plan.potrf(s["F"], s["info"])
        plan.potrs(s["F"], s["X"])
        plan.potrs_adjoint(s["F"], s["X"], s["GB"], s["GA"])
        plan.potrf_adjoint(s["F"], s["GA"])
        return {"F": s["F"], "X": s["X"], "GA": s["GA"], "GB": s["GB"], "info": s["info"]}
    if kind == "pbsv":
        n, kd = case["n"], case["kd"]
        s["F"].copy_(s["A"])
        s["X"].copy_(s["B"])
        _ok(L.plasma_dpbsv(pb.PlasmaLower, n, kd, case["nrhs"], s["F"].data_ptr(), kd + 1,
                           s["X"].data_ptr(), n), "pbsv")
        return {"F": s["F"], "X": s["X"]}
    # the pivots are left out: the FP32 factor's choice between entries that
    # agree to its rounding is free, and one other choice renumbers the rest
    n = case["n"]
    _ok(L.plasma_dsgesv(n, case["nrhs"], s["A"].data_ptr(), n, s["ipiv"].ctypes.data,
                        s["B"].data_ptr(), n, s["X"].data_ptr(), n, ctypes.byref(s["iter"])),
        "dsgesv")
    return {"X": s["X"]}


# ---------------------------------------------------------- what it must cost
def _mean_power(case, p):
    lo, hi = case["nmin"], case["nmax"]
    return sum(float(k) ** p for k in range(lo, hi + 1)) / (hi - lo + 1)


def work(case):
    kind = case["kind"]
    e = 4 if case.get("dtype") == "f32" else 8
    n, r = float(case.get("n", 0)), float(case.get("nrhs", 1))
    if kind == "posv":         # one triangle in, its factor out; the solve
        return {"bytes": e * (n * (n + 1) + 2 * n * r), "flops": n ** 3 / 3 + 2 * n * n * r}
    if kind == "mixed":
        return {"bytes": 8 * (n * (n + 1) / 2 + 2 * n * r),
                "flops": n ** 3 / 3 + 2 * n * n * r}
    if kind == "nll":          # the factor, the solve, the inverse (2/3 n^3)
        return {"bytes": e * (2 * n * n + 3 * n * r), "flops": n ** 3 + 6 * n * n * r}
    if kind == "batch":
        c, m1, m2, m3 = float(case["count"]), *(_mean_power(case, p) for p in (1, 2, 3))
        if case["op"] == "posv":
            return {"bytes": c * e * (m2 + 2 * m1), "flops": c * (m3 / 3 + 2 * m2)}
        # factor and solve; the solve's adjoint (8 n^2); the factor's (n^3)
        return {"bytes": c * e * (2.5 * m2 + 4 * m1), "flops": c * (4 * m3 / 3 + 10 * m2)}
    if kind == "pbsv":
        kd = float(case["kd"])
        return {"bytes": 8 * (2 * n * (kd + 1) + 2 * n * r),
                "flops": n * kd * kd + 4 * n * kd * r}
    return {"bytes": 8 * (n * n + 2 * n * r), "flops": 2 * n ** 3 / 3 + 2 * n * n * r}


def tolerance(case):
    kind = case["kind"]
    if kind == "mixed":
        # the refinement stops at ||r|| <= sqrt(n) eps ||A|| ||x||
        n, kappa = case["n"], 10.0 ** case["logk"]
        return {"rel": 2.0 * kappa * math.sqrt(n) * 2.2e-16 + 1e-13, "max": 1e-5}
    if kind == "gesv":         # the same stopping rule, kappa about 1e4 to 1e6
        return {"rel": 1e-8, "max": 1e-6}
    if case.get("dtype") == "f32":
        # seen against 64 bits: 2e-7 (posv), 2e-6 (batch), 1e-5 (nll)
        return {"rel": {"posv": 2e-6, "batch": 1e-5, "nll": 1e-4}[kind]}
    # seen: 4e-15 (posv, pbsv), 3e-15 (batch), 5e-15 (nll)
    return {"rel": 2e-14}


# ------------------------------------------------------------ in 64 bits
def exact(case, seed):
    kind = case["kind"]
    if kind == "posv":
        n = case["n"]
        a, b = _diag_dominant(n, case["nrhs"], _dtype(case), _gen(seed))
        a, b = a.double(), b.double()
        low = torch.linalg.cholesky(a)
        x = torch.cholesky_solve(b.t(), low).t()
        # (columns, rows): the stored triangle of a column-major lower factor
        # is the upper one of this tensor
        if case["upper"]:
            f = torch.tril(low) + torch.triu(a, 1)
        else:
            f = torch.triu(low.t()) + torch.tril(a, -1)
        return {"F": f, "X": x.contiguous()}
    if kind == "mixed":
        a, b = _mixed_inputs(case, seed)
        x = torch.cholesky_solve(b.t(), torch.linalg.cholesky(a)).t().contiguous()
        return {"X": x.cpu().numpy() if case["host"] else x}
    if kind == "nll":
        a, b = (t.double() for t in _likelihood_inputs(case, seed))
        low = torch.linalg.cholesky(a)
        x = torch.cholesky_solve(b, low)
        f = 2 * torch.log(torch.diagonal(low)).sum() + (b * x).sum()
        return {"f": f, "gA": torch.cholesky_inverse(low) - x @ x.t(), "gB": 2 * x}
    if kind == "batch":
        return _exact_batch(case, seed)
    if kind == "pbsv":
        return _exact_band(case, seed)
    a, b = _general_inputs(case, seed)
    return {"X": torch.linalg.solve(a.t(), b.t()).t().contiguous()}


def _exact_batch(case, seed):
    sizes, groups = _batch_inputs(case, seed)
    outs = []
    for idx, a, b, lb, xb in groups:
        a, b, lb, xb = a.double(), b.double(), lb.double(), xb.double()
        low = torch.linalg.cholesky(a)
        x = torch.cholesky_solve(b[:, :, None], low)[:, :, 0]
        f = low + torch.triu(a, 1)
        if case["op"] == "posv":
            outs.append((idx, f, x))
            continue
        gb = torch.cholesky_solve(xb[:, :, None], low)[:, :, 0]
        y = gb[:, :, None] * x[:, None, :]
        lb = lb - torch.tril((y + y.transpose(1, 2)) @ low)
        p = torch.tril(low.transpose(1, 2) @ lb)
        p.diagonal(dim1=1, dim2=2).mul_(0.5)
        t = torch.linalg.solve_triangular(low.transpose(1, 2), p, upper=True)
        t = torch.linalg.solve_triangular(low, t, upper=False, left=False)
        outs.append((idx, f, x, (t + t.transpose(1, 2)) * 0.5, gb))
    names = ["F", "X", "GA", "GB"]
    got = {names[w - 1]: _pack(sizes, outs, w, w in (2, 4))
           for w in range(1, len(outs[0]))}
    got["info"] = torch.zeros(len(sizes), dtype=torch.int32, device="cuda")
    return got


def _exact_band(case, seed):
    """Block tridiagonal Cholesky with blocks at least as wide as the band."""
    ab, b = _band_inputs(case, seed)
    n, kd = case["n"], case["kd"]
    w = max(kd, 256)
    rows = torch.arange(n, device="cuda")[:, None] + torch.arange(kd + 1, device="cuda")

    def block(i, j, ni, nj):                        # A[i:i+ni, j:j+nj], i >= j
        r = torch.arange(i, i + ni, device="cuda")[:, None]
        c = torch.arange(j, j + nj, device="cuda")[None, :]
        d = r - c
        inside = (d >= 0) & (d <= kd)
        return torch.where(inside, ab[c.expand_as(d), d.clamp(0, kd)], 0.0)

    fac = torch.zeros_like(ab)
    starts = list(range(0, n, w))
    x = b.t().clone()
    diag, low = [], []
    carry = None
    for i in starts:
        m = min(w, n - i)
        d = block(i, i, m, m)
        d = d + torch.tril(d, -1).t()
        if carry is not None:
            d = d - carry @ carry.t()
            x[i:i + m] -= carry @ x[i - w:i]
        ld = torch.linalg.cholesky(d)
        x[i:i + m] = torch.linalg.solve_triangular(ld, x[i:i + m], upper=False)
        diag.append(ld)
        m2 = min(w, n - i - m)
        both = ld
        if m2 > 0:
            e = block(i + m, i, m2, m)
            carry = torch.linalg.solve_triangular(ld, e.t(), upper=False).t()
            low.append(carry)
            both = torch.cat([ld, carry], 0)
        c = torch.arange(m, device="cuda")[:, None]
        r = c + torch.arange(kd + 1, device="cuda")[None, :]
        ok = r < both.shape[0]
        fac[i:i + m] = torch.where(ok, both[r.clamp(max=both.shape[0] - 1), c.expand_as(r)], 0.0)
    for t in range(len(starts) - 1, -1, -1):
        i = starts[t]
        m = min(w, n - i)
        if t + 1 < len(starts):
            x[i:i + m] -= low[t].t() @ x[i + m:i + m + low[t].shape[0]]
        x[i:i + m] = torch.linalg.solve_triangular(diag[t].t(), x[i:i + m], upper=True)
    fac[rows >= n] = 0
    return {"F": fac, "X": x.t().contiguous()}
