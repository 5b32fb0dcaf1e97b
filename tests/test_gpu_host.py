"""LAPACK-layout calls on a C program's own (pageable) arrays, each in a process
of its own: the staging copies are the library's first use of threads there.
"""
import os
import subprocess
import sys
import textwrap

import pytest
import torch  # noqa: F401  (CUDA context)

from conftest import ROOT

pytestmark = pytest.mark.gpu


def child(code, env=None):
    """Runs `code` (with L, pb, np, torch, ct) and returns its output."""
    pre = f"""
        import sys, ctypes as ct, time
        sys.path.insert(0, {ROOT!r})
        import numpy as np, torch
        import plasma_b200 as pb
        L = pb.lib()
        assert L.plasma_init() == 0
        """
    r = subprocess.run([sys.executable, "-c", textwrap.dedent(pre) + textwrap.dedent(code)],
                       env=dict(os.environ, **(env or {})), capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout


@pytest.mark.parametrize("policy", ["", "active"])
def test_pageable_keeps_pace(policy):
    """The copy threads leave the calling thread and CUDA's callback thread a
    CPU each, whatever the OpenMP runtime's waiting policy: dpotrf on pageable
    arrays takes about what it takes on page-locked ones (7 ms each on the
    B200 hosts).  With a team as large as the machine it took 240 ms; four
    times is far from both."""
    env = {"OMP_WAIT_POLICY": policy} if policy else {}
    out = child("""
        n = 4100
        a = np.full((n, n), 0.25) + n * np.eye(n)
        # (numpy only: a parallel region of torch on this thread is another team,
        # and the runtime waits in another way once there are two)
        pin = torch.empty(n, n, dtype=torch.float64, pin_memory=True).numpy()
        def best(make):
            t = []
            for _ in range(6):
                x, p = make()
                t0 = time.perf_counter()
                assert L.plasma_dpotrf(pb.PlasmaLower, n, p, n) == 0
                t.append(time.perf_counter() - t0)
            return min(t)
        def pageable():
            x = a.copy()
            return x, x.ctypes.data
        def locked():
            pin[...] = a
            return pin, pin.ctypes.data
        print(best(pageable), best(locked))
        """, env)
    pageable, locked = map(float, out.split())
    assert pageable <= 4 * locked


def test_no_host_memory(tmp_path):
    """dsposv out of host memory reports it before it has enqueued a copy of
    the caller's matrix: what still read the arrays after the call failed
    would show as launches of the upload's kernels (one per column group)."""
    shim = tmp_path / "shim.c"
    shim.write_text("""
        #include <errno.h>
        #include <stddef.h>
        extern void *__libc_malloc(size_t);
        static size_t refuse;
        void refuse_malloc(size_t n) { refuse = n; }
        size_t refusal_left(void) { return refuse; }
        void *malloc(size_t n)
        {
            if (n != 0 && n == refuse) { refuse = 0; errno = ENOMEM; return NULL; }
            return __libc_malloc(n);
        }
        """)
    so = tmp_path / "shim.so"
    subprocess.run(["gcc", "-shared", "-fPIC", "-fno-builtin", "-o", str(so), str(shim)],
                   check=True)
    child("""
        n, nb = 5000, 192
        L.plasma_set(pb.PlasmaTuning, pb.PlasmaDisabled)
        L.plasma_set(pb.PlasmaNb, nb)
        a = np.full((n, n), 0.25) + n * np.eye(n)
        b, x, it = np.ones((1, n)), np.zeros((1, n)), ct.c_int()
        def solve():
            return L.plasma_dsposv(pb.PlasmaLower, n, 1, a.ctypes.data, n, b.ctypes.data, n,
                                   x.ctypes.data, n, ct.byref(it))
        assert solve() == 0
        self = ct.CDLL(None)
        self.refuse_malloc.argtypes, self.refusal_left.restype = [ct.c_size_t], ct.c_size_t
        before = L.plasma_kernel_launches()
        self.refuse_malloc(4 * ((n + nb - 1) // nb * nb))       # one float a row
        rc = solve()
        assert self.refusal_left() == 0
        assert rc == pb.PlasmaErrorOutOfMemory, rc
        assert L.plasma_kernel_launches() - before < 10
        assert solve() == 0 and np.abs(x @ a - b).max() < 1e-12
        """, {"LD_PRELOAD": str(so)})


MEMORY = """
        MB = 1 << 20
        L.plasma_set(pb.PlasmaTuning, pb.PlasmaDisabled)
        L.plasma_set(pb.PlasmaNb, 256)
        def free():
            torch.cuda.synchronize()
            return torch.cuda.mem_get_info()[0]
        def spd(n, dtype=torch.float64):
            return torch.full((n, n), 0.25, device="cuda", dtype=dtype) + \\
                   n * torch.eye(n, device="cuda", dtype=dtype)
        def factor(a):
            return L.plasma_dpotrf(pb.PlasmaLower, a.shape[0], a.data_ptr(), a.shape[0])
        held = []
        def leave(mb):
            torch.cuda.empty_cache()
            held.append(torch.empty(max(free() - mb * MB, 0), dtype=torch.uint8, device="cuda"))
            return free() // MB
        assert factor(spd(5000)) == 0            # loads the kernels
        """


def test_scratch_that_just_fits():
    """A tile copy that fits, but not with an eighth on top, is allocated at
    its own size: n = 20000 packed takes 1580 MB, 197 more with headroom."""
    child(MEMORY + """
        a = spd(20000)
        L.plasma_set_stream(ct.c_void_p(1))
        kept = free()
        left = leave(1640)
        assert 1600 <= left <= 1740, left
        assert factor(a) == 0
        """)


def test_idle_slots_give_way():
    """Right-hand sides that an earlier call left in their slot do not keep a
    later call from the memory it needs."""
    child(MEMORY + """
        n, nrhs = 4096, 24000                   # 752 MiB of right-hand sides
        f, b = spd(n), torch.ones(nrhs, n, device="cuda", dtype=torch.float64)
        L.plasma_set_stream(ct.c_void_p(1))
        assert L.plasma_dposv(pb.PlasmaLower, n, nrhs, f.data_ptr(), n, b.data_ptr(), n) == 0
        del f, b
        a = spd(20000)
        left = leave(1000)
        assert left <= 1100, left
        assert factor(a) == 0
        """)


def test_large_operands_are_returned():
    """Right-hand sides and adjoint operands above 1 GiB do not stay allocated
    after the call: what remains of an adjoint is its n x n work matrices."""
    child(MEMORY + """
        n = 12288                               # 1152 MiB a matrix
        a = spd(n)
        L.plasma_set_stream(ct.c_void_p(1))
        g = torch.eye(n, device="cuda", dtype=torch.float64)
        torch.cuda.empty_cache()
        before = free()
        assert L.plasma_dpotrf_adjoint(pb.PlasmaLower, n, a.data_ptr(), n, g.data_ptr(), n) == 0
        assert before - free() <= 2 * 1152 * 1.125 * MB + 256 * MB
        """)
