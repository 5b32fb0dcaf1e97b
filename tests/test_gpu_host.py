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
        pin = torch.from_numpy(a.copy()).pin_memory()
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
            pin.copy_(torch.from_numpy(a))
            return pin, pin.data_ptr()
        print(best(pageable), best(locked))
        """, env)
    pageable, locked = map(float, out.split())
    assert pageable <= 4 * locked
