"""The fixed-point solve's device code compiled for the CPU (tests/host)."""
import ctypes
import os
import subprocess
import tempfile

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "vectorized-eigensolver_gb300", "csrc")
_libs = {}


def lib(src="fx_host.cpp"):
    if src not in _libs:
        with tempfile.TemporaryDirectory() as d:
            so = os.path.join(d, "fx_host.so")
            # no contraction, as in the device code's written-out fma: the same bits in every form
            subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-ffp-contract=off", "-fno-strict-aliasing", "-shared", "-fPIC",
                            "-I" + os.path.join(HERE, "host"), "-I" + CSRC, os.path.join(HERE, "host", src), "-o", so],
                           check=True)
            _libs[src] = ctypes.CDLL(so)
    return _libs[src]


def solve(A, form="l1", vec=True, order=0):
    """Solve the batch A (N, n, n) in one block of `form` (l1, l2, l4, l8: lanes
    per matrix in the workspace; g4 .. g64: in shared memory), the threads taking
    turns in the given order.  Returns dict: E, V, ok (0: left to the FP64
    kernels, else 1 + status), sweeps, and error (why the block did not end)."""
    N, n, _ = A.shape
    cols = np.ascontiguousarray(A.transpose(0, 2, 1))
    re, im = np.ascontiguousarray(cols.real), np.ascontiguousarray(cols.imag)
    E, V = np.full((2, N, n), np.nan), np.full((2, N, n, n), np.nan)
    ok, sweeps = np.full(N, -1, np.int32), np.full(N, -1, np.int32)
    msg = ctypes.create_string_buffer(256)
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    lib().fxh_solve(ord(form[0]), int(form[1:]), int(vec), order, n, N, p(re), p(im), p(E[0]), p(E[1]), p(V[0]), p(V[1]),
                    p(ok), p(sweeps), msg)
    return dict(E=E[0] + 1j * E[1], V=(V[0] + 1j * V[1]).transpose(0, 2, 1), ok=ok, sweeps=sweeps, error=msg.value.decode())
