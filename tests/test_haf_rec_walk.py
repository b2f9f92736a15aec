"""The walk of the hafnian recursion (gbskernels_b200/csrc/haf_rec.cuh) on the CPU: the
kernel's own layout, lane and node functions drive a sequential walk
(tests/rec_host.cu) whose every access must lie inside the workspace the planner asks
for and read a written word, for every split into blocks, and whose sums must equal the
oracle's hafnian / loop hafnian.  The double-double walk's layout and steps too: there no
lane may touch a word that another one writes before the next barrier."""

from __future__ import annotations

import ctypes
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

HERE = Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def reclib():
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if Path("/usr/local/cuda/bin/nvcc").exists() else None)
    if nvcc is None:
        pytest.skip("nvcc not available")
    out = HERE / "_build" / "librechost.so"
    out.parent.mkdir(exist_ok=True)
    src = HERE / "rec_host.cu"
    csrc = HERE.parent / "gbskernels_b200" / "csrc"
    deps = [src, *csrc.glob("*.cuh")]
    if not out.exists() or out.stat().st_mtime < max(p.stat().st_mtime for p in deps):
        cmd = [nvcc, "-x", "cu", "-O2", "-std=c++17", "--expt-relaxed-constexpr", "-shared", "-Xcompiler", "-fPIC",
               "-gencode", "arch=compute_100a,code=sm_100a", "-I", str(csrc), str(src), "-o", str(out)]
        subprocess.run(cmd, check=True, capture_output=True)
    lib = ctypes.CDLL(str(out))
    lib.t_haf_rec_sum.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_int, ctypes.c_uint,
                                  ctypes.c_int, ctypes.c_void_p]
    return lib


def _sum(lib, A, loop, is_dd, lo, clog):
    A = np.ascontiguousarray(A, dtype=np.complex128)
    out = np.zeros(2)
    bad = lib.t_haf_rec_sum(A.ctypes.data, A.shape[0] // 2, int(loop), is_dd, lo, clog, out.ctypes.data)
    assert bad == 0, (A.shape, loop, is_dd, lo, clog, bad)
    return complex(out[0], out[1])


def _sym(N, seed):
    g = np.random.default_rng(seed)
    X = g.standard_normal((N, N)) + 1j * g.standard_normal((N, N))
    return (X + X.T) / 4


@pytest.mark.parametrize("is_dd", [0, 1])
@pytest.mark.parametrize("n", range(1, 11))
def test_sums_equal_the_oracle_for_every_split(reclib, orc, n, is_dd):
    A = _sym(2 * n, n)
    for loop in (False, True):
        t, absn = getattr(orc, "lhaf" if loop else "haf")(A, "quad", with_absnorm=True)
        for clog in range(n + 1):
            v = sum(_sum(reclib, A, loop, is_dd, lo, clog) for lo in range(0, 1 << n, 1 << clog))
            # the recursion's terms are smaller than the power trace's (absn), so their
            # rounding stays within a few n u of absn
            assert abs(v - t) <= 32 * n * 2.0 ** -53 * absn, (loop, clog)


@pytest.mark.parametrize("is_dd", [0, 1])
@pytest.mark.parametrize("n", [11, 12, 13, 14, 15, 16])
def test_accesses_stay_inside_the_workspace(reclib, n, is_dd):
    A = _sym(2 * n, n)
    g = np.random.default_rng(n)
    for loop in (False, True):
        for clog in sorted({0, 1, 4, 5, 6, 7, 8, n}):
            if clog > n or (clog == n and n > 12):
                continue
            full = (1 << n) - (1 << clog)
            for lo in {0, full, int(g.integers(0, 1 << n)) & full, int(g.integers(0, 1 << n)) & full}:
                _sum(reclib, A, loop, is_dd, lo, clog)
