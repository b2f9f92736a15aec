"""The walk of the torontonian recursion (gbskernels_b200/csrc/tor_rec.cuh) on the CPU: the
kernel's own layout and node functions drive a sequential walk (tests/tor_host.cu) whose
every access must lie inside the workspace the planner asks for and read a written word,
for every split into items, and whose sums must equal the oracle's torontonian."""

from __future__ import annotations

import ctypes
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

HERE = Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def torlib():
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if Path("/usr/local/cuda/bin/nvcc").exists() else None)
    if nvcc is None:
        pytest.skip("nvcc not available")
    out = HERE / "_build" / "libtorhost.so"
    out.parent.mkdir(exist_ok=True)
    src = HERE / "tor_host.cu"
    csrc = HERE.parent / "gbskernels_b200" / "csrc"
    deps = [src, *csrc.glob("*.cuh")]
    if not out.exists() or out.stat().st_mtime < max(p.stat().st_mtime for p in deps):
        cmd = [nvcc, "-x", "cu", "-O2", "-std=c++17", "--expt-relaxed-constexpr", "-shared", "-Xcompiler", "-fPIC",
               "-gencode", "arch=compute_100a,code=sm_100a", "-I", str(csrc), str(src), "-o", str(out)]
        subprocess.run(cmd, check=True, capture_output=True)
    lib = ctypes.CDLL(str(out))
    lib.t_tor_rec_item.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_uint, ctypes.c_int,
                                   ctypes.c_int, ctypes.c_void_p]
    return lib


def _item(lib, O, g, lo, is_dd, cert):
    O = np.ascontiguousarray(O, dtype=np.float64)
    out = np.zeros(1)
    bad = lib.t_tor_rec_item(O.ctypes.data, O.shape[0] // 2, g, lo, is_dd, cert, out.ctypes.data)
    assert bad == 0, (O.shape, g, lo, is_dd, cert, bad)
    return float(out[0])


def _phys_O(n, seed):
    X = np.random.default_rng(seed).standard_normal((2 * n, 2 * n))
    O = np.eye(2 * n) - np.linalg.inv(X @ X.T / (2 * n) + np.eye(2 * n))
    return (O + O.T) / 2


@pytest.mark.parametrize("k", range(1, 12))
def test_sums_equal_the_oracle_for_every_split(torlib, orc, k):
    O = _phys_O(k, k)
    t, absn = orc.tor(O.astype(complex), "quad", with_absnorm=True)
    for g in range(k):
        for is_dd in (0, 1):
            v = sum(_item(torlib, O, g, lo, is_dd, 1) for lo in range(1 << g))
            # m roundings per factor entry, m^2 entries: a few k^2 u of the sum of the moduli
            assert abs(v - t.real) <= 64 * k * k * 2.0 ** -53 * absn, (g, is_dd)


@pytest.mark.parametrize("k", [13, 15, 17, 24, 32])
def test_accesses_stay_inside_the_workspace(torlib, k):
    O = _phys_O(k, k)
    for is_dd in (0, 1):
        for cert in (0, 1):
            for f in (1, 5, 10, 12, 14) if k > 14 else (k, 9):
                g = k - f
                for lo in (0, (1 << g) - 1, (0x55555555 & ((1 << g) - 1))):
                    _item(torlib, O, g, lo, is_dd, cert)


@pytest.mark.parametrize("k,g", [(15, 0), (16, 1), (16, 0)])
def test_more_free_modes_than_are_walked_at_a_time(torlib, orc, k, g):
    O = _phys_O(k, k)
    t, absn = orc.tor(O.astype(complex), "quad", with_absnorm=True)
    for is_dd in (0, 1):
        v = sum(_item(torlib, O, g, lo, is_dd, 1) for lo in range(1 << g))
        assert abs(v - t.real) <= 64 * k * k * 2.0 ** -53 * absn, is_dd


@pytest.mark.parametrize("k", [2, 5, 6, 9])
def test_an_asymmetric_O_reads_one_entry_of_each_pair(torlib, orc, k):
    from test_gpu_tor_order import asymmetric_O, entries_read
    O = asymmetric_O(k, k)
    for is_dd, tail in ((0, 5), (1, 4)):
        v = _item(torlib, O, 0, 0, is_dd, 0)
        assert v == _item(torlib, entries_read(O, tail), 0, 0, is_dd, 0)
        if k <= tail:
            assert v == pytest.approx(orc.tor(O.astype(complex)).real, rel=1e-10)
