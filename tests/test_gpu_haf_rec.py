"""The hafnian recursion (csrc/haf_rec.cuh) at the sizes and splits where its walk changes:
no prefix, a prefix, the depth-first part (blocks of 6 and 7 pairs), several blocks per
item, single-subset items; real and complex, hafnian and loop hafnian, against the
binary128 oracle; the indicator and certified tiers give the same value; the
double-double tier to its last bit."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def _mat(N, real, seed):
    g = np.random.default_rng(seed)
    X = g.standard_normal((N, N)) + (0 if real else 1j * g.standard_normal((N, N)))
    return ((X + X.T) / 4).astype(np.complex128)


@pytest.mark.parametrize("N", [1, 2, 4, 9, 10, 12, 14, 15, 16, 18])
def test_every_split_vs_oracle(gpu, lib, orc, N):
    n = (N + 1) // 2
    for func, code in (("haf", 1), ("lhaf", 2)):
        if func == "haf" and N % 2:
            continue
        for real in (False, True):
            A = _mat(N, real, 100 + N)
            t, absn = getattr(orc, func)(A, "quad", with_absnorm=True)
            # the recursion's terms are smaller than the power trace's (absn): a few n u of it
            tol = 32 * n * U * absn
            f = getattr(gpu, f"{func}_batched")
            for split in sorted({0, 1, 4, 5, 6, 7, 8, n} | {-1}):
                if split > n:
                    continue
                assert lib.gbs_set_split(code, 0, 2 * n, split, 0) == 0
                assert lib.gbs_set_split(code, 1, 2 * n, split, 0) == 0
                try:
                    v = f(A[None])[0]
                    vc, dc = f(A[None], precision="certified", return_diagnostics=True)
                    _, dk = f(A[None], precision="auto", return_diagnostics=True)
                    vd = f(A[None], precision="dd")[0]
                finally:
                    lib.gbs_set_split(code, 1, 2 * n, -1, 0)
                    lib.gbs_set_split(code, 0, 2 * n, -1, 0)
                assert abs(v - t) <= tol, (func, real, split, v, t)
                assert vc[0] == v and abs(v - t) <= dc[0]["abs_error_bound"] + U * abs(t), (func, real, split)
                assert abs(vd - t) <= 2 * U * abs(t) + 1e-20 * absn, (func, real, split, vd, t)
                assert dk[0]["cancellation"] == pytest.approx(absn / abs(t), rel=1e-6), (func, real, split)


@pytest.mark.parametrize("N", [30, 32])
def test_largest_sizes_factorise(gpu, N):
    """A direct sum: the hafnians of the blocks multiply (complex and real).  Proven bounds of
    the factors and of the product have to meet; the binary64 value of these matrices errs by
    4.5e-11 at most (measured; u times the sum of moduli of the power-trace terms is 8e-10 ..
    3e-6), allowed four times that; the double-double one is good to its rounding."""
    for real in (True, False):
        A, B = _mat(14, real, 1), _mat(N - 14, real, 2)
        blk = np.zeros((N, N), complex)
        blk[:14, :14], blk[14:, 14:] = A, B
        p = np.random.default_rng(3).permutation(N)
        blk = blk[np.ix_(p, p)]
        for name in ("haf", "lhaf"):
            f = getattr(gpu, name)
            (v, d), (a, da), (b, db) = (f(X, precision="certified", return_diagnostics=True) for X in (blk, A, B))
            ea, eb = da["abs_error_bound"], db["abs_error_bound"]
            slack = abs(a) * eb + abs(b) * ea + ea * eb + 4 * U * abs(a * b)  # + the rounding of a * b
            assert abs(v - a * b) <= d["abs_error_bound"] + slack, (name, real, v, a * b)
            want = f(A, precision="dd") * f(B, precision="dd")  # good to a few u
            kappa = f(blk, precision="auto", return_diagnostics=True)[1]["cancellation"]
            assert abs(v - want) <= min(2e-10, U * kappa) * abs(want), (name, real, v, want, kappa)
            vd = f(blk, precision="dd")
            assert abs(vd - want) <= (8 * U + 1e-20 * kappa) * abs(want), (name, real, vd, want, kappa)
