"""Certified hafnians of matrices whose symmetric part cannot be formed: (A + A^T) / 2 of two
entries near the bottom of the number range can round by half a unit of 2^-1074, which no
radius relative to the entries covers, so both certified tiers refuse (NaN, infinite bound)
and the ladder ends in its refusal.  A halving that is exact is no reason to refuse."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SUB = 2.0 ** -1074


def _cert(gpu, func, A, tier):
    lib = gpu._lib.load()
    cm = np.ascontiguousarray(A[None], dtype=np.complex128)
    out, bnd = np.empty(1, np.complex128), np.empty(1)
    name = f"gbs_{func}_{tier}_host"
    gpu._lib.check(getattr(lib, name)(gpu._lib.dptr(cm.view(np.float64)), cm.shape[1], 1,
                                      gpu._lib.dptr(out.view(np.float64)), gpu._lib.dptr(bnd)), name)
    return out[0], bnd[0]


def _mat(upper, lower, func, n, unit):
    """A_01 = upper, A_10 = lower, the other pairs 2^(500 / (n / 2 - 1)), times `unit`."""
    A = np.zeros((n, n), complex)
    A[0, 1], A[1, 0] = upper * unit, lower * unit
    for i in range(2, n, 2):
        A[i, i + 1] = A[i + 1, i] = 2.0 ** (500 // (n // 2 - 1))
    if func == "lhaf":
        A[np.arange(n), np.arange(n)] = 0.25
    return A


def _lost_by_halving(x, y):
    s = np.longdouble(x) + np.longdouble(y)  # exact: 64 bits hold both words of these sums
    return np.longdouble(0.5 * float(s)) * 2 + np.longdouble(0.5 * float(s - np.longdouble(float(s)))) * 2 != s


@pytest.mark.parametrize("func", ["haf", "lhaf"])
@pytest.mark.parametrize("n", [4, 6, 18])
@pytest.mark.parametrize("unit", [1.0, 1j, 1.0 + 1.0j])
@pytest.mark.parametrize("upper,lower", [(3 * SUB, 0.0), (0.0, SUB), (2.0 ** -1030, 3 * SUB), (-5 * SUB, 2 * SUB)])
def test_a_halving_that_rounds_is_refused_by_both_tiers(gpu, func, n, unit, upper, lower):
    assert _lost_by_halving(upper, lower)
    A = _mat(upper, lower, func, n, unit)
    for tier in ("certified", "dd_certified"):
        v, b = _cert(gpu, func, A, tier)
        assert np.isnan(v.real) and np.isposinf(b), (tier, v, b)
    with pytest.raises(Exception):
        getattr(gpu, f"{func}_batched")(A[None], precision="certified", return_diagnostics=True, rtol=1e-12)


@pytest.mark.parametrize("func", ["haf", "lhaf"])
def test_a_low_word_that_rounds_is_refused_in_double_double(gpu, func):
    # the high word 2^-1021 halves exactly, the low word 2^-1074 does not; in binary64 the
    # sum rounds to 2^-1021, a relative error that its radius holds
    assert _lost_by_halving(2.0 ** -1021, SUB)
    A = _mat(2.0 ** -1021, SUB, func, 4, 1.0)
    v, b = _cert(gpu, func, A, "dd_certified")
    assert np.isnan(v.real) and np.isposinf(b)
    v, b = _cert(gpu, func, A, "certified")
    assert np.isfinite(v.real) and np.isfinite(b)


@pytest.mark.parametrize("func", ["haf", "lhaf"])
@pytest.mark.parametrize("n", [4, 18])
def test_an_exact_halving_is_certified_in_double_double(gpu, orc, func, n):
    for upper, lower in ((4 * SUB, 0.0), (3 * SUB, 3 * SUB), (2.0 ** -1020, 2.0 ** -1072), (SUB, SUB)):
        assert not _lost_by_halving(upper, lower)
        A = _mat(upper, lower, func, n, 1.0)
        v, b = _cert(gpu, func, A, "dd_certified")
        S = A.copy()
        S[0, 1] = S[1, 0] = (upper + lower) / 2
        if func == "haf":  # one perfect matching
            want = np.prod(np.longdouble(1) * np.real(S[np.arange(0, n, 2), np.arange(1, n, 2)]).astype(np.longdouble))
            assert np.isfinite(b) and abs(np.longdouble(v.real) - want) <= b, (upper, lower, v, b)
        else:
            assert np.isfinite(b) and v == gpu.lhaf_batched(S[None], precision="dd")[0]
