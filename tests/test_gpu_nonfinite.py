"""The hafnian and torontonian recursions at the limits of the number range: an infinity or a
NaN that counts gives NaN (the certified tiers refuse) in every tier, real or complex, and
leaves the rest of the batch alone; a matrix times a power of two gives the same digits as
long as nothing over- or underflows, NaN or a refusal beyond."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mat(func, n, real, seed=5):
    g = np.random.default_rng([seed, n, real])
    if func == "tor":
        X = g.standard_normal((n, n))
        O = np.eye(n) - np.linalg.inv(X @ X.T / n + np.eye(n))
        return (O + O.T) / 2
    A = g.standard_normal((n, n)) + (0 if real else 1j * g.standard_normal((n, n)))
    return (A + A.T) / 4


CASES = [(f, n, r) for f in ("haf", "lhaf") for n in (2, 4, 10, 12, 14, 18) for r in (True, False)]
CASES += [("lhaf", n, r) for n in (1, 3, 9) for r in (True, False)] + [("tor", n, True) for n in (2, 8, 12, 22, 32)]


@pytest.mark.parametrize("func,n,real", CASES)
def test_an_entry_that_is_not_finite(gpu, func, n, real):
    f = getattr(gpu, f"{func}_batched")
    A = _mat(func, n, real)
    bad = [A]
    for v in (np.nan, np.inf, -np.inf):
        B = A.copy()
        B[n - 1, 0] = B[0, n - 1] = v
        bad.append(B)
        if func == "lhaf":
            B = A.copy()
            B[n // 2, n // 2] = v
            bad.append(B)
    bad.append(A)
    bad = np.stack(bad)
    with np.errstate(invalid="ignore"):
        for precision in ("fp64", "dd", "auto"):
            if func == "tor" and precision == "auto":
                continue
            v = f(bad, precision=precision)
            alone = f(A[None], precision=precision)[0]
            assert v[0] == v[-1] == alone and np.isfinite(alone), precision
            assert np.isnan(v[1:-1].real).all(), (precision, v)
            if func != "tor" or precision == "fp64":
                assert np.isnan(v[1:-1].imag).all(), (precision, v)
        with pytest.raises((RuntimeError, ValueError), match="finite input"):
            f(bad, precision="certified", return_diagnostics=True)


@pytest.mark.parametrize("func,n,real", [c for c in CASES if c[0] != "tor" and c[1] % 2 == 0])
def test_powers_of_two(gpu, func, n, real):
    f = getattr(gpu, f"{func}_batched")
    A = _mat(func, n, real)
    one = {p: f(A[None], precision=p)[0] for p in ("fp64", "dd")}
    # every edge times 2^e, every loop times 2^(e / 2): the value times 2^(e n / 2).  Double
    # words need their low parts above 2^-1022, entries their products below 2^1024.
    for e in {2 * (400 // n), -2 * (400 // n), 2 * (900 // n), 2 * (9000 // n)}:
        S = A * 2.0 ** min(e, 1000)
        if func == "lhaf":
            S[np.arange(n), np.arange(n)] = np.diag(A) * 2.0 ** (min(e, 1000) // 2)
        for p in ("fp64", "dd"):
            v = f(S[None], precision=p)[0]
            if e * n // 2 < 1000:
                assert v == one[p] * 2.0 ** (e * n // 2), (p, e)
            elif n > 2:
                assert np.isnan(v.real) and np.isnan(v.imag), (p, e, v)
    if n > 2:
        with pytest.raises(FloatingPointError):
            f(A[None] * 2.0 ** 1000, precision="certified", return_diagnostics=True)
