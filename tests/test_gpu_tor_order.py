"""Which entries of a torontonian's O are read when it is not symmetric: the lower triangle in
the order (mode, x before p), as the reference does, but the upper one in the block of the
last 5 (double-double 4) modes against those before them.  So a call gives bit for bit what
the symmetric matrix of those entries gives, and up to 5 (4) modes the oracle's value."""

from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_err


def asymmetric_O(k, seed):
    g = np.random.default_rng(seed)
    X = g.standard_normal((2 * k, 2 * k))
    O = np.eye(2 * k) - np.linalg.inv(X @ X.T / (2 * k) + np.eye(2 * k))
    return (O + O.T) / 2 + 0.01 * g.uniform(-1, 1, (2 * k, 2 * k)) / k


def entries_read(O, tail):
    """The symmetric matrix of the entries that count."""
    k = O.shape[0] // 2
    S = O.copy()
    for a in range(2 * k):
        for b in range(2 * k):
            late, early = (a % k, a // k), (b % k, b // k)
            if late > early:
                r, c = (b, a) if early[0] < k - tail <= late[0] else (a, b)
                S[a, b] = S[b, a] = O[r, c]
    return S


@pytest.mark.gpu
@pytest.mark.parametrize("k", [1, 2, 4, 5, 6, 7, 9, 10, 13, 16])
def test_an_asymmetric_O_reads_the_entries_it_always_read(gpu, orc, k):
    O = np.stack([asymmetric_O(k, 10 * k + i) for i in range(3)])
    for precision, tail in (("fp64", 5), ("certified", 5), ("dd", 4)):
        S = np.stack([entries_read(o, tail) for o in O])
        assert k == 1 or not np.array_equal(O, S)
        got, want = (gpu.tor_batched(x, precision=precision, return_diagnostics=precision == "certified") for x in (O, S))
        if precision == "certified":
            got, want = got[0], want[0]
        assert np.array_equal(got, want), precision
        if k <= tail:
            for o, v in zip(O, got):
                assert rel_err(v, orc.tor(o.astype(complex), "quad")) < 1e-10, precision
    # a NaN in an entry that is not read changes nothing, in one that is it refuses
    if k > 1:
        P, Q = O.copy(), O.copy()
        r, c = (k - 1, 0) if k <= 5 else (0, k - 1)  # x of the last and the first mode
        P[:, c, r], Q[:, r, c] = np.nan, np.nan
        assert np.array_equal(gpu.tor_batched(P), gpu.tor_batched(O))
        assert np.isnan(gpu.tor_batched(Q).real).all()
