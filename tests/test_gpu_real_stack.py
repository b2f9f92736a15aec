"""Real stacks go to the library as float64 (gbs_uniform_real_host, gbs_auto_real_host,
gbs_certified_ladder_real_host): every result must be the complex path's for the same
numbers bit for bit -- small batches (one upload, widened on the host), large ones (widened
on the device), odd loop hafnians (augmented), every function and tier, and inputs that need
converting (float32, integers, booleans, strides, a list)."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _stack(func, n, B, seed=5):
    g = np.random.default_rng(seed)
    X = g.standard_normal((B, n, n))
    S = (X + np.transpose(X, (0, 2, 1))) / 2
    if func == "tor":
        return 0.2 * S / np.sqrt(n)
    return X if func == "perm" else S


def _all(G, func, A):
    f = getattr(G, f"{func}_batched")
    vc, dc = f(A, precision="certified", return_diagnostics=True)
    vr, dr = f(A, precision="certified", return_diagnostics=True, rtol=1e-13)
    va, da = f(A, precision="auto", return_diagnostics=True)
    return [f(A), f(A, precision="dd"), vc, [d["abs_error_bound"] for d in dc], vr,
            [d["abs_error_bound"] for d in dr], va, [d["cancellation"] for d in da]]


@pytest.mark.parametrize("func,n", [("perm", 1), ("perm", 7), ("haf", 2), ("haf", 7), ("haf", 8), ("lhaf", 1), ("lhaf", 7),
                                    ("lhaf", 8), ("tor", 2), ("tor", 8)])
@pytest.mark.parametrize("B", [1, 3, 1500])
def test_real_equals_complex_bitwise(gpu, func, n, B):
    A = _stack(func, n, B)
    for a, b in zip(_all(gpu, func, A), _all(gpu, func, A.astype(np.complex128))):
        assert np.array_equal(np.asarray(a), np.asarray(b)), func


def test_inputs_that_need_converting(gpu):
    A = _stack("haf", 8, 4)
    wide = np.zeros((4, 16, 8))
    wide[:, ::2] = A
    forms = [A.astype(np.float32), np.rint(3 * A).astype(np.int32), A > 0, wide[:, ::2], list(A), np.asfortranarray(A)]
    for x in forms:
        want = gpu.haf_batched(np.ascontiguousarray(np.asarray(x, dtype=np.complex128)))
        assert np.array_equal(gpu.haf_batched(x), want)
    assert gpu.haf(np.ones((4, 4), dtype=np.int64)) == 3.0
    with pytest.raises(ValueError, match="finite"):
        B = A.copy()
        B[1, 2, 3] = np.nan
        gpu.haf_batched(B, precision="certified", return_diagnostics=True)
    with pytest.raises(ValueError):
        gpu.haf_batched([np.eye(2), np.eye(4)])
