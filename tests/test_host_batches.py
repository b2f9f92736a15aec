"""How the Python layer takes a batch (no GPU): a list is stacked by one conversion, whatever
its numbers, and gives the stack's numbers; refused batches stay refused."""

from __future__ import annotations

import numpy as np
import pytest


class Counted:
    """A matrix that counts how often it is converted."""

    calls = 0

    def __init__(self, a):
        self.a = a

    def __array__(self, dtype=None, copy=None):
        Counted.calls += 1
        return np.array(self.a, dtype=dtype)


def _conversions(f, mats):
    Counted.calls = 0
    f(mats)
    return Counted.calls


@pytest.mark.parametrize("dtype", [np.complex128, np.complex64, np.float64, np.float32, np.int64, np.longdouble])
def test_a_list_is_converted_once(G, dtype):
    mats = [Counted(np.arange(16).reshape(4, 4).astype(dtype)) for _ in range(5)]
    once = _conversions(lambda m: np.asarray(m, dtype=np.complex128), mats)
    assert once > 0
    assert _conversions(G._as_stack, mats) == once


@pytest.mark.parametrize("wrap", [list, tuple, lambda s: s.tolist(), lambda s: [list(m) for m in s]])
def test_a_complex_list_is_read_once_as_complex(G, monkeypatch, wrap):
    # the type of nested lists costs numpy as much to find as the numbers to read
    batch, seen, asarray = wrap(np.arange(18.0).reshape(2, 3, 3) + 1j), [], np.asarray
    monkeypatch.setattr(G.np, "asarray", lambda a, dtype=None: (seen.append(dtype), asarray(a, dtype=dtype))[1])
    G._as_stack(batch)
    assert seen == [np.complex128]


@pytest.mark.parametrize("dtype", [np.complex128, np.complex64, np.clongdouble, np.longdouble, np.float64, np.float32,
                                   np.float16, np.int64, np.uint8, bool, object, "U32"])
def test_a_list_gives_the_numbers_of_its_stack(G, dtype):
    g = np.random.default_rng(3)
    base = g.integers(0, 2, (3, 4, 4)) if dtype is bool else g.integers(0, 100, (3, 4, 4)) / 4
    if np.dtype(dtype).kind == "c" or dtype is object:
        base = base + 1j * g.integers(0, 100, (3, 4, 4))
    stack = base.astype(dtype)
    want = np.asarray(stack, dtype=np.complex128)
    for batch in (stack, list(stack), stack.tolist(), np.asfortranarray(stack), stack[:, ::-1][:, ::-1]):
        got = G._as_stack(batch)
        assert got.flags.c_contiguous and got.dtype in (np.complex128, np.float64)
        assert np.array_equal(got.astype(np.complex128), want)


def test_a_mixed_list_is_complex(G):
    a, b = np.arange(4.0).reshape(2, 2), 1j * np.eye(2)
    assert np.array_equal(G._as_stack([a, b]), np.array([a, b], dtype=np.complex128))


@pytest.mark.parametrize("batch", [[np.eye(2), np.eye(3)], [np.ones((2, 3))] * 2, np.eye(4), [], [["a"]], [[None]]])
def test_refused_batches(G, batch):
    with pytest.raises((ValueError, TypeError)):
        G._as_stack(batch)


class _Recorder:
    """A library whose queue call notes the function and tier codes it gets."""

    def gbs_queue_evaluate_ptrs(self, session, B, fns, tiers, dims, *rest):
        self.codes = [fns[i] for i in range(B)], [tiers[i] for i in range(B)], [dims[i] for i in range(B)]
        return 0


@pytest.mark.parametrize("wrap", [list, tuple, iter, lambda x: (y for y in x), lambda x: map(str, x),
                                  lambda x: np.array(x), lambda x: dict(enumerate(x)).values()])
def test_names_of_a_mixed_batch_may_be_any_iterable(G, monkeypatch, wrap):
    rec = _Recorder()
    monkeypatch.setattr(G._lib, "load", lambda: rec)
    ws = G.Workspace()
    ws._session = object()
    mats = [np.eye(n, dtype=complex) for n in (2, 4, 6)]
    for call in (ws.evaluate, ws.evaluate_full):
        call(wrap(["haf", "lhaf", "tor"]), mats, wrap(["fp64", "dd", "fp64"]))
        assert rec.codes == ([1, 2, 3], [0, 1, 0], [2, 4, 6])
    ws._session = None
