"""The indicator tier of hafnians and loop hafnians: the value is the fp64 one bit for bit and
the sum of the moduli of the power-trace terms the oracle's, whatever the entry point, the
launch mode and the company: sides around the split of the terms into items, real and
complex, odd, trivial, several tiers in one batch."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mat(N, real, seed):
    g = np.random.default_rng([seed, N, real])
    X = g.standard_normal((N, N)) + (0 if real else 1j * g.standard_normal((N, N)))
    return ((X + X.T) / 4).astype(np.complex128)


def _one_shot(gpu, func, A):
    lib = gpu._lib.load()
    out, aux = np.empty(1, np.complex128), np.empty(1)
    name = f"gbs_{func}_kappa_host"
    gpu._lib.check(getattr(lib, name)(gpu._lib.dptr(A.view(np.float64)), A.shape[0], 1,
                                      gpu._lib.dptr(out.view(np.float64)), gpu._lib.dptr(aux)), name)
    return out[0], aux[0]


@pytest.mark.parametrize("N", [1, 2, 7, 8, 10, 11, 12, 14, 18])
@pytest.mark.parametrize("real", [True, False])
def test_against_the_oracle(gpu, orc, N, real):
    for func in ("haf", "lhaf"):
        if func == "haf" and N % 2:
            continue
        A = _mat(N, real, 1)
        _, absn = getattr(orc, func)(A, "quad", with_absnorm=True)
        v, a = _one_shot(gpu, func, A)
        assert v == getattr(gpu, f"{func}_batched")(A[None])[0]
        assert a == pytest.approx(absn, rel=1e-9), func


def test_every_way_in_gives_the_same(gpu):
    sizes = [0, 1, 2, 5, 6, 8, 9, 10, 11, 12, 13, 14, 16, 20, 20]
    mats, funcs, tiers = [], [], []
    for i, N in enumerate(sizes):
        for func in ("haf", "lhaf"):
            for tier in ("kappa", "fp64", "kappa", "certified", "dd"):
                mats.append(_mat(N, bool(len(mats) % 2), 2))
                funcs.append(func)
                tiers.append(tier)
    g = np.random.default_rng(3)
    for k in (2, 6, 11):
        X = g.standard_normal((2 * k, 2 * k))
        O = np.eye(2 * k) - np.linalg.inv(X @ X.T / (2 * k) + np.eye(2 * k))
        mats += [((O + O.T) / 2).astype(complex)] * 2 + [_mat(2 * k, False, 4)] * 2
        funcs += ["tor", "tor", "perm", "perm"]
        tiers += ["kappa", "fp64"] * 2
    order = g.permutation(len(mats))
    mats, funcs, tiers = [mats[i] for i in order], [funcs[i] for i in order], [tiers[i] for i in order]
    with gpu.Workspace() as ws, gpu.Workspace(persistent=False) as per_size:
        out, aux, st = ws.evaluate_full(funcs, mats, tiers)
        for other in (ws, per_size):
            o, a, s = other.evaluate_full(funcs, mats, tiers)
            assert np.array_equal(o, out, equal_nan=True) and np.array_equal(a, aux) and np.array_equal(s, st)
        r = ws.evaluate_resident(funcs, mats, tiers)
        assert np.array_equal(r.numpy(), out, equal_nan=True) and np.array_equal(r.aux.numpy(), aux)
        r.close()
        plain = ws.evaluate(funcs, mats, ["fp64" if t == "kappa" else t for t in tiers])
        assert np.array_equal(plain, out, equal_nan=True)
    assert (st == 0).all()
    for i, (f, m, t) in enumerate(zip(funcs, mats, tiers)):
        if t == "kappa" and f in ("haf", "lhaf"):
            assert (out[i], aux[i]) == _one_shot(gpu, f, m), (f, m.shape)
