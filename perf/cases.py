"""Workloads whose speed this repository tracks: the calls its users make, through
the public entry points, from one small matrix to a ragged batch of thousands.

A case is a dict of plain values.  `prepare` makes the host inputs a program has in
hand (and the Workspace it keeps open), `run` is one call, `exact` the same numbers
by an independent formula in plain 64-bit torch.  The sizes of a ragged batch are a
function of the case alone; only the values depend on the seed.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import gbskernels_b200 as G
from gbskernels_b200 import workloads as W
from gbskernels_b200.sampler import sample_resident


def listed():
    return [
        # one matrix, one answer: an interactive call or a step of a host-side sampler
        {"name": "one haf 8", "kind": "one", "func": "haf", "n": 8, "real": False},
        # a uniform batch of real matrices (graph problems: perfect matchings, dense subgraphs)
        {"name": "haf real 16", "kind": "stack", "func": "haf", "n": 16, "batch": 4096, "real": True,
         "precision": "fp64"},
        # the ragged haf / lhaf queue a sampler fills per step: a small and a large fill
        {"name": "queue 256", "kind": "queue", "lo": 8, "hi": 28, "batch": 256},
        {"name": "queue 4096", "kind": "queue", "lo": 8, "hi": 28, "batch": 4096},
        # the tier a careful user picks by default: binary64 with the cancellation check,
        # even and odd sizes
        {"name": "lhaf auto", "kind": "auto", "lo": 6, "hi": 21, "batch": 512},
        # proven values: every bound within 1e-6 of its value
        {"name": "haf certified 16", "kind": "stack", "func": "haf", "n": 16, "batch": 512, "real": False,
         "precision": "certified"},
        # the high-precision tier
        {"name": "lhaf dd 14", "kind": "stack", "func": "lhaf", "n": 14, "batch": 128, "real": False,
         "precision": "dd"},
        # boson sampling: output probabilities of 20 photons in a 400-mode interferometer
        {"name": "perm 20", "kind": "stack", "func": "perm", "n": 20, "batch": 512, "real": False,
         "precision": "fp64"},
        # threshold detectors: click patterns of 10..22 modes, and a proven batch of 12
        {"name": "tor clicks", "kind": "clicks", "lo": 10, "hi": 22, "batch": 256},
        {"name": "tor certified 12", "kind": "stack", "func": "tor", "n": 12, "batch": 512, "real": True,
         "precision": "certified"},
        # photon patterns with repeats over one kernel matrix
        {"name": "sieve 2048", "kind": "sieve", "modes": 12, "most": 3, "batch": 2048},
        # samples of an 8-mode lossy squeezed state, drawn on the device
        {"name": "sampler", "kind": "sampler", "modes": 8, "cutoff": 2, "samples": 50000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["one", "stack", "stack", "stack", "queue", "queue", "auto", "clicks", "sieve", "sampler"])
    if kind == "one":
        func = rng.choice(["haf", "lhaf", "perm", "tor"])
        n = {"haf": 2 * rng.randint(1, 10), "lhaf": rng.randint(1, 20), "perm": rng.randint(1, 18),
             "tor": rng.randint(1, 14)}[func]
        return {"kind": kind, "func": func, "n": n, "real": func == "tor" or rng.random() < 0.3}
    if kind == "stack":
        func = rng.choice(["haf", "lhaf", "perm", "tor"])
        precision = rng.choice(["fp64", "fp64", "dd", "certified"])
        top = {"fp64": 0, "certified": 2, "dd": 4}[precision]
        n = {"haf": 2 * rng.randint(2, 10 - top // 2), "lhaf": rng.randint(4, 20 - top),
             "perm": rng.randint(5, 18 - top), "tor": rng.randint(4, 14 - top // 2)}[func]
        return {"kind": kind, "func": func, "n": n, "batch": _log(rng, 2, 1024),
                "real": func == "tor" or rng.random() < 0.4, "precision": precision}
    if kind in ("queue", "auto", "clicks"):
        lo, hi, most = {"queue": (4, 28, 800), "auto": (3, 20, 512), "clicks": (6, 22, 200)}[kind]
        a, b = sorted((rng.randint(lo, hi), rng.randint(lo, hi)))
        if kind == "queue":
            a, b = a - a % 2, b - b % 2
        return {"kind": kind, "lo": a, "hi": b, "batch": _log(rng, 3, most)}
    if kind == "sieve":
        return {"kind": kind, "modes": rng.randint(4, 12), "most": rng.randint(1, 3), "batch": _log(rng, 8, 3000)}
    modes = rng.randint(2, 8)
    return {"kind": kind, "modes": modes, "cutoff": rng.randint(1, min(4, 16 // modes)),
            "samples": _log(rng, 500, 50000)}


# ------------------------------------------------------------------ inputs
def _sizes(case):
    """Sizes of a ragged batch: every size of the range equally often, in a fixed order."""
    step = 2 if case["kind"] == "queue" else 1
    span = np.arange(case["lo"], case["hi"] + 1, step)
    out = np.resize(span, case["batch"])
    return [int(x) for x in np.random.default_rng(11).permutation(out)]


def _photons(A, gamma, n, loop, rng):
    """The submatrix of a random n-photon pattern (repeated modes), loop weights on its diagonal."""
    idx = np.sort(rng.integers(0, A.shape[0], size=n))
    S = np.ascontiguousarray(A[np.ix_(idx, idx)])
    if loop:
        np.fill_diagonal(S, gamma[idx])
    return S


def _kernel(seed, modes=100):
    rng = np.random.default_rng([seed, 1])
    return W.gbs_kernel(modes, 1.0, seed), np.sqrt(0.05) * (rng.standard_normal(modes) + 1j * rng.standard_normal(modes)), rng


def _clicks(Ox, k, rng):
    S = np.sort(rng.choice(Ox.shape[0] // 2, size=k, replace=False))
    idx = np.concatenate([S, S + Ox.shape[0] // 2])
    return np.ascontiguousarray(Ox[np.ix_(idx, idx)])


def _uniform(func, n, batch, real, seed):
    if func == "haf" and real:
        return W.haf_real_batch(batch, n, seed)
    if func == "perm":
        A = W.perm_haar_batch(batch, n, max(60, n * n), seed) if n * n <= 400 else W.perm_haar_batch(batch, n, 400, seed)
        return np.ascontiguousarray(A.real) if real else A
    if func == "tor":
        rng = np.random.default_rng([seed, 2])
        Ox = W.threshold_O(W.lossy_squeezed_cov(50, seed=seed))
        return np.stack([_clicks(Ox, n, rng) for _ in range(batch)])
    A, gamma, rng = _kernel(seed)
    S = np.stack([_photons(A, gamma, n, func == "lhaf", rng) for _ in range(batch)])
    return np.ascontiguousarray(S.real) if real else S


def _inputs(case, seed):
    kind = case["kind"]
    if kind == "one":
        return {"mat": _uniform(case["func"], case["n"], 1, case["real"], seed)[0]}
    if kind == "stack":
        return {"stack": _uniform(case["func"], case["n"], case["batch"], case["real"], seed)}
    if kind == "clicks":
        rng = np.random.default_rng([seed, 3])
        Ox = W.threshold_O(W.lossy_squeezed_cov(50, seed=seed))
        return {"mats": [_clicks(Ox, k, rng).astype(np.complex128) for k in _sizes(case)]}
    if kind in ("queue", "auto"):
        A, gamma, rng = _kernel(seed)
        loops = [kind == "auto" or i % 2 == 1 for i in range(case["batch"])]
        return {"mats": [_photons(A, gamma, n, loop, rng) for n, loop in zip(_sizes(case), loops)],
                "funcs": ["lhaf" if loop else "haf" for loop in loops]}
    if kind == "sieve":
        A, gamma, _ = _kernel(seed, case["modes"])
        reps = np.random.default_rng([seed, 4]).integers(0, case["most"] + 1, size=(case["batch"], case["modes"]))
        return {"A": A, "gamma": gamma, "reps": reps.astype(np.int32)}
    return {"cov": W.lossy_squeezed_cov(case["modes"], seed=seed), "seed": seed}


class _State(dict):
    """The inputs of one pass and the Workspace the program keeps open."""

    def __del__(self):
        ws = self.get("ws")
        if ws is not None:
            ws.close()


def prepare(case, seed):
    state = _State(_inputs(case, seed), case=case)
    if case["kind"] in ("queue", "auto", "clicks"):
        state["ws"] = G.Workspace().__enter__()
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "one":
        return getattr(G, case["func"])(state["mat"]).real if case["real"] else _parts(getattr(G, case["func"])(state["mat"]))
    if kind == "stack":
        f = getattr(G, case["func"] + "_batched")
        if case["precision"] == "certified":
            values, diags = f(state["stack"], precision="certified", return_diagnostics=True)
            # the radius is any proven one, so what a program asks of it is whether it is small enough
            return values, np.array([d["abs_error_bound"] <= max(1e-6 * abs(v), 1e-6) for v, d in zip(values, diags)])
        return f(state["stack"], precision=case["precision"])
    if kind == "queue":
        return state["ws"].evaluate(state["funcs"], state["mats"], ["fp64"] * len(state["mats"]))
    if kind == "auto":
        return state["ws"].lhaf_batched(state["mats"], precision="auto")
    if kind == "clicks":
        return state["ws"].tor_batched(state["mats"])
    if kind == "sieve":
        return G.lhaf_repeated(state["A"], state["gamma"], state["reps"])
    return sample_resident(state["cov"], case["samples"], cutoff=case["cutoff"], seed=state["seed"])


def _parts(v):
    return [v.real, v.imag]


# ------------------------------------------------------------------ work and tolerance
def _haf_flops(n2, loop, real):
    """Sums over the pairs of a matrix of side n2 (odd: one row more) by the recursion over
    pairs with polynomials in the number of pairs used (Bjorklund 2012): with m pairs left,
    2^(n-m) states each join 2 (m-1) (2m-3) (loop: (2m-1)) products of n-m+1 coefficients."""
    n = (n2 + 1) // 2
    macs = 0.0
    for m in range(1, n + 1):
        t = n - m
        polys = (m - 1) * (2 * m - 3 + (2 if loop else 0))
        macs += 2.0 ** t * (polys * (t + 1) * (t + 2) + (t + 1) * (t + 2) / 2 * (2 if loop else 1))
    return macs * (2.0 if real else 8.0)


def _tor_flops(k):
    """Sums over 2^k subsets by the recursion over modes on Schur complements: including a
    mode with m left updates m (2m + 1) entries with two products each."""
    return sum(2.0 ** (k - m - 1) * (4.0 * m * (2 * m + 1) + 20.0) for m in range(k))


def _flops(func, n, real):
    if func == "perm":
        return 2.0 ** (n - 1) * (3 * n - 1 if real else 10 * n - 4)
    if func == "tor":
        return _tor_flops(n)
    return _haf_flops(n, func == "lhaf", real)


def work(case):
    kind = case["kind"]
    width = {"dd": 20.0, "certified": 2.0}.get(case.get("precision"), 1.0)
    if kind in ("one", "stack"):
        b, n = case.get("batch", 1), case["n"]
        side = 2 * n if case["func"] == "tor" else n
        return {"bytes": b * ((8 if case["real"] else 16) * side * side + 16), "flops": b * width * _flops(case["func"], n, case["real"])}
    if kind in ("queue", "auto", "clicks"):
        sizes = _sizes(case)
        f = {"auto": lambda i, n: _haf_flops(n, True, False), "queue": lambda i, n: _haf_flops(n, i % 2 == 1, False),
             "clicks": lambda i, n: _tor_flops(n)}[kind]
        entry = 32 if kind == "clicks" else 16
        return {"bytes": sum(entry * n * n * (2 if kind == "clicks" else 1) + 16 for n in sizes),
                "flops": sum(f(i, n) for i, n in enumerate(sizes))}
    if kind == "sieve":
        m, most = case["modes"], case["most"]
        terms = case["batch"] * (1 + most / 2.0) ** m / 2  # the mean pattern, v and n - v counted once
        return {"bytes": case["batch"] * (4 * m + 16) + 16 * m * m, "flops": terms * (8 * m + 8 * m * most / 2.0 + 12)}
    # every distinct prefix once: at most (cutoff + 1)^k, no more than the samples
    flops = 0.0
    for k in range(1, case["modes"] + 1):
        prefixes = min(case["samples"], (case["cutoff"] + 1) ** (k - 1))
        flops += prefixes * sum(_haf_flops(2 * (j + k // 2), False, False) for j in range(1, case["cutoff"] + 1))
    return {"bytes": 8 * case["samples"] * case["modes"] + 64 * case["modes"] ** 3, "flops": flops}


def tolerance(case):
    kind = case["kind"]
    if kind == "sampler":
        return {"rel": 0.0, "differ": 1e-5}  # a draw on the edge of its interval
    if kind == "clicks":
        # the alternating sum of 2^k determinants cancels by a factor of about 10^(k - 2)
        return {"rel": 1e-2 if case["hi"] > 16 else 1e-4 if case["hi"] > 10 else 1e-6}
    if case.get("precision") == "dd":
        return {"rel": 4e-15}
    if case.get("func") == "tor":
        return {"rel": 1e-4 if case["n"] > 12 else 1e-6 if case["n"] > 8 else 1e-9}
    if case.get("func") == "perm":
        return {"rel": 1e-12}
    return {"rel": 1e-10}


# ------------------------------------------------------------------ the same numbers, in 64 bits
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _signs(bits, n):
    s = torch.ones(bits.shape[0], dtype=torch.float64, device=bits.device)
    return s * (1.0 - 2.0 * ((n - bits.sum(1)) % 2).double())


def _bits(lo, hi, n, dev):
    ids = torch.arange(lo, hi, device=dev)
    return (ids[:, None] >> torch.arange(n, device=dev)[None]) & 1


def _haf64(A, loop):
    """Sum over subsets of pairs of the z^n coefficient of exp(traces): the power-trace formula."""
    if A.shape[0] % 2:
        A = np.block([[A, np.zeros((A.shape[0], 1))], [np.zeros((1, A.shape[0])), np.ones((1, 1))]])
    n = A.shape[0] // 2
    dev = _device()
    B = torch.as_tensor(A.astype(np.complex128), device=dev)
    d = torch.diagonal(B).clone()
    B = (B + B.T) / 2
    swap = torch.arange(2 * n, device=dev) ^ 1
    total = 0.0
    step = max(1, 1 << 25 >> (2 * int(math.log2(2 * n)) + 1))
    for lo in range(0, 1 << n, step):
        bits = _bits(lo, min(lo + step, 1 << n), n, dev)
        mask = bits.repeat_interleave(2, 1).to(B.dtype)
        C = (B[None] * mask[:, :, None] * mask[:, None, :])[:, :, swap]
        dm = d[None] * mask
        y = dm
        P = C
        e = [torch.ones(bits.shape[0], dtype=B.dtype, device=dev)]
        kg = []
        for k in range(1, n + 1):
            g = torch.einsum("bii->b", P) / 2
            if loop:
                g = g + k * (dm[:, swap] * y).sum(1) / 2
                y = torch.einsum("bij,bj->bi", C, y)
            kg.append(g)
            e.append(sum(kg[i] * e[k - 1 - i] for i in range(k)) / k)
            if k < n:
                P = P @ C
        total = total + (_signs(bits, n).to(B.dtype) * e[n]).sum()
    return complex(total)


def _perm64(A):
    """Ryser's sum over subsets of columns."""
    n = A.shape[0]
    dev = _device()
    B = torch.as_tensor(A.astype(np.complex128), device=dev)
    total = 0.0
    for lo in range(0, 1 << (n - 1), 1 << 18):  # Glynn: the first sign is +
        bits = _bits(lo, min(lo + (1 << 18), 1 << (n - 1)), n - 1, dev)
        delta = torch.cat([torch.ones(bits.shape[0], 1, device=dev, dtype=torch.float64), 1.0 - 2.0 * bits.double()], 1)
        total = total + (torch.prod(delta, 1).to(B.dtype) * torch.prod(delta.to(B.dtype) @ B.T, 1)).sum()
    return complex(total) / 2.0 ** (n - 1)


def _tor64(O):
    k = O.shape[0] // 2
    dev = _device()
    M = torch.as_tensor(np.eye(2 * k) - np.real(O), device=dev)
    eye = torch.eye(2 * k, dtype=torch.float64, device=dev)
    total = 0.0
    for lo in range(0, 1 << k, 1 << 14):
        bits = _bits(lo, min(lo + (1 << 14), 1 << k), k, dev)
        mask = torch.cat([bits, bits], 1).double()
        S = M[None] * mask[:, :, None] * mask[:, None, :] + eye[None] * (1.0 - mask)[:, None, :]
        det = torch.prod(torch.diagonal(torch.linalg.cholesky(S), dim1=1, dim2=2), 1)
        total = total + (_signs(bits, k) / det).sum()
    return float(total)


def _lhaf_repeated64(A, gamma, reps):
    idx = np.repeat(np.arange(len(reps)), reps)
    S = A[np.ix_(idx, idx)].copy()
    np.fill_diagonal(S, gamma[idx])
    return _haf64(S, True) if len(idx) else 1.0


def _value64(func, A):
    if func == "perm":
        return _perm64(A)
    if func == "tor":
        return _tor64(A)
    if func == "haf" and A.shape[0] % 2:
        return 0.0
    return _haf64(A, func == "lhaf")


def _cost64(func, n):
    if func == "perm":
        return 2.0 ** n * n * n + 1e6
    if func == "tor":
        return 2.0 ** n * (2 * n) ** 3 * 2 + 2e7
    return 2.0 ** ((n + 1) // 2) * 8 * (n / 2 + 1) * n ** 3 + 4e7


def exact(case, seed):
    kind = case["kind"]
    if kind in ("sieve", "sampler"):
        if kind == "sampler" or case["modes"] * case["most"] > 14 or case["batch"] > 400:
            return None
        s = _inputs(case, seed)
        return np.array([_lhaf_repeated64(s["A"], s["gamma"], r) for r in s["reps"]], dtype=np.complex128)
    if kind in ("one", "stack"):
        cost = case.get("batch", 1) * _cost64(case["func"], case["n"])
    elif kind == "clicks":
        cost = sum(_cost64("tor", n) for n in _sizes(case))
    else:
        cost = sum(_cost64("lhaf", n) for n in _sizes(case))
    if cost > (4e12 if _device().type == "cuda" else 1e11):
        return None
    s = _inputs(case, seed)
    if kind == "one":
        v = complex(_value64(case["func"], s["mat"]))
        return v.real if case["real"] else _parts(v)
    if kind == "stack":
        values = np.array([_value64(case["func"], m) for m in s["stack"]], dtype=np.complex128)
        return (values, None) if case["precision"] == "certified" else values
    if kind == "clicks":
        return np.array([_value64("tor", m) for m in s["mats"]], dtype=np.complex128)
    return np.array([_value64(f, m) for f, m in zip(s["funcs"], s["mats"])], dtype=np.complex128)
