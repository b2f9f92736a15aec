#!/usr/bin/env python
"""bench.py -- persistent mixed-size hafnian / loop-hafnian throughput on B200.

Workload (one "step"): one pass of the work-item kernel over the persistent
mixed-size batch -- 65,536 complex instances, N uniform over the even sizes 8..28,
function 50/50 haf / lhaf, each a submatrix (repeated rows of a random photon
pattern) of A = U diag(tanh 1) U^T, U a seeded Haar 100 x 100 unitary, with loop
weights gamma ~ CN(0, 0.1) on the loop-hafnian diagonals (gbskernels_b200.workloads).

  value    instances/s of the persistent queue, inputs resident in HBM (CUDA events
           on the launching stream, max over ranks)
  e2e      the same through the public API (Workspace.evaluate) from host numpy
           buffers, H2D of the matrices and D2H of the results inside the timed region
  plain_per_size  the same batch as one launch per (function, size) bucket
  roofline FP64 flops of the batch by the algorithm in use (workloads.walk_flops) /
           kernel time, against the FP64 peak measured live by gbs_probe_fp64_peak
  cpu_baseline    the oracle (binary64 restatement of the reference algorithm) on the
           host cores, stratified sample: three haf + three lhaf instances per size class
  plain_per_size_sync  the reference's plain per-size path (gbskernels/__init__.py:
           813-852 over core/host_api.cu:537-590): one synchronous session call per
           (function, size) bucket -- stack, H2D, launch, D2H, sync -- and a host
           scatter, end to end from numpy, against this library's e2e
  batch_sweep     the persistent queue against both per-size paths at 256..16384
           instances of the same mix (where one launch per size underfills the GPU)
  configs  the other benchmark configurations, each on its own batch: real 16 x 16
           hafnians (fp64, certified), Haar 20 x 20 permanents (fp64, dd), threshold
           torontonians at 10..24 modes (fp64, certified), with parity spot checks;
           the repeated-row sieve and the resident sampler chain (host-call rates)
  serving  the chain-rule query stream from resident states at 0.8 x and 3 x the
           offline rate (the second saturates: its throughput is the capacity), and
           at the configuration's arrival rates 1e3 .. 1e5 requests/s
  check    one haf + one lhaf instance per size class 8..28 of this batch against
           the binary128 oracle (N <= 20) or the binary64 oracle port scaled by the
           instance's cancellation indicator (N >= 22)

Multi-GPU (torchrun): replicas only -- each rank evaluates its own batch (weak
scaling), no collective on the data path; the barrier and the max-over-ranks time
use torch.distributed.

--impl reference times the reference's own CPU implementation of the path (the
reference kernels compiled on the host, oracle/_ref, for the sizes they support,
N <= 20; the oracle port above) on the same workload and metric.
"""

from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import threading
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

METRIC = "mixed-size instances/s (persistent queue) & p99 latency vs plain per-size launch; rel err <= 1e-10"
SIZES = tuple(range(8, 29, 2))


def _args():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--batch", type=int, default=65536)
    ap.add_argument("--seed", type=int, default=3)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-per-size", action="store_true")
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--no-serving", action="store_true")
    ap.add_argument("--no-sweep", action="store_true")
    ap.add_argument("--no-configs", action="store_true")
    ap.add_argument("--tuned", default=None,
                    help="apply an autotuner table (gbskernels_b200.autotune JSON) before timing")
    ap.add_argument("--profile-small", action="store_true",
                    help="small case for ncu captures: 256 instances, 1 step, no extras")
    return ap.parse_args()


# ---------------------------------------------------------------- distributed plumbing
class Dist:
    def __init__(self):
        self.world = int(os.environ.get("WORLD_SIZE", "1"))
        self.rank = int(os.environ.get("RANK", "0"))
        self.local = int(os.environ.get("LOCAL_RANK", "0"))
        self.pg = None

    def init(self, backend="nccl"):
        if self.world > 1:
            import datetime
            import torch.distributed as dist
            dist.init_process_group(backend, timeout=datetime.timedelta(seconds=600))
            self.pg = dist

    def barrier(self):
        if self.pg:
            self.pg.barrier()

    def max(self, x: float) -> float:
        if not self.pg:
            return x
        import torch
        t = torch.tensor([x], dtype=torch.float64, device="cuda")
        self.pg.all_reduce(t, op=self.pg.ReduceOp.MAX)
        return float(t.item())

    def close(self):
        if self.pg:
            self.pg.destroy_process_group()


# ---------------------------------------------------------------- clocks sampler
class Clocks:
    """nvidia-smi sampled every 200 ms during the timed region."""

    FIELDS = ("clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu: int):
        self.gpu = gpu
        self.proc = None
        self.lines: list[str] = []

    def start(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.gpu), f"--query-gpu={self.FIELDS}",
                 "--format=csv,noheader,nounits", "-lms", "200"],
                stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except OSError:
            self.proc = None

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def stop(self) -> dict:
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        sm, smax, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            parts = [p.strip() for p in ln.split(",")]
            if len(parts) < 8:
                continue
            try:
                sm.append(float(parts[0]))
                smax.append(float(parts[1]))
            except ValueError:
                continue
            for nm, v in zip(names, parts[4:8]):
                if v.lower().startswith("active"):
                    reasons.add(nm)
        return {"sm_mhz": statistics.median(sm) if sm else None,
                "sm_max_mhz": max(smax) if smax else None,
                "reasons": sorted(reasons), "samples": len(sm)}


# ---------------------------------------------------------------- CPU baselines
def _cpu_task(args):
    """Evaluate one instance on the host; returns (func, N, seconds, value, code) with
    code "reference" when the reference's own kernel ran, "port" for the oracle."""
    impl, func, mat = args
    sys.path.insert(0, str(ROOT))
    import oracle
    t0 = time.perf_counter()
    if impl == "reference" and mat.shape[0] <= 20 and oracle.ref_available():
        v = complex(oracle.ref_batched(func, mat[None])[0])
        code = "reference"
    else:
        v = getattr(oracle, func)(mat)
        code = "port"
    return func, mat.shape[0], time.perf_counter() - t0, v, code


PER_CLASS = 3  # sampled instances per (function, size) class


def cpu_sample_rate(impl: str, funcs, mats, cores: int):
    """Stratified sample: the first PER_CLASS haf and lhaf instances of every size
    class.  Returns (instances/s on `cores` cores for the uniform-over-sizes mix,
    details).  impl "reference": the reference's own kernels (compiled on the host)
    where they accept the size (N <= 20: core/hafnian.cu:28 and
    core/loop_hafnian.cu:24 fix 20-wide per-thread arrays), the oracle port above;
    details record the share of the sampled time each one took."""
    picked: dict = {}
    for f, m in zip(funcs, mats):
        lst = picked.setdefault((f, m.shape[0]), [])
        if len(lst) < PER_CLASS:
            lst.append(m)
    tasks = [(impl, f, m) for (f, _), ms in sorted(picked.items(), key=lambda kv: -kv[0][1]) for m in ms]
    import multiprocessing as mp
    ctx = mp.get_context("spawn")
    t0 = time.perf_counter()
    with ctx.Pool(min(cores, len(tasks))) as pool:
        res = pool.map(_cpu_task, tasks, chunksize=1)
    wall = time.perf_counter() - t0
    per: dict = {}
    for f, N, t, _, _ in res:
        per.setdefault((f, N), []).append(t)
    # uniform over the classes, as the batch is: the mean of the class means
    mean_t = float(np.mean([np.mean(v) for v in per.values()]))
    rate = cores / mean_t  # instances are independent: every core runs its own
    t_ref = sum(r[2] for r in res if r[4] == "reference")
    t_all = sum(r[2] for r in res)
    return rate, {"cpu_seconds": float(t_all), "wall_s": wall, "instances": len(res),
                  "reference_code_share_of_time": float(t_ref / t_all) if t_all else 0.0,
                  "per_class_s": {f"{f}{N}": round(float(np.mean(t)), 4) for (f, N), t in sorted(per.items())}}


def run_reference(a, dist: Dist):
    """--impl reference: the reference's own CPU implementation, rank 0 only."""
    if dist.rank != 0:
        return
    from gbskernels_b200 import workloads
    import oracle
    funcs, mats = workloads.mixed_haf_lhaf(2 * len(SIZES) * 8, seed=a.seed)
    cores = len(os.sched_getaffinity(0))
    kind = "reference" if oracle.ref_available() else "port"
    for _ in range(max(a.warmup, 0)):
        cpu_sample_rate("reference", funcs, mats, cores)
    times, rates = [], []
    for _ in range(a.steps):
        t0 = time.perf_counter()
        rate, det = cpu_sample_rate("reference", funcs, mats, cores)
        times.append(time.perf_counter() - t0)
        rates.append(rate)
    v = float(np.median(rates))
    sample = (f"{PER_CLASS} haf + {PER_CLASS} lhaf instances per size class N = 8..28 of the mixed batch; "
              "the reference's own kernels (core/hafnian.cu, core/loop_hafnian.cu built on the host) "
              "for N <= 20, the oracle port of the same algorithm above (both reference kernels fix "
              "20-wide per-thread arrays); rate = cores / mean of the class-mean times; "
              f"{100 * det['reference_code_share_of_time']:.1f} % of the sampled time ran reference code")
    line = {"metric": METRIC, "value": v, "unit": "instances/s", "n_gpus": a.gpus, "steps": a.steps,
            "warmup": a.warmup, "ms_per_step": 1e3 * float(np.median(times)), "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "impl": "reference",
            "config": {"workload": "persistent mixed-size haf+lhaf, complex, N uniform over 8..28",
                       "batch": a.batch},
            "cpu_baseline": {"value": v, "unit": "instances/s", "cores": cores, "kind": kind,
                             "sample": sample,
                             "reference_code_share_of_time": det["reference_code_share_of_time"]},
            "e2e": {"value": v, "unit": "instances/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)



# ---------------------------------------------------------------- parity spot check
def _check_task(args):
    func, mat, prec = args
    sys.path.insert(0, str(ROOT))
    import oracle
    if prec == "quad":
        return complex(getattr(oracle, func)(mat, "quad")), None
    v, absn = getattr(oracle, func)(mat, "fp64", with_absnorm=True)
    return complex(v), float(absn)


def parity_check(funcs, mats, out, cores):
    """One haf + one lhaf per size class against the oracle: binary128 for N <= 20,
    the binary64 port above with the tolerance max(1e-10, 16 N u kappa), kappa the
    port's sum|term| / |value| (both walks err by about N u kappa)."""
    picked = {}
    for i, (f, m) in enumerate(zip(funcs, mats)):
        picked.setdefault((f, m.shape[0]), i)
    idx = sorted(picked.values(), key=lambda i: -mats[i].shape[0])
    tasks = [(funcs[i], mats[i], "quad" if mats[i].shape[0] <= 20 else "fp64") for i in idx]
    import multiprocessing as mp
    with mp.get_context("spawn").Pool(min(cores, len(tasks))) as pool:
        res = pool.map(_check_task, tasks, chunksize=1)
    worst_q, worst_p, ok = 0.0, 0.0, True
    for i, (ref, absn) in zip(idx, res):
        err = abs(out[i] - ref) / abs(ref)
        if absn is None:
            worst_q = max(worst_q, err)
            ok &= err <= 1e-10
        else:
            tol = max(1e-10, 16 * mats[i].shape[0] * 2.0 ** -53 * absn / abs(ref))
            worst_p = max(worst_p, err / tol)
            ok &= err <= tol
    return {"instances": len(idx), "max_rel_err_vs_binary128_N<=20": float(worst_q),
            "max_err_over_tol_vs_binary64_port_N>=22": float(worst_p), "pass": bool(ok)}


# ---------------------------------------------------------------- reference-style per-size path
def per_size_sync(lib, sess, funcs, mats):
    """The reference's plain per-size path (gbskernels/__init__.py:813-852): group by
    (function, size) in first-seen order, one synchronous session call per bucket
    (stack, H2D, launch, D2H, sync: gbs_session_evaluate, as core/host_api.cu:537-590),
    scatter to input order."""
    from gbskernels_b200 import _lib
    buckets: dict = {}
    for i, (f, m) in enumerate(zip(funcs, mats)):
        buckets.setdefault((f, m.shape[0]), []).append(i)
    out = np.empty(len(mats), np.complex128)
    code = {"perm": 0, "haf": 1, "lhaf": 2, "tor": 3}
    for (f, d), idxs in buckets.items():
        stack = np.ascontiguousarray(np.stack([mats[i] for i in idxs]))
        res = np.empty(len(idxs), np.complex128)
        _lib.check(lib.gbs_session_evaluate(sess, code[f], 0, _lib.dptr(stack.view(np.float64)), d, len(idxs),
                                            _lib.dptr(res.view(np.float64))), "gbs_session_evaluate")
        out[idxs] = res
    return out


def batch_sweep(G, lib, sizes, seed, stream, sptr):
    """Persistent queue vs the two per-size paths at several batch sizes of the mix."""
    import torch
    from gbskernels_b200 import _lib, workloads
    rows = []
    for B in sizes:
        funcs, mats = workloads.mixed_haf_lhaf(B, seed=seed + 100 + B)
        fcode = np.array([{"haf": 1, "lhaf": 2}[f] for f in funcs], np.int32)
        tiers = np.zeros(B, np.int32)
        buf, dims, offs = G._pack(mats)
        row = {"batch": B}
        with G.Workspace() as ws, G.Workspace() as ws2:
            reps = 3 if B <= 4096 else 2
            for mode, key in ((0, "persistent_ms"), (1, "per_size_ms")):
                _lib.check(lib.gbs_queue_prepare(ws._session, B, _lib.iptr(fcode), _lib.iptr(tiers), _lib.iptr(dims),
                                                 _lib.llptr(offs), _lib.dptr(buf.view(np.float64)), mode), "prepare")
                for _ in range(2):
                    _lib.check(lib.gbs_queue_run(ws._session, sptr), "run")
                torch.cuda.synchronize()
                e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                e0.record(stream)
                for _ in range(reps):
                    _lib.check(lib.gbs_queue_run(ws._session, sptr), "run")
                e1.record(stream)
                torch.cuda.synchronize()
                row[key] = e0.elapsed_time(e1) / reps
            precs = ["fp64"] * B
            ref = ws.evaluate(funcs, mats, precs)
            per_size_sync(lib, ws2._session, funcs, mats)  # warm
            t_e, t_s = [], []
            for _ in range(reps):
                t0 = time.perf_counter()
                r1 = ws.evaluate(funcs, mats, precs)
                t_e.append(time.perf_counter() - t0)
                t0 = time.perf_counter()
                r2 = per_size_sync(lib, ws2._session, funcs, mats)
                t_s.append(time.perf_counter() - t0)
            row["e2e_persistent_ms"] = 1e3 * float(np.median(t_e))
            row["e2e_per_size_sync_ms"] = 1e3 * float(np.median(t_s))
            row["speedup_resident_vs_per_size"] = row["per_size_ms"] / row["persistent_ms"]
            row["speedup_e2e_vs_per_size_sync"] = row["e2e_per_size_sync_ms"] / row["e2e_persistent_ms"]
            row["values_equal"] = bool(np.array_equal(r1, ref) and np.array_equal(r2, ref))
        rows.append(row)
    return rows


# ---------------------------------------------------------------- the other configurations
def _cfg_task(args):
    kind, mat = args
    sys.path.insert(0, str(ROOT))
    import oracle
    return complex(getattr(oracle, kind)(mat, "quad"))


def other_configs(G, peak, cores):
    """Configs 1, 2 and 4 on their own batches (persistent queue, kernel time by the
    session's CUDA events; warm-up run first), with parity spot checks."""
    from gbskernels_b200 import configs, workloads
    out = {}
    flops = workloads.walk_flops
    jobs = []
    # config 1: 4096 real symmetric 16 x 16 hafnians
    c1 = list(workloads.haf_real_batch(4096, 16, seed=1))
    f1 = 4096 * flops("haf", 16, real=True)
    r, v, a, st = configs.run("haf", c1, "fp64", reps=3)
    rc, vc, ac, stc = configs.run("haf", c1, "certified", reps=2)
    out["config1_haf16_real"] = {
        "batch": 4096, "value": r["instances_per_s"], "unit": "instances/s", "kernel_ms": r["kernel_ms"],
        "roofline_frac": f1 / (r["kernel_ms"] * 1e-3) / 1e12 / peak,
        "certified": {"value": rc["instances_per_s"], "rel_bound_median": rc["rel_bound_median"],
                      "values_equal_fp64": bool(np.array_equal(vc, v))}}
    jobs += [("c1", i, "haf", c1[i].astype(np.complex128), v[i], ac[i]) for i in range(4)]
    # config 2: 1024 Haar 20 x 20 permanents
    c2 = list(workloads.perm_haar_batch(1024, 20, seed=2))
    f2 = 1024 * flops("perm", 20)
    r, v2, _, _ = configs.run("perm", c2, "fp64", reps=3)
    rd, vd, _, _ = configs.run("perm", c2, "dd", reps=1)
    out["config2_perm20"] = {
        "batch": 1024, "value": r["instances_per_s"], "unit": "instances/s", "kernel_ms": r["kernel_ms"],
        "roofline_frac": f2 / (r["kernel_ms"] * 1e-3) / 1e12 / peak,
        "dd": {"value": rd["instances_per_s"], "kernel_ms": rd["kernel_ms"]}}
    jobs += [("c2", i, "perm", c2[i], v2[i], vd[i]) for i in range(2)]
    # config 4: 8192 threshold torontonians, 10..24 modes
    c4 = workloads.tor_click_batch(8192, seed=4)
    f4 = sum(flops("tor", m.shape[0]) for m in c4)
    r, v4, _, st4 = configs.run("tor", c4, "fp64", reps=2)
    rc4, vc4, ac4, stc4 = configs.run("tor", c4, "certified", reps=1)
    out["config4_tor_k10to24"] = {
        "batch": 8192, "value": r["instances_per_s"], "unit": "instances/s", "kernel_ms": r["kernel_ms"],
        "roofline_frac": f4 / (r["kernel_ms"] * 1e-3) / 1e12 / peak, "status_ok": int((st4 == 0).sum()),
        "certified": {"value": rc4["instances_per_s"], "rel_bound_median": rc4["rel_bound_median"],
                      "values_equal_fp64": bool(np.array_equal(vc4, v4))}}
    small = [i for i, m in enumerate(c4) if m.shape[0] <= 28][:4]
    jobs += [("c4", i, "tor", c4[i], v4[i], ac4[i]) for i in small]
    import multiprocessing as mp
    with mp.get_context("spawn").Pool(min(cores, len(jobs))) as pool:
        truth = pool.map(_cfg_task, [(k, m) for _, _, k, m, _, _ in jobs], chunksize=1)
    checks = {"config1_haf16_real": [], "config2_perm20": [], "config4_tor_k10to24": []}
    keyof = {"c1": "config1_haf16_real", "c2": "config2_perm20", "c4": "config4_tor_k10to24"}
    for (c, i, kind, m, val, extra), t in zip(jobs, truth):
        e = {"rel_err": abs(val - t) / abs(t)}
        if c in ("c1", "c4"):
            e["certified_encloses"] = bool(abs(val - t) <= extra)  # extra = certified bound
        else:
            e["dd_rel_err"] = abs(extra - t) / abs(t)
        checks[keyof[c]].append(e)
    for k, lst in checks.items():
        out[k]["check_vs_binary128_oracle"] = {
            "instances": len(lst), "max_rel_err": float(max(x["rel_err"] for x in lst)),
            "certified_enclose": all(x.get("certified_encloses", True) for x in lst),
            "max_dd_rel_err": max((float(x["dd_rel_err"]) for x in lst if "dd_rel_err" in x), default=None)}
    # beside the power-trace path: the repeated-row sieve and the resident sampler chain
    out["sieve_lhaf_repeated"] = configs.sieve_rate()
    out["sampler_chain"] = configs.sampler_rate()
    return out

# ---------------------------------------------------------------- our implementation
def main():
    a = _args()
    dist = Dist()
    if a.impl == "reference":
        dist.init("gloo")
        try:
            run_reference(a, dist)
        finally:
            dist.close()
        return
    import torch
    torch.cuda.set_device(dist.local)
    dist.init("nccl")
    import ctypes
    import gbskernels_b200 as G
    from gbskernels_b200 import _lib, workloads
    lib = _lib.load()

    if a.tuned:
        from gbskernels_b200 import autotune
        autotune.load(a.tuned)
    B = 256 if a.profile_small else a.batch
    funcs, mats = workloads.mixed_haf_lhaf(B, seed=a.seed + dist.rank)
    fcode = np.array([{"haf": 1, "lhaf": 2}[f] for f in funcs], dtype=np.int32)
    tiers = np.zeros(B, dtype=np.int32)
    buf, dims, offs = G._pack(mats)
    in_bytes = buf.nbytes
    algo_flops = float(sum(workloads.walk_flops(f, m.shape[0]) for f, m in zip(funcs, mats)))
    ref_flops = float(sum(workloads.ref_flops(f, m.shape[0]) for f, m in zip(funcs, mats)))

    ws = G.Workspace()
    ws.__enter__()
    sess = ws._session
    # a dedicated stream: the launches and the CUDA events that time them share it
    stream = torch.cuda.Stream()
    torch.cuda.set_stream(stream)
    sptr = ctypes.c_void_p(stream.cuda_stream)

    def prepare(mode):
        _lib.check(lib.gbs_queue_prepare(sess, B, _lib.iptr(fcode), _lib.iptr(tiers), _lib.iptr(dims),
                                         _lib.llptr(offs), _lib.dptr(buf.view(np.float64)), mode),
                   "gbs_queue_prepare")

    def run_steps(k):
        for _ in range(k):
            _lib.check(lib.gbs_queue_run(sess, sptr), "gbs_queue_run")

    def timed(k):
        dist.barrier()
        torch.cuda.synchronize()
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        run_steps(k)
        e1.record(stream)
        torch.cuda.synchronize()
        dist.barrier()
        return e0.elapsed_time(e1) / 1e3

    # ---- persistent mixed queue, inputs resident in HBM
    prepare(0)
    run_steps(max(a.warmup, 1))
    torch.cuda.synchronize()
    clocks = Clocks(dist.local)
    clocks.start()
    t_local = timed(a.steps)
    clk = clocks.stop()
    t = dist.max(t_local)
    out = np.empty(B, dtype=np.complex128)
    st = np.zeros(B, dtype=np.int32)
    _lib.check(lib.gbs_queue_read(sess, sptr, _lib.dptr(out.view(np.float64)), None, _lib.iptr(st)),
               "gbs_queue_read")
    stats = ws.last_stats()
    launches_per_step = stats["launches"]
    value = dist.world * B * a.steps / t
    step_s = t / a.steps
    achieved = algo_flops / step_s / 1e12

    # ---- roofline denominator: FP64 tensor-core throughput of this GPU
    tf = np.zeros(1)
    pms = ctypes.c_float(0)
    _lib.check(lib.gbs_probe_fp64_peak(_lib.dptr(tf), ctypes.byref(pms)), "gbs_probe_fp64_peak")
    peak = float(tf[0])

    # ---- parity spot check on this run's own results: one haf + one lhaf per size
    # class 8..28 against the oracle (the checker; nothing timed depends on it)
    check = {"finite": bool(np.all(np.isfinite(out))), "status_ok": bool(np.all(st == 0))}
    if dist.rank == 0 and not a.profile_small:
        check.update(parity_check(funcs, mats, out, len(os.sched_getaffinity(0))))

    line = {"metric": METRIC, "value": value, "unit": "instances/s", "n_gpus": dist.world,
            "steps": a.steps, "warmup": a.warmup, "ms_per_step": 1e3 * step_s,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
            "data": "synthetic",
            "config": {"workload": f"persistent mixed-size queue, {B} complex instances, haf/lhaf 50/50, "
                                   f"N uniform over even 8..28, A = U diag(tanh 1) U^T (Haar 100x100), "
                                   f"photon-pattern submatrices, gamma ~ CN(0,0.1)",
                       "batch": B, "parallelism": f"replicas x{dist.world}",
                       "l2": f"inputs {in_bytes / 1e6:.0f} MB per rank > 126 MB L2 (no flush needed)"},
            "roofline": {"bound": "fp64", "achieved": achieved, "peak": peak, "unit": "TFLOP/s",
                         "frac": achieved / peak,
                         # each matrix is read once and each value written once
                         "traffic": in_bytes + 28 * B,
                         "traffic_unit": "bytes per launch (inputs and results, not measured)",
                         "peak_source": "FP64 mma.m16n8k8 throughput measured live (gbs_probe_fp64_peak), the "
                                        "same as the FMA pipe's; MEASURED_PEAKS.json has no FP64 figure",
                         "flops_per_step": algo_flops, "reference_flops_per_step": ref_flops,
                         "flops_note": "flops of the recursion over pairs; the reference's power trace would "
                                       "take reference_flops_per_step"},
            "clocks": clk, "gpu_launches": launches_per_step * a.steps, "check": check}

    if a.profile_small:
        if dist.rank == 0:
            print(json.dumps(line), flush=True)
        ws.close()
        dist.close()
        return

    # ---- plain per-size launches of the same batch
    if not a.no_per_size:
        prepare(1)
        run_steps(1)
        torch.cuda.synchronize()
        k2 = max(1, min(a.steps, 3))
        t2 = dist.max(timed(k2))
        ps_launches = ws.last_stats()["launches"]
        out2 = np.empty(B, dtype=np.complex128)
        _lib.check(lib.gbs_queue_read(sess, sptr, _lib.dptr(out2.view(np.float64)), None, None), "read")
        v2 = dist.world * B * k2 / t2
        line["plain_per_size"] = {"value": v2, "unit": "instances/s", "ms_per_step": 1e3 * t2 / k2,
                                  "launches_per_step": ps_launches,
                                  "persistent_speedup": value / v2,
                                  "bitwise_equal_to_persistent": bool(np.array_equal(out, out2))}

    # ---- end to end through the public API (host buffers)
    if not a.no_e2e:
        precs = ["fp64"] * B
        ws.evaluate(funcs, mats, precs)  # warm
        k3 = max(1, min(a.steps, 3))
        dist.barrier()
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        for _ in range(k3):
            r = ws.evaluate(funcs, mats, precs)
        torch.cuda.synchronize()
        t3 = dist.max(time.perf_counter() - t0)
        line["e2e"] = {"value": dist.world * B * k3 / t3, "unit": "instances/s",
                       "h2d_bytes_per_step": int(in_bytes + B * 56),
                       "d2h_bytes_per_step": int(B * (16 + 8 + 4)),
                       "path": "gbskernels_b200.Workspace.evaluate (numpy in, numpy out)",
                       "equal_to_resident_run": bool(np.array_equal(r, out))}

    # ---- the reference's plain per-size path, end to end from numpy (one synchronous
    # session call per (function, size) bucket), against the e2e line above
    if not a.no_per_size and not a.no_e2e:
        with G.Workspace() as ws2:
            per_size_sync(lib, ws2._session, funcs, mats)  # warm
            k4 = max(1, min(a.steps, 3))
            dist.barrier()
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            for _ in range(k4):
                r4 = per_size_sync(lib, ws2._session, funcs, mats)
            torch.cuda.synchronize()
            t4 = dist.max(time.perf_counter() - t0)
        v4 = dist.world * B * k4 / t4
        line["plain_per_size_sync"] = {
            "value": v4, "unit": "instances/s", "ms_per_step": 1e3 * t4 / k4,
            "buckets": len({(f, m.shape[0]) for f, m in zip(funcs, mats)}),
            "path": "per (function, size) bucket: np.stack, gbs_session_evaluate (H2D, launch, D2H, sync), "
                    "host scatter -- gbskernels/__init__.py:813-852 over core/host_api.cu:537-590",
            "e2e_persistent_speedup": line["e2e"]["value"] / v4,
            "values_equal": bool(np.array_equal(r4, out))}

    # ---- batch-size sweep: where one launch per size underfills the GPU
    if not a.no_sweep and dist.world == 1:
        line["batch_sweep"] = batch_sweep(G, lib, (256, 1024, 4096, 16384), a.seed, stream, sptr)

    # ---- the other configurations (own batches)
    if not a.no_configs and dist.world == 1:
        line["configs"] = other_configs(G, peak, len(os.sched_getaffinity(0)))

    # ---- CPU baseline (rank 0, one GPU)
    if not a.no_cpu_baseline and dist.world == 1:
        cores = len(os.sched_getaffinity(0))
        rate, det = cpu_sample_rate("port", funcs, mats, cores)
        line["cpu_baseline"] = {"value": rate, "unit": "instances/s", "cores": cores, "kind": "port",
                                "sample": f"{PER_CLASS} haf + {PER_CLASS} lhaf instances per size class "
                                          "N = 8..28 of this batch, oracle (binary64 restatement of the "
                                          "reference power trace) one process per core; rate = cores / "
                                          f"mean of the class-mean times ({det['cpu_seconds']:.1f} CPU-s)"}

    # ---- serving loop: chain-rule queries on resident states, p50 / p99 latency
    # beside throughput, below and above the offline rate
    if not a.no_serving and dist.world == 1:
        from gbskernels_b200.serving import offline_rate, serve_stream
        off = offline_rate(2000, 5)
        line["serving"] = serve_stream(rate=None, rate_frac=0.8, n_req=2000, seed=5, offline=off)
        line["serving_saturated"] = serve_stream(rate=None, rate_frac=3.0, n_req=2000, seed=5, offline=off)
        # the configuration's own arrival rates (Poisson, 2000 requests each)
        keep = ("offered_rate", "throughput", "throughput_vs_offline", "p50_ms", "p99_ms", "batches",
                "values_equal_to_offline_batch")
        line["serving_rate_sweep"] = [
            {k: r[k] for k in keep} for r in
            (serve_stream(rate=lam, n_req=2000, seed=5, offline=off) for lam in (1e3, 3e3, 1e4, 3e4, 1e5))]

    if dist.rank == 0:
        print(json.dumps(line), flush=True)
    ws.close()
    dist.close()


if __name__ == "__main__":
    main()
