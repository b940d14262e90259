"""Benchmark of the block-sparse contraction (one JSON line of a few KB on standard output, rank 0; the full
record, with every configuration, serving phase and CPU leg, goes to standard error as one more line).

Headline workload (``--workload c1``, the default): C[i,j,a,b] = sum_P A[i,a,P] B[j,b,P] at full
size (i,j extent 64 in blocks of {5,9,13}; a,b 512 in {13,25,32}; P 2048 in {32,48,64}; 15%
block occupancy; seeded values).  A step is one full contraction C = A.B on the device: block
matching, result pattern, work list and the tile kernel, inputs resident in HBM.  Metric:
effective GFLOP/s = sum over pairs of 2*m*n*k / step time.  Every FP64-accurate form is timed
and the fastest is `value`; all are listed under `forms`, each checked against the CPU oracle
on the full workload (pattern and pair list bit-exact, values bit-exact for the FP64 forms and
within 1e-12 relative Frobenius for the split form).  The other configurations (c0, c2, c3)
are timed and checked the same way under `configs`.

`--impl reference` times the reference's CPU path of the same contraction (the LAPACK
path of src/Kernel/KernelImpl.cpp:142-208 with the reference's own Utils::reshape, compiled
from its sources into oracle/_ref, and OpenBLAS dgemm, one C block per OpenMP thread) on a
bounded sample of the workload, on the host cores.

Multi-GPU: the contraction does not shard in this build ("replicas only"): with --gpus N
every rank runs the same workload on its own GPU, timing is the max over ranks and `value`
the sum of the ranks' work over that time.
"""
from __future__ import annotations

import argparse
import json
import os
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "block-sparse contract GFLOP/s (FP64-accurate)"
WORKLOADS = {
    "c0": "C[i,j,k]=sum_l A[i,j,l]*B[l,k]; 20 blocks per mode of U{5..15}; occ 0.3; U[-1,1] values",
    "c1": "C[i,j,a,b]=sum_P A[i,a,P]*B[j,b,P]; i,j=64 in {5,9,13}; a,b=512 in {13,25,32}; P=2048 in {32,48,64}; occ 15%",
    "c2": "c1 shapes with per-block magnitudes 10^U(-6,2)",
    "c3": ("C[a,b,i,j]=sum_cd V[a,b,c,d]*T[c,d,i,j]; a..d extent 96 in blocks of 24-48, i,j 12 in 8-16 "
           "(the configuration's extents x 1/8); V block kept iff exp(-0.5 spread) >= 0.1; product screening 1e-10"),
}
FORM_KERNEL = {"plain": "k_tiles", "batched": "k_tiles", "split": "k_slice + k_split"}


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--workload", default="c1", choices=sorted(WORKLOADS), help="the headline workload")
    ap.add_argument("--forms", default="plain,batched,split")
    ap.add_argument("--split-tol", type=float, default=1e-12,
                    help="relative Frobenius error vs the FP64 oracle below which the split form counts as FP64-accurate")
    ap.add_argument("--scale", type=float, default=1.0, help="extent scale of the c0-c2 workloads (1.0 = full size)")
    ap.add_argument("--seed", type=int, default=1)
    ap.add_argument("--cpu-sample-seconds", type=float, default=15.0)
    ap.add_argument("--cpu-runs", type=int, default=5, help="runs per CPU leg (the median is reported)")
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--no-count", action="store_true", help="skip the CUPTI launch count (use under ncu)")
    ap.add_argument("--no-autotune", action="store_true")
    ap.add_argument("--no-oracle", action="store_true", help="skip the oracle checks (use under ncu)")
    ap.add_argument("--no-configs", action="store_true", help="skip the other configurations")
    ap.add_argument("--pool-gb", type=float, default=60.0)
    ap.add_argument("--no-serving", action="store_true", help="skip the serving-loop phase")
    ap.add_argument("--serve-rate", type=float, default=200.0, help="Poisson arrival rate (requests/s)")
    ap.add_argument("--serve-seconds", type=float, default=2.0, help="length of the arrival stream")
    ap.add_argument("--serve-templates", type=int, default=16,
                    help="distinct requests (resident inputs) the stream draws from")
    ap.add_argument("--serve-seeds", type=int, default=3, help="Poisson streams (seeds) of the serving phase")
    return ap.parse_args()


# ------------------------------------------------------------------------------ helpers
class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled while the timed region runs."""

    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device: int):
        self.device = device
        self.rows = []
        self._stop = threading.Event()
        self._t = None

    def _run(self):
        while not self._stop.is_set():
            try:
                out = subprocess.run(["nvidia-smi", "-i", str(self.device), f"--query-gpu={self.Q}",
                                      "--format=csv,noheader,nounits"], capture_output=True, text=True, timeout=5)
                for line in out.stdout.strip().splitlines():
                    self.rows.append([x.strip() for x in line.split(",")])
            except Exception:
                pass
            self._stop.wait(0.2)

    def __enter__(self):
        self._t = threading.Thread(target=self._run, daemon=True)
        self._t.start()
        return self

    def __exit__(self, *exc):
        self._stop.set()
        self._t.join(timeout=10)

    def summary(self):
        if not self.rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"], "samples": 0}
        sm = [float(r[1]) for r in self.rows if r[1].replace(".", "").isdigit()]
        mx = [float(r[2]) for r in self.rows if r[2].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[i] for r in self.rows for i in range(4) if len(r) > 5 + i and r[5 + i] == "Active"})
        return {"sm_mhz": float(np.median(sm)) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": reasons, "samples": len(self.rows)}


def dist_env():
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return rank, world, local


def reduce_max(x: float) -> float:
    """Max of x over the ranks of the default process group (1 rank: x itself)."""
    import torch
    import torch.distributed as dist
    if not dist.is_available() or not dist.is_initialized() or dist.get_world_size() == 1:
        return x
    dev = "cuda" if dist.get_backend() == "nccl" else "cpu"
    t = torch.tensor([x], dtype=torch.float64, device=dev)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def replica_rate(work_per_rank: float, ms_per_rank: float, world: int) -> float:
    """Whole-job rate of `world` independent replicas timed by their slowest rank (work/ms → work/s/1e6)."""
    return world * work_per_rank / reduce_max(ms_per_rank) / 1e6


def build_workload(name: str, seed: int = 1, scale: float = 1.0):
    from shtensor_b200 import workloads as W
    if name == "c0":
        return W.c0(seed=seed)
    if name == "c1":
        return W.c1(seed=seed, scale=scale)
    if name == "c2":
        return W.c2(seed=seed, scale=scale)
    return W.c3(seed=seed)


def host(t):
    import oracle
    return oracle.HostTensor(t.block_sizes, t.ids, t.offsets, t.data)


def pair_flops_per_a_block(w) -> np.ndarray:
    """Algorithmic flops of each A block's pairs (no screening): 2 m_a k_a times the summed n
    of the B blocks that share its contracted block indices."""
    import oracle
    mp = oracle.contract_info(w.expr, [1] * w.A.order, [1] * w.B.order, [1] * len(w.C.block_sizes))
    ia, ib = w.A.index_lists(), w.B.index_lists()
    da, db = w.A.block_dims(), w.B.block_dims()
    ka = [tuple(int(ia[d][x]) for d in mp.colA) for x in range(len(w.A.ids))]
    kb = [tuple(int(ib[d][x]) for d in mp.rowB) for x in range(len(w.B.ids))]
    nb = db[:, mp.colB].prod(axis=1) if len(mp.colB) else np.ones(len(w.B.ids))
    nsum: dict = {}
    for key, n in zip(kb, nb):
        nsum[key] = nsum.get(key, 0) + int(n)
    m = da[:, mp.rowA].prod(axis=1).astype(np.float64)
    k = da[:, mp.colA].prod(axis=1).astype(np.float64)
    return np.array([2.0 * m[x] * k[x] * nsum.get(ka[x], 0) for x in range(len(w.A.ids))])


def sample_workload(w, target_flops: float):
    """The same contraction with A restricted to its first stored blocks, as many as make the
    sample's pair flops reach about target (a bounded CPU sample)."""
    from shtensor_b200 import workloads as W
    fl = np.cumsum(pair_flops_per_a_block(w))
    n = len(w.A.ids)
    k = int(min(n, max(1, np.searchsorted(fl, target_flops) + 1)))
    sizes = w.A.block_dims().prod(axis=1)[:k]
    offs = np.concatenate([[0], np.cumsum(sizes)[:-1]]).astype(np.int64)
    data = w.A.data[:int(w.A.offsets[k - 1] + sizes[-1])].copy()
    A = W.HostBlockSparse(w.A.block_sizes, w.A.ids[:k], offs, data)
    return W.Workload(w.name, w.expr, A, w.B, w.C, screen_eps=w.screen_eps), k, n


def cpu_leg(w, seconds: float, nthreads: int, ref: bool, runs: int):
    """Median rate (GFLOP/s) of `runs` runs of the CPU contraction on a sample sized to take about
    `seconds` per run: ref=True is the reference's path (its own Utils::reshape + OpenBLAS dgemm
    per pair, compiled from its sources into oracle/_ref), ref=False the oracle's bit-exact
    XMM-order restatement.  OpenMP over C blocks with `nthreads` threads."""
    import oracle
    probe, k, n0 = sample_workload(w, (0.5e9 if ref else 0.15e9) * max(nthreads, 1))
    r = oracle.contract(probe.expr, 1.0, host(probe.A), host(probe.B), 0.0, host(probe.C), eps=probe.screen_eps,
                        nthreads=nthreads, ref=ref)
    rate = r.flops / max(r.seconds, 1e-6)
    samp, k, n0 = sample_workload(w, rate * seconds)
    vals, secs, flops, npairs = [], [], 0.0, 0
    for _ in range(max(runs, 1)):
        r = oracle.contract(samp.expr, 1.0, host(samp.A), host(samp.B), 0.0, host(samp.C), eps=samp.screen_eps,
                            nthreads=nthreads, ref=ref)
        vals.append(r.flops / r.seconds / 1e9)
        secs.append(r.seconds)
        flops, npairs = r.flops, len(r.pairs)
    what = ("the reference's Utils::reshape + OpenBLAS dgemm per pair (LAPACK path)" if ref
            else "the oracle's XMM-order restatement (bit-exact to the asmjit kernel's order)")
    return {"value": float(np.median(vals)), "unit": "GFLOP/s", "cores": nthreads, "runs": len(vals),
            "seconds_median": float(np.median(secs)), "kind": "reference" if ref else "port",
            "sample": (f"A restricted to its first {k} of {n0} stored blocks: {npairs} pairs, {flops / 1e9:.3f} GFLOP; "
                       f"{what}; OpenMP over C blocks, {nthreads} thread(s)")}


def count_launches(fn):
    """Kernels launched by fn(), counted from the CUDA activity trace (CUPTI via torch), and the
    device time per kernel name (microseconds summed over its launches)."""
    import torch
    try:
        from torch.profiler import ProfilerActivity, profile
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            fn()
            torch.cuda.synchronize()
        evs = [e for e in prof.events() if e.device_type.name == "CUDA" and "memcpy" not in e.name.lower()
               and "memset" not in e.name.lower()]
        per = {}
        for e in evs:
            key = e.name.split("(")[0].replace("void ", "")
            n, us = per.get(key, (0, 0.0))
            per[key] = (n + 1, us + float(e.time_range.elapsed_us()))
        kernels = {k: {"launches": n, "us": round(us, 1)} for k, (n, us) in sorted(per.items(), key=lambda x: -x[1][1])}
        return len(evs), kernels
    except Exception as ex:  # profiler unavailable
        return None, {"error": str(ex)}


def measure_peak(sht, ctx, which):
    try:
        return sht.measure_peak(ctx, which)
    except Exception:
        return None


def pcie_bandwidth():
    """Pinned host <-> device copy bandwidth (GB/s) over 1 GiB, best of 3 each way."""
    import torch
    n = 1 << 27
    d = torch.empty(n, dtype=torch.float64, device="cuda")
    h = torch.empty(n, dtype=torch.float64).pin_memory()
    out = {}
    for name, fn in (("h2d", lambda: d.copy_(h, non_blocking=True)), ("d2h", lambda: h.copy_(d, non_blocking=True))):
        best = 0.0
        for _ in range(3):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            fn()
            e1.record()
            torch.cuda.synchronize()
            best = max(best, n * 8 / (e0.elapsed_time(e1) * 1e-3) / 1e9)
        out[name] = best
    del d, h
    return out


def run_serving(args, sht, ctx, upload):
    """Serving phase: seeded Poisson streams of mixed contractions through sht.Server, in the
    batched FP64 form and in the split-precision form.

    Requests are drawn from `serve_templates` distinct contractions of the c0..c3 families
    (extents x U(0.25,1), occupancy U(0.05,0.4)), whose inputs stay resident; each request
    writes its own fresh C, released when it completes.  Per form: `serve_seeds` streams at
    `serve_rate` (p50/p99 per seed and over all), a burst of one stream submitted at once (the
    loop's capacity), and a bit-equality check of served results against the same requests run
    alone in that form.  Beside them: each request run alone on the plain path (synchronous
    sht_contract, no queueing)."""
    import torch

    from shtensor_b200 import workloads as W
    rng = np.random.default_rng(args.seed + 1000)
    t_gen = time.perf_counter()
    temps = [W.c4_request(rng) for _ in range(args.serve_templates)]
    gen_s = time.perf_counter() - t_gen
    ins = [(upload(w.A), upload(w.B)) for w in temps]
    n = max(1, int(round(args.serve_rate * args.serve_seconds)))

    def fresh_c(w):
        return upload(W.empty_tensor(w.C.block_sizes))

    def alone_times(mode):
        ms, fl = [], []
        for w, (A, B) in zip(temps, ins):
            ts = []
            for r in range(4):
                C = fresh_c(w)
                torch.cuda.synchronize()
                t0 = time.perf_counter()
                rep = sht.contract(ctx, w.expr, 1.0, A, B, 0.0, C, w.screen_eps, mode=mode)
                ctx.stream_sync()
                ts.append((time.perf_counter() - t0) * 1e3)
                del C
            ms.append(float(np.median(ts[1:])))
            fl.append(rep["flops"])
        return ms, fl

    def pct(v, q):
        v = np.sort(np.asarray(v))
        return float(v[min(len(v) - 1, max(0, int(np.ceil(q * len(v))) - 1))])

    alone_ms, tflops = alone_times(sht.Mode.PLAIN_FP64)
    alone_split_ms, _ = alone_times(sht.Mode.SPLIT)
    streams = []
    for k in range(max(1, args.serve_seeds)):
        r = np.random.default_rng(args.seed + 2000 + k)
        streams.append((r.integers(0, len(temps), n), np.cumsum(r.exponential(1.0 / args.serve_rate, n))))
    picks0, arr0 = streams[0]
    alone_stream = np.array([alone_ms[k] for k in picks0])
    stream_flops = float(sum(tflops[k] for k in picks0))
    out = {"rate_per_s": args.serve_rate, "requests_per_stream": n, "seeds": len(streams),
           "templates": [{"family": w.meta["family"], "u": round(w.meta["u"], 3),
                          "occupancy": round(w.meta["occupancy"], 3), "gflop": f / 1e9,
                          "alone_plain_ms": a, "alone_split_ms": b}
                         for w, f, a, b in zip(temps, tflops, alone_ms, alone_split_ms)],
           "template_gen_s": gen_s, "offered_gflops": stream_flops / float(arr0[-1]) / 1e9,
           "alone_plain": {"p50_ms": pct(alone_stream, 0.5), "p99_ms": pct(alone_stream, 0.99),
                           "gflops": stream_flops / (alone_stream.sum() / 1e3) / 1e9,
                           "busy_s": float(alone_stream.sum() / 1e3)}}

    def run_phase(srv, picks, arrivals, burst, keep=None):
        srv.reset_stats()
        pending, reps = {}, []
        t0 = time.perf_counter()
        i = 0
        while i < len(picks) or pending:
            now = time.perf_counter() - t0
            while i < len(picks) and (burst or arrivals[i] <= now):
                k = int(picks[i])
                w, (A, B) = temps[k], ins[k]
                C = fresh_c(w)
                pending[srv.submit(w.expr, 1.0, A, B, 0.0, C, w.screen_eps)] = (C, k, time.perf_counter() - t0)
                i += 1
            for rid in list(pending):
                if srv.poll(rid):
                    rep = srv.wait(rid, 300)
                    C, k, t_sub = pending.pop(rid)
                    rep.update(template=k, submit_s=round(t_sub, 4))
                    reps.append(rep)
                    if keep is not None and k not in keep and len(keep) < 6:
                        keep[k] = (C, rep["form"])
                    del C
            time.sleep(0.0002)
        st = srv.stats()
        return {"p50_ms": st["p50_ms"], "p99_ms": st["p99_ms"], "max_ms": st["max_ms"], "gflops": st["gflops"],
                "span_s": st["span_s"], "completed": st["completed"], "failed": st["failed"],
                "launches": st["batches"], "mean_batch": st["mean_batch"], "max_active": st["max_active_seen"],
                "deferrals": st["deferrals"],
                "mean_queue_ms": float(np.mean([r["queue_ms"] for r in reps])),
                "mean_plan_ms": float(np.mean([r["plan_ms"] for r in reps])),
                "mean_run_ms": float(np.mean([r["run_ms"] for r in reps])),
                "slowest": [{k: (round(v, 3) if isinstance(v, float) else v) for k, v in r.items()
                             if k in ("template", "submit_s", "queue_ms", "plan_ms", "run_ms", "gpu_ms",
                                      "latency_ms", "batch_size", "form")}
                            for r in sorted(reps, key=lambda r: -r["latency_ms"])[:4]]}, reps

    for fname, mode in (("batched", sht.Mode.BATCHED_FP64), ("split", sht.Mode.SPLIT)):
        keep = {}
        res = {}
        with sht.Server(ctx, mode=mode) as srv:
            for w, (A, B) in zip(temps, ins):  # warm-up: every template once
                C = fresh_c(w)
                srv.wait(srv.submit(w.expr, 1.0, A, B, 0.0, C, w.screen_eps), 300)
                del C
            per_seed, lat = [], []
            for k, (picks, arrivals) in enumerate(streams):
                ph, reps = run_phase(srv, picks, arrivals, False, keep if k == 0 else None)
                per_seed.append(ph)
                lat += [r["latency_ms"] for r in reps]
            res["streams"] = per_seed
            res["stream"] = {"p50_ms": pct(lat, 0.5), "p99_ms": pct(lat, 0.99), "max_ms": max(lat),
                             "mean_batch": float(np.mean([p["mean_batch"] for p in per_seed])),
                             "gflops": float(np.mean([p["gflops"] for p in per_seed])),
                             "requests": len(lat)}
            res["burst"], _ = run_phase(srv, picks0, arr0, True)
        # served results against the same requests run alone in the form that served them
        same = True
        for k, (Cs, form) in keep.items():
            w, (A, B) = temps[k], ins[k]
            Cr = fresh_c(w)
            sht.contract(ctx, w.expr, 1.0, A, B, 0.0, Cr, w.screen_eps,
                         mode=sht.Mode.SPLIT if form == int(sht.Mode.SPLIT) else sht.Mode.PLAIN_FP64)
            same = same and Cs.nnz == Cr.nnz and sht.bitdiff(Cs, Cr) == 0
            del Cr
        res["mix_equals_alone"] = {"checked": len(keep), "bit_equal_values": bool(same)}
        keep.clear()
        out[fname] = res
    busy = out["alone_plain"]["busy_s"] / float(arr0[-1])
    out["load_note"] = (f"offered load {out['offered_gflops']:.0f} GFLOP/s; run alone back to back the stream keeps "
                        f"the GPU busy {100 * busy:.0f}% of its span on the plain path, so most requests arrive "
                        "to an idle GPU and launch at once (batch 1); requests that arrive while a launch runs "
                        "join the next one")
    del ins
    return out


# ------------------------------------------------------------------------------ the printed line
def digits(x, n=6):
    """x with its floats at n significant digits."""
    if isinstance(x, float):
        return float(f"{x:.{n}g}")
    if isinstance(x, dict):
        return {k: digits(v, n) for k, v in x.items()}
    return [digits(v, n) for v in x] if isinstance(x, (list, tuple)) else x


def summary_line(full):
    """The full record with its long parts cut to their figures: a reader of the last few KB of the output
    gets the whole line."""
    def forms(fs):
        return {k: {"ms_per_step": f["ms_per_step"], "gflops": f["gflops"], "exec_ms": f.get("exec_ms"),
                    "frac": (f.get("roofline") or {}).get("frac"),
                    **{e: (f.get("error_vs_oracle") or {}).get(e) for e in ("rel_fro", "bits_differ")}}
                for k, f in fs.items()}

    def served(s):
        keep = ("p50_ms", "p99_ms", "gflops", "mean_batch", "mean_plan_ms", "completed", "failed")
        return {ph: {k: s[ph][k] for k in keep if k in s[ph]} for ph in ("stream", "burst") if ph in s}

    line = dict(full)
    line["forms"] = forms(full["forms"])
    line["configs"] = {k: forms(c["forms"]) for k, c in (full.get("configs") or {}).items()} or None
    if full.get("serving"):
        sv = full["serving"]
        line["serving"] = {"alone_plain_gflops": sv["alone_plain"]["gflops"],
                           **{k: served(sv[k]) for k in ("batched", "split") if k in sv}}
    if full.get("cpu_baseline"):
        line["cpu_baseline"] = {k: v for k, v in full["cpu_baseline"].items() if k != "legs"}
    if full.get("kernels_per_step"):
        line["kernels_per_step"] = {k: v["launches"] if isinstance(v, dict) else v
                                    for k, v in dict(full["kernels_per_step"]).items()}
    roof = {k: v for k, v in (full.get("roofline") or {}).items() if k != "traffic_source"}
    line["roofline"] = roof or None
    return digits(line)


# ------------------------------------------------------------------------------ device legs
FORMS = {"plain": 0, "batched": 1, "split": 2}


def form_mode(sht, fname):
    return {"plain": sht.Mode.PLAIN_FP64, "batched": sht.Mode.BATCHED_FP64, "split": sht.Mode.SPLIT}[fname]


def time_contract(sht, ctx, w, A, B, C, mode, steps, warmup, stream, barrier, max_over_ranks):
    """Full contractions (plan + execute) back to back: device ms per step (max over ranks)."""
    import torch
    rep = None
    for _ in range(warmup):
        rep = sht.contract(ctx, w.expr, 1.0, A, B, 0.0, C, w.screen_eps, mode=mode, stream=stream)
    torch.cuda.synchronize()
    barrier()
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for _ in range(steps):
        rep = sht.contract(ctx, w.expr, 1.0, A, B, 0.0, C, w.screen_eps, mode=mode, stream=stream)
    e1.record(stream)
    torch.cuda.synchronize()
    barrier()
    ctx.stream_sync(stream)  # raises if a split launch recorded a failure
    return max_over_ranks(e0.elapsed_time(e1)) / steps, rep


def time_execute(sht, ctx, w, A, B, C, mode, steps, stream):
    """Execute-only (plan reused): mean device ms per execute, directly and by graph replay."""
    import torch
    plan = sht.Plan(ctx, w.expr, A, B, C, w.screen_eps, mode=mode, stream=stream)
    out = {}
    for graph in (False, True):
        for _ in range(3):
            plan.execute(1.0, 0.0, stream=stream, graph=graph)
        ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(steps)]
        for a, b in ev:
            a.record(stream)
            plan.execute(1.0, 0.0, stream=stream, graph=graph)
            b.record(stream)
        torch.cuda.synchronize()
        out["exec_graph_ms" if graph else "exec_ms"] = float(np.mean([a.elapsed_time(b) for a, b in ev]))
    ctx.stream_sync(stream)
    rep = plan.report()
    plan.close()
    return out, rep


def oracle_parity(sht, ctx, w, A, B, forms, T, stream, slices_sweep=()):
    """Every form on the whole workload against the CPU oracle (the XMM-order restatement, all
    host cores): pattern and pair list compared exactly, values by bit count and by max abs /
    relative Frobenius error on the device.  slices_sweep: split slice counts whose error is
    also measured."""
    import oracle
    t0 = time.perf_counter()
    want = oracle.contract(w.expr, 1.0, host(w.A), host(w.B), 0.0, host(w.C), eps=w.screen_eps)
    oracle_s = time.perf_counter() - t0
    from shtensor_b200 import workloads as W
    Cor = T(W.HostBlockSparse(w.C.block_sizes, want.C.ids, want.C.offsets, want.C.data))
    nnz = int(want.C.data.size)
    del want.C.data
    out = {}

    def one(mode):
        C = T(w.C)
        plan = sht.Plan(ctx, w.expr, A, B, C, w.screen_eps, mode=mode, stream=stream)
        plan.execute(1.0, 0.0, stream=stream)
        ctx.stream_sync(stream)
        pairs = plan.pairs()
        plan.close()
        ids, offs, _ = C.get_sparse_info()
        res = {"pattern_equal": bool(np.array_equal(ids, want.C.ids) and np.array_equal(offs, want.C.offsets)),
               "pairs_equal": bool(np.array_equal(pairs, want.pairs))}
        if res["pattern_equal"]:
            mx, fro = sht.compare(C, Cor, stream=stream)
            res.update(max_abs=mx, rel_fro=fro, bits_differ=sht.bitdiff(C, Cor, stream=stream))
        del C
        return res

    for f in forms:
        out[f] = one(form_mode(sht, f))
    sweep = {}
    for S in slices_sweep:
        ctx.set_split_slices(S)
        try:
            r = one(sht.Mode.SPLIT)
            sweep[str(S)] = {"rel_fro": r.get("rel_fro"), "max_abs": r.get("max_abs")}
        finally:
            ctx.set_split_slices(7)
    del Cor
    return out, sweep, {"seconds": oracle_s, "pairs": int(len(want.pairs)), "c_nnz": nnz,
                        "kind": "oracle XMM-order restatement, OpenMP over C blocks"}


def roofline_of(fname, flops, kern_ms, peaks, S=7):
    """Achieved rate of the form's kernels against the measured peak of the pipe that bounds it."""
    tf = flops / kern_ms / 1e9  # TFLOP/s (FP64-equivalent)
    if fname == "split":
        ach = flops * S * (S + 1) / 2 / kern_ms / 1e9
        pk = peaks.get("int8")
        return {"bound": "tensor", "pipe": f"int8 (tcgen05 kind::i8, {S} slices) with FP64 reassembly",
                "achieved": ach, "peak": pk, "unit": "TOPS", "frac": ach / pk if pk else None,
                "fp64_equivalent": {"achieved": tf, "peak": peaks.get("dmma"), "unit": "TFLOP/s",
                                    "frac": tf / peaks["dmma"] if peaks.get("dmma") else None,
                                    "peak_source": "FP64 tensor-core (mma.sync m8n8k4) probe, this run"},
                "operand_pipeline": {"achieved": ach, "peak": peaks.get("split_pipe"), "unit": "TOPS",
                                     "frac": ach / peaks["split_pipe"] if peaks.get("split_pipe") else None,
                                     "peak_source": "the split kernel's stage copies (from L2) and 7-slice MMA "
                                                    "triangle alone, no epilogue (sht_measure_peak 3), this run"}}
    pk = peaks.get("dmma")
    return {"bound": "tensor", "pipe": "fp64 tensor core (mma.sync m8n8k4)", "achieved": tf, "peak": pk,
            "unit": "TFLOP/s", "frac": tf / pk if pk else None}


def workload_leg(sht, ctx, w, forms, steps, warmup, stream, T, barrier, max_over_ranks, world, peaks,
                 check=True, tol=1e-12, sweep=(), autotune=False, clocks=None):
    """Time every form on one workload (full contraction and execute-only), check each against
    the oracle and give its roofline.  clocks: a dict that receives the clock samples taken
    while the forms were timed."""
    import torch
    A, B, C = T(w.A), T(w.B), T(w.C)
    res = {}
    flops = None
    cs = ClockSampler(torch.cuda.current_device()) if clocks is not None else None
    if cs:
        cs.__enter__()
    for fname in forms:
        mode = form_mode(sht, fname)
        if fname == "batched" and autotune:
            tuner = sht.Plan(ctx, w.expr, A, B, C, w.screen_eps, mode=mode, stream=stream)
            tuner.autotune(stream=stream)
            tuner.close()
        ms, rep = time_contract(sht, ctx, w, A, B, C, mode, steps, warmup, stream, barrier, max_over_ranks)
        flops = rep["flops"]
        ex, prep = time_execute(sht, ctx, w, A, B, C, mode, steps, stream)
        r = {"ms_per_step": ms, "gflops": world * flops / ms / 1e6, "plan_ms": rep["plan_ms"],
             "npairs": rep["npairs"], "tiles": rep["nwork"], **ex,
             "exec_gflops": flops / ex["exec_ms"] / 1e6, "kernel": FORM_KERNEL[fname]}
        r["roofline"] = roofline_of(fname, prep["flops"], ex["exec_ms"], peaks, prep.get("slices") or 7)
        res[fname] = r
    if cs:
        cs.__exit__(None, None, None)
        clocks.update(cs.summary())
    sweep_out, oinfo = {}, None
    if check:
        par, sweep_out, oinfo = oracle_parity(sht, ctx, w, A, B, list(res), T, stream, sweep)
        for f, v in par.items():
            res[f]["error_vs_oracle"] = v
            exact = v["pattern_equal"] and v["pairs_equal"]
            res[f]["fp64_accurate"] = bool(exact and v.get("rel_fro", 1.0) <= tol) if f == "split" else \
                bool(exact and v.get("bits_differ", 1) == 0)
    del A, B, C
    return res, flops, sweep_out, oinfo


# ------------------------------------------------------------------------------ arms
def run_reference(args):
    rank, world, _ = dist_env()
    if rank != 0:
        return
    import oracle
    ref = oracle.ref_lib() is not None  # without the reference's sources: the restatement, as "port"
    nthreads = os.cpu_count() or 1
    w = build_workload(args.workload, args.seed, args.scale)
    vals = []
    leg = None
    for _ in range(args.warmup):
        cpu_leg(w, max(args.cpu_sample_seconds / 5, 1.0), nthreads, ref, 1)
    for _ in range(args.steps):
        leg = cpu_leg(w, args.cpu_sample_seconds / max(args.steps, 1), nthreads, ref, 1)
        vals.append(leg["value"])
    value = float(np.median(vals))
    line = {
        "impl": "reference", "metric": METRIC, "value": value, "unit": "GFLOP/s", "n_gpus": args.gpus,
        "steps": args.steps, "warmup": args.warmup, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f64", "data": "synthetic (seeded)",
        "config": {"workload": WORKLOADS[args.workload], "scale": args.scale, "seed": args.seed},
        "cpu_baseline": {"value": value, "unit": "GFLOP/s", "cores": nthreads, "kind": leg["kind"],
                         "sample": leg["sample"]},
        "e2e": {"value": value, "unit": "GFLOP/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


def run_ours(args):
    import torch

    import shtensor_b200 as sht

    rank, world, local = dist_env()
    if world > 1:
        import torch.distributed as dist
        torch.cuda.set_device(local)
        dist.init_process_group("nccl", timeout=__import__("datetime").timedelta(seconds=120))
    else:
        torch.cuda.set_device(0)
    dev = torch.cuda.current_device()
    ctx = sht.Context(int(args.pool_gb * (1 << 30)), device=dev)
    # a stream of the benchmark's own: graph replay needs a non-default stream
    stream = torch.cuda.Stream()

    def T(h):
        t = sht.Tensor(ctx, h.block_sizes)
        t.reserve(h.index_lists() if len(h.ids) else [[] for _ in h.block_sizes])
        if h.nnz:
            t.upload(h.data)
        return t

    def barrier():
        if world > 1:
            torch.distributed.barrier()

    forms = [f for f in args.forms.split(",") if f]
    peaks = {k: measure_peak(sht, ctx, k) for k in ("fp64", "dmma", "int8", "split_pipe")}
    w = build_workload(args.workload, args.seed, args.scale)
    check = not args.no_oracle and world == 1 and rank == 0

    # ---- headline workload: every form timed (clocks sampled meanwhile), checked against the oracle
    clocks = {}
    results, flops, sweep, oinfo = workload_leg(
        sht, ctx, w, forms, args.steps, args.warmup, stream, T, barrier, reduce_max, world, peaks, check=check,
        tol=args.split_tol, sweep=(5, 6) if "split" in forms else (), autotune=not args.no_autotune, clocks=clocks)
    eligible = [k for k in results if results[k].get("fp64_accurate", True)]
    best = max(eligible, key=lambda k: results[k]["gflops"])
    if "split" in results:
        sweep["7"] = {k: results["split"].get("error_vs_oracle", {}).get(k) for k in ("rel_fro", "max_abs")}
    ratios = {}
    if "split" in results and "batched" in results:
        ratios["split_over_batched"] = results["split"]["gflops"] / results["batched"]["gflops"]
        ratios["split_over_batched_exec"] = results["split"]["exec_gflops"] / results["batched"]["exec_gflops"]
    if "split" in results and "plain" in results:
        ratios["split_over_plain"] = results["split"]["gflops"] / results["plain"]["gflops"]
        ratios["split_over_plain_exec"] = results["split"]["exec_gflops"] / results["plain"]["exec_gflops"]

    # ---- the other configurations
    configs = {}
    if not args.no_configs and world == 1:
        for name in [n for n in ("c0", "c2", "c3") if n != args.workload]:
            wx = build_workload(name, args.seed, args.scale)
            fx = {"c0": forms, "c2": [f for f in forms if f in ("batched", "split")],
                  "c3": [f for f in forms if f in ("batched", "split")]}[name]
            rx, flx, swx, ox = workload_leg(sht, ctx, wx, fx, max(3, args.steps // 2), args.warmup, stream, T, barrier,
                                            reduce_max, world, peaks, check=check, tol=args.split_tol,
                                            sweep=(5, 6) if name in ("c2", "c3") and "split" in fx else ())
            if "split" in rx:
                swx["7"] = {k: rx["split"].get("error_vs_oracle", {}).get(k) for k in ("rel_fro", "max_abs")}
            configs[name] = {"workload": WORKLOADS[name], "gflop_per_step": flx / 1e9, "forms": rx,
                             "split_slices_error": swx or None, "oracle": ox}
            del wx

    A, B, Cd = T(w.A), T(w.B), T(w.C)
    sht.contract(ctx, w.expr, 1.0, A, B, 0.0, Cd, w.screen_eps, mode=form_mode(sht, best), stream=stream)
    ctx.stream_sync(stream)
    c_nnz = Cd.nnz
    # serving runs before the launch count (the CUPTI profiler it uses slows later launches),
    # the CPU baseline (its OpenMP threads) and the end-to-end copies
    serving = None
    if world == 1 and not args.no_serving:
        serving = run_serving(args, sht, ctx, T)
    launches, names = (None, []) if args.no_count else count_launches(
        lambda: sht.contract(ctx, w.expr, 1.0, A, B, 0.0, Cd, w.screen_eps, mode=form_mode(sht, best), stream=stream))
    kern = results[best]
    roofline = dict(kern["roofline"])
    traffic = None
    try:  # DRAM bytes per launch of the dominant kernel, from the committed ncu summary
        with open(os.path.join(ROOT, "profiles", "roofline_traffic.json")) as f:
            traffic = json.load(f).get(best, {}).get("traffic_bytes_per_launch")
    except (OSError, ValueError):
        traffic = None
    roofline.update({"traffic": traffic,
                     "traffic_source": "profiles/roofline_traffic.json (ncu capture of a smaller case of the same "
                                       "kernel, scaled to the full workload)",
                     "algorithmic_bytes": 8.0 * (c_nnz + w.A.nnz + w.B.nnz), "kernel_ms": kern["exec_ms"],
                     "kernel": FORM_KERNEL[best],
                     "peak_source": "measured in this run by the library's own probe kernels "
                                    "(tcgen05 kind::i8 / mma.sync m8n8k4 / DFMA chains)"})

    # end to end through the public API: host buffers in pinned memory, copies timed
    e2e = None
    if not args.no_e2e:
        bw = pcie_bandwidth()
        ha = torch.from_numpy(w.A.data).pin_memory()
        hb = torch.from_numpy(w.B.data).pin_memory()
        hc = torch.empty(Cd.nnz, dtype=torch.float64).pin_memory()
        torch.cuda.synchronize()
        barrier()
        t0 = time.perf_counter()
        ee0, ee1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        ee0.record(stream)
        nrep = max(2, min(args.steps, 4))
        for _ in range(nrep):
            A.upload(ha.numpy(), stream=stream)
            B.upload(hb.numpy(), stream=stream)
            sht.contract(ctx, w.expr, 1.0, A, B, 0.0, Cd, w.screen_eps, mode=form_mode(sht, best), stream=stream)
            Cd.download(hc.numpy(), stream=stream)
        ee1.record(stream)
        torch.cuda.synchronize()
        ms = reduce_max(ee0.elapsed_time(ee1)) / nrep
        h2d, d2h = int(ha.numel() * 8 + hb.numel() * 8), int(hc.numel() * 8)
        floor_ms = (h2d / bw["h2d"] + d2h / bw["d2h"]) / 1e6
        e2e = {"value": world * flops / ms / 1e6, "unit": "GFLOP/s", "h2d_bytes_per_step": h2d,
               "d2h_bytes_per_step": d2h, "ms_per_step": ms, "wall_ms_per_step": (time.perf_counter() - t0) * 1e3 / nrep,
               "copy_floor_ms": floor_ms, "pcie_gbs": bw,
               "note": "the copies alone (pinned, measured bandwidth) take copy_floor_ms per step"}
        del ha, hb, hc

    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu:
        ncores = os.cpu_count() or 1
        import oracle
        ref = oracle.ref_lib() is not None  # without the reference's sources: the restatement alone
        main_leg = "reference_openmp" if ref else "xmm_restatement_openmp"
        legs = {main_leg: cpu_leg(w, args.cpu_sample_seconds / args.cpu_runs, ncores, ref, args.cpu_runs)}
        if ref:
            legs["reference_1thread"] = cpu_leg(w, 2.0, 1, True, args.cpu_runs)
        legs["xmm_restatement_1thread"] = cpu_leg(w, 2.0, 1, False, args.cpu_runs)
        cpu = dict(legs[main_leg])
        cpu["legs"] = legs

    del A, B, Cd

    if rank == 0:
        r = results[best]
        line = {
            "metric": METRIC, "value": r["gflops"], "unit": "GFLOP/s", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": r["ms_per_step"], "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f64", "data": "synthetic (seeded)",
            "config": {"workload": WORKLOADS[args.workload], "name": args.workload, "form": best, "scale": args.scale,
                       "seed": args.seed, "npairs": r["npairs"], "gflop_per_step": flops / 1e9,
                       "l2": "inputs and output larger than L2 (C alone is GBs); no flush",
                       "c_nnz": c_nnz, "parallelism": f"replicas x{world}"},
            "forms": results, "ratios": ratios, "split_slices_error": sweep or None, "oracle": oinfo,
            "roofline": roofline, "peaks": peaks, "cpu_baseline": cpu, "e2e": e2e, "clocks": clocks,
            "gpu_launches": (launches * args.steps) if launches is not None else None,
            "gpu_launches_per_step": launches, "kernels_per_step": names or None,
            "configs": configs or None, "serving": serving,
        }
        print(json.dumps(line), file=sys.stderr, flush=True)
        print(json.dumps(summary_line(line)), flush=True)
    ctx.close()
    if world > 1:
        torch.distributed.destroy_process_group()


def main():
    args = parse()
    if args.impl == "reference":
        run_reference(args)
    else:
        run_ours(args)


if __name__ == "__main__":
    main()
