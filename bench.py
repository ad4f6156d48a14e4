#!/usr/bin/env python3
"""Benchmark of the GB300 Black-Scholes map (options/s and % HBM roofline).

Default workload (the headline): the plain map over 10,000,000 seeded options
(S~U[10,200], K=S*U[0.5,1.5], r~U[0.01,0.10], v~U[0.05,0.65], t~U[0.05,2],
calls/puts 50/50), FP32, NUM_RUNS = 100 passes per step -- one step is one
whole ROI of the reference benchmark (blackscholes.c:781-913).  The 280 MB
working set is larger than the 129 MB L2, but only 2.2x: cross-pass L2 hits
serve part of it (the line says so), so the same line carries nested
records measured in the same run:

* ``roofline_2p28`` -- the map over 2^28 options (7.5 GB, 55x the L2): the
  HBM-roofline fraction with nothing L2-resident;
* ``batch`` -- 4,096 books of log-uniform size in one persistent CUDA-graph
  launch per pass vs one plain launch per book per pass;
* ``serve`` -- an open-loop Poisson trace through the continuous-batching
  server vs one plain launch per request, with the throughput each sustains
  under p99 bounds of 0.5, 1 and 2 ms (medians of repeated traces);
* ``swaptions`` -- the swaptions application's HJM Monte Carlo, 128
  swaptions x 1,000,000 paths in one call, with the CPU oracle on a sample;
* ``precision`` -- 2^28 options with deep in/out-of-the-money tails, each
  arithmetic mode's error against the FP64 kernel per |d1| bucket;
* ``fp64`` -- the FP64 product mode (double storage) against the CPU FP64
  oracle; ``io`` -- the reference's file formats, parsed and written, against
  the reference's fscanf / fprintf loops.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
                    [--config map|batch|precision|serve|serve-blocks|io|fp64|prefix-sweep|swaptions]
                    [--records FILE]

One JSON line on stdout (rank 0), with the figures of each nested record;
--records FILE keeps the records whole.  Under torchrun each rank prices its own
book on its own GPU (weak scaling, no collective on the data path); the
nested records are measured at one GPU only.
"""
from __future__ import annotations

import argparse
import json
import os
import subprocess
import sys
import tempfile
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

N_OPTIONS = 10_000_000
N_2P28 = 1 << 28
NUM_RUNS = 100
BYTES_PER_OPTION = 28  # 5 float inputs + int32 otype + float price
METRIC = "options/sec & %HBM roofline"
UNIT = "options/s"
SEED = 20241203
L2_FALLBACK = 126.5e6  # bytes, when the device does not report its L2


# ------------------------------------------------------------------ ranks
def dist_env():
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return rank, world, local


def shard_range(n: int, rank: int, world: int):
    """Contiguous (offset, len) of rank's share of n independent options
    (the same rule as the reference's static partition)."""
    q, r = divmod(n, world)
    off = rank * q + min(rank, r)
    return off, q + (1 if rank < r else 0)


def init_group(world: int, backend: str):
    if world <= 1:
        return None
    import torch.distributed as dist
    dist.init_process_group(backend=backend)
    return dist


def barrier(dist, device=None):
    if dist is not None:
        if device is not None:
            dist.barrier(device_ids=[device])
        else:
            dist.barrier()


def reduce_max(dist, x: float, device=None) -> float:
    """Max over ranks (timing only; the data path has no collective)."""
    if dist is None:
        return x
    import torch
    t = torch.tensor([x], dtype=torch.float64,
                     device=f"cuda:{device}" if device is not None else "cpu")
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


# ----------------------------------------------------------------- clocks
CLOCK_QUERY = ("timestamp,index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
               "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
               "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")


class ClockSampler:
    """nvidia-smi samples every 50 ms around the timed region; the summary
    keeps the samples whose timestamps fall inside it (all samples, with
    window_samples = 0, if the region was shorter than the sampling gap)."""

    def __init__(self, device: int):
        self.device = device
        self.proc = None
        self.path = None

    def __enter__(self):
        fd, self.path = tempfile.mkstemp(suffix=".csv")
        os.close(fd)
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.device), f"--query-gpu={CLOCK_QUERY}",
                 "--format=csv,noheader,nounits", "-lms", "50"],
                stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
            time.sleep(0.3)
        except OSError:
            self.proc = None
        self.t0 = time.time()
        return self

    def __exit__(self, *exc):
        self.t1 = time.time()
        if self.proc is not None:
            time.sleep(0.12)
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def summary(self):
        if not self.path or not os.path.exists(self.path):
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
        import datetime
        rows = []
        for line in open(self.path):
            f = [x.strip() for x in line.split(",")]
            if len(f) >= 10:
                try:
                    f[0] = datetime.datetime.strptime(f[0], "%Y/%m/%d %H:%M:%S.%f").timestamp()
                except ValueError:
                    continue
                rows.append(f[:1] + f[2:])  # drop the index column
        os.unlink(self.path)
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
        inside = [r for r in rows if self.t0 - 0.01 <= r[0] <= self.t1 + 0.01]
        use = inside if inside else rows
        sm = [float(r[1]) for r in use if r[1].replace(".", "").isdigit()]
        mx = [float(r[2]) for r in use if r[2].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[i] for r in use for i in range(4) if r[5 + i].lower() == "active"})
        return {"sm_mhz": float(np.median(sm)) if sm else None,
                "sm_max_mhz": max(mx) if mx else None, "reasons": reasons,
                "samples": len(use), "window_samples": len(inside),
                "window_s": round(self.t1 - self.t0, 4)}


def measured_hbm_peak():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            return float(json.load(f)["hbm_gbs"]), "measured"
    except (OSError, KeyError, ValueError):
        return 6800.0, "fallback"


# -------------------------------------------------------------- CPU baseline
PORT_NOTE = ("the oracle port of the reference's FastFlow map (blackscholes.c:315-348): the "
             "reference's FP32 arithmetic, FastFlow's static partition, a join per pass, on this "
             "host's cores, compiled as PARSEC compiles the reference (gcc.bldconf:74-75: -O3 "
             "-funroll-loops -fprefetch-loop-arrays, the compiler's default contraction, so on "
             "aarch64 with fused multiply-adds as a native build would); the reference's own "
             "build needs its source tree, which is not on this host")


def cpu_baseline(book, target_s: float = 10.0):
    """The oracle port of the reference's FastFlow map, built with PARSEC's
    flags, on every host core, over the same book, with as many passes as
    fit in ~target_s seconds."""
    import oracle
    threads = os.cpu_count() or 1
    _, t1 = oracle.bs_map(book, threads, 1, parsec_flags=True)
    runs = int(max(1, min(NUM_RUNS, target_s / max(t1, 1e-6))))
    _, secs = oracle.bs_map(book, threads, runs, parsec_flags=True)
    return {"value": len(book) * runs / secs, "unit": UNIT, "cores": threads, "kind": "port",
            "sample": f"{len(book)} options x {runs} passes (of {NUM_RUNS}) of the same book, "
                      f"static partition over {threads} threads, {secs:.2f} s",
            "note": PORT_NOTE}


def map_config(n: int, runs: int, world: int) -> dict:
    """The workload description both arms print for the map."""
    ws = BYTES_PER_OPTION * n
    return {"workload": f"plain map, {n} European options FP32 SoA, NUM_RUNS={runs} "
                        "passes per step", "options": n, "num_runs": runs,
            "parallelism": f"replicas x{world} (independent books)",
            "l2": (f"inputs ({ws / 1e6:.0f} MB) larger than L2 (129 MB); no flush"
                   if ws > 129e6 else
                   f"inputs ({ws / 1e6:.1f} MB) fit in L2 (129 MB): an L2-resident run, "
                   "not an HBM measurement"),
            "mode": "fast"}


def l2_bytes(device: int) -> float:
    import torch
    v = getattr(torch.cuda.get_device_properties(device), "L2_cache_size", 0)
    return float(v) if v else L2_FALLBACK


def prefix_bytes(tune: dict, n: int, l2: float) -> int:
    """Bytes of the book the resident-prefix load path keeps in L2 (the
    library's rule: resident_32nds of the L2, whole 8-option groups)."""
    if tune.get("load_path") != 7:
        return 0
    r32 = tune.get("resident_32nds") or 15
    groups = int(l2) * r32 // 32 // (BYTES_PER_OPTION * 8)
    return min(groups, n // 8) * 8 * BYTES_PER_OPTION


def time_steps(stream, step, steps, warmup, clocks_device=None):
    """warmup untimed steps, then `steps` timed with CUDA events on `stream`;
    returns (seconds, clock summary or None)."""
    import torch
    for _ in range(warmup):
        step()
    torch.cuda.synchronize()
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    clk = ClockSampler(clocks_device) if clocks_device is not None else None
    if clk:
        clk.__enter__()
    e0.record(stream)
    for _ in range(steps):
        step()
    e1.record(stream)
    e1.synchronize()
    if clk:
        clk.__exit__(None, None, None)
    return e0.elapsed_time(e1) / 1e3, (clk.summary() if clk else None)


# ------------------------------------------------------------------ our arm
def run_ours(args, rank, world, local):
    import torch

    from p3arsec_gb300 import Context, books
    from p3arsec_gb300 import build as b
    os.environ.setdefault("BSG_TUNE_CACHE", os.path.join(b.BUILD, "tune_cache.txt"))
    b.build()
    torch.cuda.set_device(local)
    dist = init_group(world, "nccl")
    n, runs = args.n, args.runs
    book = books.generate(n, seed=SEED + rank)
    ctx = Context(local, max_options=n if not args.no_e2e else 1)
    if args.tune:
        ctx.set_tune(*(int(x) for x in args.tune.split(",")))
        tune = ctx.get_tune()
    else:
        tune = ctx.autotune(n)
    dev = [torch.from_numpy(a).to(f"cuda:{local}") for a in book.arrays()]
    out = torch.empty(n, dtype=torch.float32, device=f"cuda:{local}")
    stream = torch.cuda.ExternalStream(ctx.stream, device=f"cuda:{local}")

    def step():
        ctx.price_soa(*dev, out, n=n, num_runs=runs, device=True, asynchronous=True)

    for _ in range(args.warmup):
        step()
    torch.cuda.synchronize()
    barrier(dist, local)
    torch.cuda.synchronize()
    l0 = ctx.launches
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    repeat_ms = []
    with ClockSampler(local) as clk:
        e0.record(stream)
        for _ in range(args.steps):
            step()
        e1.record(stream)
        e1.synchronize()
        launches = ctx.launches - l0
        # the same K steps timed again, to show the spread of the number
        # (and to give the clock sampler a longer window under load)
        for _ in range(args.repeats):
            r0 = torch.cuda.Event(enable_timing=True)
            r1 = torch.cuda.Event(enable_timing=True)
            r0.record(stream)
            for _ in range(args.steps):
                step()
            r1.record(stream)
            r1.synchronize()
            repeat_ms.append(r0.elapsed_time(r1))
    torch.cuda.synchronize()
    ms = e0.elapsed_time(e1)
    barrier(dist, local)
    ms_max = reduce_max(dist, ms, local)
    secs = ms_max / 1e3
    value = world * n * runs * args.steps / secs
    per_launch_s = secs / (runs * args.steps)
    achieved = BYTES_PER_OPTION * n / per_launch_s / 1e9
    peak, peak_src = measured_hbm_peak()
    l2 = l2_bytes(local)

    # accuracy of the timed output against the FP64 oracle kernel
    accuracy = None
    if not args.no_accuracy:
        edges = np.array([0.0, 0.5, 1.0, 2.0, 3.0, 4.0, 6.0, np.inf])
        rep = ctx.error_report(dev, out, n, edges)
        accuracy = {"max_abs_vs_fp64": max(x["max_abs"] for x in rep),
                    "rms_abs_vs_fp64": (sum(x["sum_sq_abs"] for x in rep) / n) ** 0.5,
                    "gate": 1e-4}

    # end to end through the public API with pinned host buffers
    e2e = None
    if not args.no_e2e:
        host = [torch.from_numpy(a).pin_memory().numpy() for a in book.arrays()]
        hout = torch.empty(n, dtype=torch.float32).pin_memory().numpy()
        # synchronous calls: each step's copies in series with its passes
        ctx.price_soa(*host, hout, n=n, num_runs=runs)  # warm (graph for the resident buffers)
        barrier(dist, local)
        t0 = time.perf_counter()
        for _ in range(args.steps):
            ctx.price_soa(*host, hout, n=n, num_runs=runs)
        sync_s = reduce_max(dist, time.perf_counter() - t0, local)
        # pipelined calls (BSG_ASYNC with host pointers): step k + 1's inputs
        # cross the host link while step k's passes run; every step still
        # copies its 240 MB in and 40 MB out inside the timed region
        for _ in range(2):  # warm both resident sets
            ctx.price_soa(*host, hout, n=n, num_runs=runs, asynchronous=True)
        ctx.synchronize()
        barrier(dist, local)
        t0 = time.perf_counter()
        for _ in range(args.steps):
            ctx.price_soa(*host, hout, n=n, num_runs=runs, asynchronous=True)
        ctx.synchronize()
        e2e_s = reduce_max(dist, time.perf_counter() - t0, local)
        e2e = {"value": world * n * runs * args.steps / e2e_s, "unit": UNIT,
               "h2d_bytes_per_step": 24 * n, "d2h_bytes_per_step": 4 * n,
               "ms_per_step": 1e3 * e2e_s / args.steps,
               "mode": "pipelined bsg_price_soa(BSG_ASYNC, pinned host arrays) + bsg_synchronize",
               "synchronous": {"value": world * n * runs * args.steps / sync_s,
                               "ms_per_step": 1e3 * sync_s / args.steps}}

    ws = BYTES_PER_OPTION * n
    pb = prefix_bytes(tune, n, l2)
    line = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms_max / args.steps,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
        "data": "synthetic (seeded book, reference config distributions)",
        "config": map_config(n, runs, world),
        "tune": tune,
        "roofline": {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s",
                     "frac": achieved / peak, "peak_source": peak_src,
                     "traffic": None,
                     "traffic_note": "DRAM bytes per pass are measured with ncu (serialised "
                                     "launches), not in this run; they are summarised with "
                                     "the kernel's profile",
                     "bytes_per_launch": ws, "avg_launch_us": per_launch_s * 1e6,
                     "l2_assisted": bool(ws < 4 * l2),
                     "l2_bytes": int(l2), "prefix_bytes": pb,
                     "note": ("achieved counts the algorithmic 28 B/option; the book is "
                              f"{ws / l2:.1f}x the L2, so lines kept in L2 from pass to pass "
                              "(the resident prefix and the evict-first slice) serve part of "
                              "each pass and frac can exceed 1; roofline_2p28 is the fraction "
                              "with nothing L2-resident")
                     if ws < 4 * l2 else "the book is far larger than the L2"},
        "accuracy": accuracy,
        "e2e": e2e,
        "gpu_launches": launches,
        "clocks": clk.summary(),
    }
    if repeat_ms:
        vals = [world * n * runs * args.steps / (m / 1e3) for m in repeat_ms]
        line["repeats"] = {"values": vals, "note": f"{len(vals)} more timed windows of the same "
                                                   f"{args.steps} steps, right after the first",
                           "spread": (max(vals + [value]) - min(vals + [value])) /
                                     float(np.median(vals + [value]))}
    ctx.close()
    del dev, out
    torch.cuda.empty_cache()
    if world == 1 and not args.no_nested:
        line["roofline_2p28"] = _nested(map_2p28_record, args, local, peak, peak_src)
        line["batch"] = _nested(batch_record, args, local, steps=3, warmup=3)
        line["serve"] = _nested(serve_record, args, local)
        line["swaptions"] = _nested(swaptions_record, args, local, steps=3, warmup=3,
                                    sample=20_000)
        line["precision"] = _nested(precision_record, args, local, n=N_2P28, runs=10, steps=1,
                                    warmup=3)
        line["fp64"] = _nested(fp64_record, args, local, n=1 << 22, runs=10, steps=3, warmup=3)
        line["io"] = _nested(io_record, args, n=1 << 20)
        torch.cuda.empty_cache()
    if rank == 0 and world == 1 and not args.no_cpu:
        line["cpu_baseline"] = cpu_baseline(book)
    if rank == 0:
        if args.records:
            with open(args.records, "w") as f:
                json.dump(line, f, indent=1)
        print(printed_line(line), flush=True)
    if dist is not None:
        dist.destroy_process_group()


LINE_LIMIT = 2800  # characters: a reader that keeps a log's last 3,000 gets all of the line


def _short(record, *keys):
    """A nested record's figures under these keys ("a.b": of its part a), or its error."""
    out = {}
    for key in ("error",) + keys:
        x = record
        for part in key.split("."):
            x = x.get(part) if isinstance(x, dict) else None
        if x is not None:
            out[key.replace("modes.", "").replace(".", "_")] = x
    return out


def _rounded(x):
    if isinstance(x, float):
        return float(f"{x:.6g}")
    if isinstance(x, dict):
        return {k: _rounded(v) for k, v in x.items()}
    return [_rounded(v) for v in x] if isinstance(x, list) else x


def printed_line(line, limit=LINE_LIMIT):
    """The map's JSON line as it is printed: the headline whole but for its prose,
    of each nested record the figures it is read for (--records FILE keeps
    everything).  Nested records, the last first, give way to the limit."""
    line = dict(line)
    for key, what in (("roofline", ("traffic_note", "note")), ("cpu_baseline", ("note",)), ("repeats", ("values", "note"))):
        if line.get(key):
            line[key] = {k: v for k, v in line[key].items() if k not in what}
    pick = {
        "roofline_2p28": ("value", "frac", "max_abs_vs_fp64", "gpu_launches"),
        "batch": ("value", "roofline.frac", "speedup_vs_plain", "bit_identical", "gpu_launches"),
        "serve": ("trace.batched.p99_ms", "trace.batched.options_per_s", "trace.plain.options_per_s"),
        "swaptions": ("value", "ms_per_step", "vs_oracle.max_rel_price_diff", "cpu_baseline.value", "gpu_launches"),
        "precision": ("modes.fast.max_abs", "modes.fast.rms_abs", "modes.fast.options_per_s",
                      "modes.libm_ref.max_abs", "modes.libm_ref.options_per_s"),
        "fp64": ("value", "max_diff_over_max_s_k", "max_rel_above_1e-6_of_max_s_k", "max_rel_vs_cpu_fp64"),
        "io": ("parse.speedup", "write.speedup", "parse.bit_identical", "write.byte_identical"),
    }
    nested = [k for k in pick if k in line]
    for key in nested:
        full = line[key]
        line[key] = _short(full, *pick[key])
        if key == "serve" and "throughput_at_equal_p99" in full:
            line[key]["equal_p99"] = [[e["p99_bound_ms"], e["batched_options_per_s"], e["plain_options_per_s"],
                                       e["ratio"]] for e in full["throughput_at_equal_p99"]]
    keep = {k: line[k] for k in ("value", "ms_per_step")}
    dump = lambda: json.dumps({**_rounded(line), **keep}, separators=(",", ":"))  # noqa: E731
    text = dump()
    while len(text) > limit and nested:
        line[nested[-1]] = "in --records"
        nested.pop()
        text = dump()
    return text


def _nested(fn, *a, **kw):
    """A nested record, or the error that stopped it (the headline stands)."""
    try:
        return fn(*a, **kw)
    except Exception as ex:  # noqa: BLE001 -- reported in the JSON line
        import traceback
        traceback.print_exc(file=sys.stderr)
        return {"error": f"{type(ex).__name__}: {ex}"}


def map_2p28_record(args, local, peak, peak_src, n=N_2P28, steps=3, warmup=3):
    """The fast map over 2^28 options (7.5 GB: nothing of the book can stay
    in L2 between passes), NUM_RUNS passes per step, autotuned at that
    size: the HBM-roofline fraction of the map."""
    import torch

    from p3arsec_gb300 import Context, books
    ctx = Context(local, max_options=1)
    tune = ctx.autotune(n)
    dev = books.generate_device(n, SEED + 28, device=f"cuda:{local}")
    out = torch.empty(n, dtype=torch.float32, device=f"cuda:{local}")
    stream = torch.cuda.ExternalStream(ctx.stream, device=f"cuda:{local}")
    runs = args.runs

    def step():
        ctx.price_soa(*dev, out, n=n, num_runs=runs, device=True, asynchronous=True)

    for _ in range(warmup):
        step()
    torch.cuda.synchronize()
    l0 = ctx.launches
    secs, clk = time_steps(stream, step, steps, 0, clocks_device=local)
    launches = ctx.launches - l0
    per_launch_s = secs / (runs * steps)
    achieved = BYTES_PER_OPTION * n / per_launch_s / 1e9
    edges = np.array([0.0, 0.5, 1.0, 2.0, 3.0, 4.0, 6.0, np.inf])
    rep = ctx.error_report(dev, out, n, edges)
    l2 = l2_bytes(local)
    rec = {"workload": f"plain map, {n} options FP32 SoA ({BYTES_PER_OPTION * n / 1e9:.2f} GB, "
                       f"{BYTES_PER_OPTION * n / l2:.0f}x the L2), NUM_RUNS={runs} passes per step, "
                       "plain distribution drawn on the GPU",
           "options": n, "num_runs": runs, "steps": steps, "warmup": warmup,
           "value": n * runs * steps / secs, "unit": UNIT, "ms_per_step": 1e3 * secs / steps,
           "tune": tune, "prefix_bytes": prefix_bytes(tune, n, l2),
           "bound": "hbm", "achieved": achieved, "peak": peak, "peak_source": peak_src,
           "unit_bw": "GB/s", "frac": achieved / peak, "avg_launch_us": per_launch_s * 1e6,
           "bytes_per_launch": BYTES_PER_OPTION * n, "gpu_launches": launches,
           "max_abs_vs_fp64": max(x["max_abs"] for x in rep),
           "clocks": clk}
    ctx.close()
    del dev, out
    torch.cuda.empty_cache()
    return rec


# ------------------------------------------------------------ batched books
def book_sizes(nbooks: int, seed: int, lo: int = 1, hi: int = 1 << 20):
    """Book sizes log-uniform in [lo, hi] (seeded)."""
    rng = np.random.default_rng(seed)
    return np.floor(np.exp(rng.uniform(np.log(lo), np.log(hi + 1), nbooks))).astype(np.int64).clip(lo, hi)


def batch_record(args, local, steps=None, warmup=None, nbooks=None, seed=SEED + 4):
    """Config 4: many uneven books in one pool, one persistent CUDA-graph
    launch per pass vs one plain launch per book per pass (both NUM_RUNS
    passes per step, the same device pool, outputs compared bit for bit)."""
    import torch

    from p3arsec_gb300 import Context, books
    steps = args.steps if steps is None else steps
    warmup = args.warmup if warmup is None else warmup
    nbooks = args.books if nbooks is None else nbooks
    sizes = book_sizes(nbooks, seed)
    segs, off = [], 0
    for nb in sizes:
        segs.append((off, int(nb)))
        off += (int(nb) + 63) // 64 * 64  # books start 256-byte aligned
    pool_len = off
    total = int(sizes.sum())
    dev = books.generate_device(pool_len, seed + 1, device=f"cuda:{local}")
    out_b = torch.zeros(pool_len, dtype=torch.float32, device=f"cuda:{local}")
    out_p = torch.zeros(pool_len, dtype=torch.float32, device=f"cuda:{local}")
    ctx = Context(local, max_options=1)
    if args.tune:
        ctx.set_tune(*(int(x) for x in args.tune.split(",")))
    else:
        ctx.autotune(1 << 16)  # plain per-book launches are small
    stream = torch.cuda.ExternalStream(ctx.stream, device=f"cuda:{local}")
    runs = args.runs
    if args.batch_tune:
        tile, bps = (int(x) for x in args.batch_tune.split(","))
        ctx.set_batch_tune(tile, bps)
        batch_tune = ctx.get_batch_tune()
    else:
        batch_tune = ctx.autotune_batch(dev, out_b, pool_len, segs)

    def timed(fn):
        for _ in range(warmup):
            fn()
        torch.cuda.synchronize()
        l0 = ctx.launches
        secs, clk = time_steps(stream, fn, steps, 0, clocks_device=local)
        return secs, ctx.launches - l0, clk

    secs_b, launches_b, clk = timed(lambda: ctx.price_batch(dev, out_b, pool_len, segs,
                                                            num_runs=runs, asynchronous=True))
    secs_p, launches_p, _ = timed(lambda: ctx.price_batch(dev, out_p, pool_len, segs,
                                                          num_runs=runs, plain=True,
                                                          asynchronous=True))
    torch.cuda.synchronize()
    same = bool(torch.equal(out_b.view(torch.int32), out_p.view(torch.int32)))
    value = total * runs * steps / secs_b
    plain = total * runs * steps / secs_p
    peak, peak_src = measured_hbm_peak()
    achieved = BYTES_PER_OPTION * total * runs * steps / secs_b / 1e9
    rec = {
        "workload": f"{nbooks} books, sizes log-uniform in [1, 2^20] (seed {seed}), "
                    f"{total} options, {runs} passes per step",
        "books": nbooks, "options": total, "num_runs": runs, "seed": seed,
        "steps": steps, "warmup": warmup,
        "value": value, "unit": UNIT, "ms_per_step": 1e3 * secs_b / steps,
        "plain_per_book": {"value": plain, "unit": UNIT, "ms_per_step": 1e3 * secs_p / steps,
                           "gpu_launches": launches_p},
        "speedup_vs_plain": value / plain,
        "bit_identical": same,
        "tune_plain": ctx.get_tune(), "tune_batch": batch_tune,
        "roofline": {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s",
                     "frac": achieved / peak, "peak_source": peak_src},
        "gpu_launches": launches_b, "clocks": clk,
    }
    ctx.close()
    del dev, out_b, out_p
    torch.cuda.empty_cache()
    return rec


def run_batch(args, rank, world, local):
    """--config batch: the batched-books record as its own JSON line."""
    import torch

    from p3arsec_gb300 import build as b
    b.build()
    torch.cuda.set_device(local)
    rec = batch_record(args, local)
    line = {"metric": "options/sec (batched books, one persistent launch per pass)",
            "value": rec["value"], "unit": UNIT, "n_gpus": world, "steps": rec["steps"],
            "warmup": rec["warmup"], "ms_per_step": rec["ms_per_step"], "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic (seeded books)",
            "config": {"workload": rec["workload"], "books": rec["books"],
                       "options": rec["options"], "num_runs": rec["num_runs"]},
            **{k: rec[k] for k in ("plain_per_book", "speedup_vs_plain", "bit_identical",
                                   "tune_plain", "tune_batch", "roofline", "gpu_launches",
                                   "clocks")}}
    if rank == 0:
        print(json.dumps(line), flush=True)


# --------------------------------------------------------- precision sweep
def precision_record(args, local, n=None, runs=None, steps=None, warmup=None):
    """Config 3: options with deep in/out-of-the-money tails (K = S*U[0.05,20],
    t ~ U[0.001,5], drawn on the GPU); the compensated FP32 path, the
    reference-order SFU path and the reference-order accurate-libm path
    against the FP64 oracle kernel, per bucket of |d1|, with the throughput
    of each."""
    import torch

    from p3arsec_gb300 import Context, books
    n = args.n if n is None else n
    runs = args.runs if runs is None else runs
    steps = args.steps if steps is None else steps
    warmup = args.warmup if warmup is None else warmup
    dev = books.generate_device(n, SEED + 3, dist="tails", device=f"cuda:{local}")
    out = torch.empty(n, dtype=torch.float32, device=f"cuda:{local}")
    ctx = Context(local, max_options=1)
    if args.tune:
        ctx.set_tune(*(int(x) for x in args.tune.split(",")))
    else:
        ctx.autotune(n)
    stream = torch.cuda.ExternalStream(ctx.stream, device=f"cuda:{local}")
    edges = np.array([0.0, 0.5, 1.0, 2.0, 3.0, 4.0, 5.0, 6.0, 8.0, 12.0, np.inf])
    res = {}
    for mode in ("fast", "sfu_ref", "libm_ref"):
        def step():
            ctx.price_soa(*dev, out, n=n, num_runs=runs, mode=mode, device=True,
                          asynchronous=True)
        secs, _ = time_steps(stream, step, steps, warmup)
        rep = ctx.error_report(dev, out, n, edges, rel_floor=1e-3)
        res[mode] = {"options_per_s": n * runs * steps / secs,
                     "max_abs": max(x["max_abs"] for x in rep),
                     "rms_abs": (sum(x["sum_sq_abs"] for x in rep) / n) ** 0.5,
                     "buckets": [{"d1": [x["d1_lo"], x["d1_hi"]], "count": x["count"],
                                  "max_abs": x["max_abs"], "rms_abs": x["rms_abs"],
                                  "max_rel": x["max_rel"], "max_price": x["max_price"]}
                                 for x in rep]}
    ctx.close()
    del dev, out
    torch.cuda.empty_cache()
    return {"workload": f"precision sweep, {n} options, tails distribution (K=S*U[0.05,20], "
                        f"t~U[0.001,5], drawn on the GPU), {runs} passes per step",
            "options": n, "num_runs": runs, "steps": steps, "warmup": warmup,
            "rel_floor": 1e-3, "modes": res,
            "note": "prices reach ~3.8e3 here, where one FP32 ulp is 2.4e-4: no FP32 output "
                    "meets 1e-4 absolute in the top buckets; the 1e-4 gate is the plain "
                    "distribution's (the headline's accuracy record)"}


def run_precision(args, rank, world, local):
    """--config precision: the precision record as its own JSON line."""
    import torch

    from p3arsec_gb300 import build as b
    b.build()
    torch.cuda.set_device(local)
    rec = precision_record(args, local)
    line = {"metric": "precision sweep: max/RMS error vs FP64 per |d1| bucket",
            "value": rec["modes"]["fast"]["options_per_s"], "unit": UNIT, "n_gpus": world,
            "steps": rec["steps"], "warmup": rec["warmup"], "higher_is_better": True,
            "dtype": "f32", "data": "synthetic (seeded, K=S*U[0.05,20], t~U[0.001,5])",
            "config": {"workload": rec["workload"], "options": rec["options"],
                       "num_runs": rec["num_runs"], "rel_floor": 1e-3},
            "modes": rec["modes"]}
    if rank == 0:
        print(json.dumps(line), flush=True)


# ----------------------------------------------------------------- serving
def host_link_bandwidth(device: int):
    """Pinned host <-> device copy bandwidth (1 GiB, CUDA events)."""
    import torch
    n = 1 << 28
    h = torch.ones(n, dtype=torch.float32).pin_memory()
    d = torch.empty(n, dtype=torch.float32, device=f"cuda:{device}")
    res = {}
    for name, fn in (("h2d_GBps", lambda: d.copy_(h, non_blocking=True)),
                     ("d2h_GBps", lambda: h.copy_(d, non_blocking=True))):
        fn()
        torch.cuda.synchronize()
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(3):
            fn()
        e1.record()
        e1.synchronize()
        res[name] = 3 * 4 * n / (e0.elapsed_time(e1) / 1e3) / 1e9
    del h, d
    return res

SERVE_BOUNDS_MS = (0.5, 1.0, 2.0)


def serve_host_pool(local, pool_n=1 << 24):
    """A pinned host pool of pool_n options (drawn on the GPU, copied out)
    that the traces slice their requests from, and a pinned prices array."""
    import torch

    from p3arsec_gb300 import books
    dev = books.generate_device(pool_n, SEED + 6, device=f"cuda:{local}")
    host = [x.cpu().pin_memory().numpy() for x in dev]
    del dev
    out = torch.zeros(pool_n, dtype=torch.float32).pin_memory().numpy()
    return host, out


def serve_point(host, out, mode, rate, seconds, args, local, seed, sizes=None):
    from p3arsec_gb300 import abi
    lo_n, hi_n = sizes or (int(x) for x in args.serve_sizes.split(","))
    return abi.serve_trace(host, out, rate_per_s=rate, duration_s=seconds, min_n=lo_n,
                           max_n=hi_n, seed=seed, device=local, budget_bytes=64 << 30,
                           max_inflight=args.serve_inflight, plain=(mode == "plain"),
                           drain_timeout_s=60.0,
                           fused=(mode == "batched" and args.serve_fused >= 1),
                           persistent=(mode == "batched" and args.serve_fused == 2),
                           persistent_blocks=args.serve_blocks,
                           persistent_window=args.serve_window)


def equal_p99(sweep, bounds_ms, link_opts):
    """Throughput at equal p99: for each bound, each loop's best median
    throughput among the swept rates whose traces all completed with median
    p99 within the bound; their ratio, and the ceiling the host link puts on
    it (link options/s over the plain loop's figure).  A loop that meets a
    bound at no rate gets a note with its median p99 at the lowest rate, and
    the ratio is null."""
    def best(mode, bound_ms):
        ok = [p for p in sweep[mode] if p["all_completed"] and p["median_p99_ms"] <= bound_ms]
        return max(ok, key=lambda p: p["median_options_per_s"]) if ok else None

    equal = []
    for bound in bounds_ms:
        bb, pp = best("batched", bound), best("plain", bound)
        equal.append({
            "p99_bound_ms": bound,
            "batched_options_per_s": bb["median_options_per_s"] if bb else None,
            "batched_rate_per_s": bb["rate_per_s"] if bb else None,
            "plain_options_per_s": pp["median_options_per_s"] if pp else None,
            "plain_rate_per_s": pp["rate_per_s"] if pp else None,
            "ratio": (bb["median_options_per_s"] / pp["median_options_per_s"]) if (bb and pp) else None,
            "ratio_ceiling_from_link": (link_opts / pp["median_options_per_s"]) if pp else None})
        for loop, got in (("plain", pp), ("batched", bb)):
            if not got:
                low = min(sweep[loop], key=lambda p: p["rate_per_s"])
                equal[-1][f"{loop}_note"] = (
                    f"the {loop} loop's median p99 exceeded {bound:g} ms at every swept rate "
                    f"(lowest {low['rate_per_s']:g} req/s: {low['median_p99_ms']:.2f} ms)")
    return equal


def serve_record(args, local, repeats=3, trace_rate=20000.0, trace_seconds=5.0,
                 batched_rates=(50000, 55000, 60000, 65000, 70000, 75000, 80000),
                 plain_rates=(500, 1000, 2500, 5000, 7500, 10000, 12500, 15000)):
    """Config 5 in bounded form: (1) the specified trace (Poisson arrivals at
    20k requests/s, sizes log-uniform in [16, 2^20], 64 GB budget) for
    trace_seconds through the continuous-batching server and through the
    plain loop (one request at a time: copies, one launch, copy back);
    (2) the throughput each loop sustains with p99 under 0.5, 1 and 2 ms:
    traces at several rates, each repeated `repeats` times, the median p99
    and median throughput per rate; a loop's figure for a bound is its best
    median throughput whose median p99 stays under the bound.  The host
    link caps the batched loop (24 B/option inbound), so the ratio at a bound
    can be no larger than link options/s over the plain loop's figure."""
    host, out = serve_host_pool(local)
    trace = {}
    for mode in ("batched", "plain"):
        r = serve_point(host, out, mode, trace_rate, trace_seconds, args, local, SEED + 20)
        trace[mode] = {"requests": r["requests"], "completed": r["completed"],
                       "options_per_s": r["options_per_s"], "p50_ms": 1e3 * r["p50_s"],
                       "p99_ms": 1e3 * r["p99_s"], "p999_ms": 1e3 * r["p999_s"],
                       "max_ms": 1e3 * r["max_s"],
                       "late_submit_max_ms": 1e3 * r["late_submit_max_s"]}
    sweep = {}
    for mode, rates in (("batched", batched_rates), ("plain", plain_rates)):
        pts = []
        for rate in rates:
            secs = float(min(3.0, max(1.0, 4000.0 / rate)))
            reps = [serve_point(host, out, mode, rate, secs, args, local, SEED + int(rate) + 7 * k)
                    for k in range(repeats)]
            ok = all(x["completed"] == x["requests"] for x in reps)
            pts.append({"rate_per_s": rate, "seconds": secs,
                        "requests": [x["requests"] for x in reps],
                        "p99_ms": [round(1e3 * x["p99_s"], 4) for x in reps],
                        "p50_ms": [round(1e3 * x["p50_s"], 4) for x in reps],
                        "median_p99_ms": float(np.median([1e3 * x["p99_s"] for x in reps])),
                        "median_options_per_s": float(np.median([x["options_per_s"] for x in reps])),
                        "late_submit_max_ms": round(1e3 * max(x["late_submit_max_s"] for x in reps), 3),
                        "all_completed": ok})
        sweep[mode] = pts

    link = host_link_bandwidth(local)
    link_opts = link["h2d_GBps"] * 1e9 / 24
    # one request's own time: 2^20-option requests, one at a time (500/s),
    # against the time its 24 MB in and 4 MB out take on the link alone
    big = 1 << 20
    alone = {m: serve_point(host, out, m, 500.0, 2.0, args, local, SEED + 99, sizes=(big, big))
             for m in ("batched", "plain")}
    single = {m: {"p50_ms": 1e3 * r["p50_s"], "p99_ms": 1e3 * r["p99_s"]} for m, r in alone.items()}
    single["link_alone_ms"] = 1e3 * (24 * big / (link["h2d_GBps"] * 1e9) +
                                     4 * big / (link["d2h_GBps"] * 1e9))
    equal = equal_p99(sweep, SERVE_BOUNDS_MS, link_opts)
    sat = max(p["median_options_per_s"] for p in sweep["batched"])
    return {
        "workload": f"open-loop Poisson trace at {trace_rate:g} req/s for {trace_seconds:g} s, "
                    f"sizes log-uniform in [{args.serve_sizes.replace(',', ', ')}], 64 GB device "
                    "budget; equal-p99 sweep: medians of "
                    f"{repeats} traces per rate",
        "batched_path": {0: "gather, batch kernel, scatter", 1: "one fused kernel per batch",
                         2: "persistent kernel over a host-memory request ring"}[args.serve_fused],
        "plain_path": "one thread, one request at a time: six H2D copies, one plain map launch, "
                      "one D2H copy, event polled",
        "trace": trace,
        "throughput_at_equal_p99": equal,
        "single_request_2p20": single,
        "host_link": link,
        "roofline": {"bound": "host link (H2D)", "achieved": sat * 24 / 1e9,
                     "peak": link["h2d_GBps"], "unit": "GB/s",
                     "frac": sat * 24 / 1e9 / link["h2d_GBps"],
                     "note": "peak measured live: pinned host-to-device copy of 1 GiB; "
                             "achieved = the best median batched options/s of the sweep x 24 B "
                             "inbound per option"},
        "sweep": sweep,
    }


def run_serve(args, rank, world, local):
    """--config serve: the serving record as its own JSON line, with the
    sweep of arrival rates given on the command line."""
    import torch

    from p3arsec_gb300 import build as b
    b.build()
    torch.cuda.set_device(local)
    brates = [float(x) for x in args.serve_batched_rates.split(",")]
    prates = [float(x) for x in args.serve_plain_rates.split(",")]
    rec = serve_record(args, local, repeats=args.serve_repeats, trace_rate=args.serve_rate,
                       trace_seconds=args.serve_seconds, batched_rates=brates,
                       plain_rates=prates)
    t = rec["trace"]["batched"]
    line = {"metric": "serving: options/s with p50/p99/p99.9 latency vs plain per-request launch",
            "value": t["options_per_s"], "unit": UNIT, "n_gpus": world, "higher_is_better": True,
            "dtype": "f32", "data": "synthetic (seeded trace and books)",
            "config": {"workload": rec["workload"], "batched_path": rec["batched_path"],
                       "plain_path": rec["plain_path"]},
            **{k: rec[k] for k in ("trace", "throughput_at_equal_p99", "single_request_2p20",
                                   "host_link", "roofline", "sweep")}}
    if rank == 0:
        print(json.dumps(line), flush=True)


def run_serve_blocks(args, rank, world, local):
    """--config serve-blocks: the persistent kernel's grid size against the
    batched loop's throughput and latency (one trace per rate and size)."""
    import torch

    from p3arsec_gb300 import build as b
    b.build()
    torch.cuda.set_device(local)
    if rank != 0:
        return
    host, out = serve_host_pool(local)
    rates = [float(x) for x in args.serve_block_rates.split(",")]
    rows = []
    for blocks in (int(x) for x in args.serve_block_list.split(",")):
        args.serve_blocks = blocks
        for rate in rates:
            r = serve_point(host, out, "batched", rate, args.serve_seconds, args, local,
                            SEED + int(rate))
            rows.append({"blocks": blocks or "default", "rate_per_s": rate,
                         "options_per_s": r["options_per_s"], "p50_ms": 1e3 * r["p50_s"],
                         "p99_ms": 1e3 * r["p99_s"], "p999_ms": 1e3 * r["p999_s"]})
            print(json.dumps(rows[-1]), file=sys.stderr, flush=True)
    print(json.dumps({"metric": "persistent serving kernel: grid size vs throughput and latency",
                      "unit": UNIT, "n_gpus": world, "higher_is_better": True, "dtype": "f32",
                      "data": "synthetic (seeded trace)",
                      "config": {"workload": f"open-loop Poisson traces of {args.serve_seconds:g} s, "
                                             f"sizes log-uniform in [{args.serve_sizes}]"},
                      "rows": rows}), flush=True)


# --------------------------------------------------------- FP64 product mode
def fp64_record(args, local, n=None, runs=None, steps=None, warmup=None):
    """The FP64 product mode (double storage, the SIMD variant's NCO = 2
    types): options/s of num_runs passes, the roofline that binds it, and
    its prices against the CPU FP64 oracle (timed single-threaded as the
    baseline of this mode)."""
    import torch

    import oracle
    from p3arsec_gb300 import Context, books
    n = args.n if n is None else n
    runs = args.runs if runs is None else runs
    steps = args.steps if steps is None else steps
    warmup = args.warmup if warmup is None else warmup
    book = books.generate(n, seed=SEED + 8)
    dev = [torch.from_numpy(a).to(f"cuda:{local}") for a in oracle.widened(book)]
    ot = torch.from_numpy(book.otype).to(f"cuda:{local}")
    out = torch.empty(n, dtype=torch.float64, device=f"cuda:{local}")
    ctx = Context(local, max_options=1)
    stream = torch.cuda.ExternalStream(ctx.stream, device=f"cuda:{local}")

    def step():
        ctx.price_soa_f64(*dev, ot, out, n=n, num_runs=runs, device=True, asynchronous=True)

    for _ in range(warmup):
        step()
    torch.cuda.synchronize()
    l0 = ctx.launches
    secs, clk = time_steps(stream, step, steps, 0, clocks_device=local)
    launches = ctx.launches - l0
    got = out.cpu().numpy()
    ctx.close()
    cpu = None
    rel = of_spot = held = None
    if n <= (1 << 22):
        t0 = time.perf_counter()
        want = oracle.price_fp64(book)
        cpu_s = time.perf_counter() - t0
        rel = float(np.max(np.abs(got - want) / np.maximum(np.abs(want), 1e-300)))
        # far out of the money a price is what the roundings of two N to 2^-53
        # leave (of either sign): there any relative figure is noise against noise
        spot = np.maximum(book.sptprice, book.strike).astype(np.float64)
        of_spot = float(np.max(np.abs(got - want) / spot))
        big = np.abs(want) > 1e-6 * spot
        held = float(np.max(np.abs(got - want)[big] / np.abs(want)[big]))
        cpu = {"value": n / cpu_s, "unit": UNIT, "cores": 1, "kind": "port",
               "sample": f"{n} options, one pass of the FP64 oracle (the same formula in double)"}
    value = n * runs * steps / secs
    return {"workload": f"FP64 map, {n} options, {runs} passes per step", "options": n,
            "num_runs": runs, "steps": steps, "warmup": warmup,
            "value": value, "unit": UNIT, "ms_per_step": 1e3 * secs / steps, "dtype": "f64",
            "roofline": {"bound": "integer multiply-add issue", "achieved_GBps": 52 * value / 1e9,
                         "note": "52 B/option would allow ~1.3e11 options/s from HBM; "
                                 "the fixed-point arithmetic binds first"},
            "max_rel_vs_cpu_fp64": rel, "max_rel_above_1e-6_of_max_s_k": held,
            "max_diff_over_max_s_k": of_spot, "cpu_baseline": cpu,
            "gpu_launches": launches, "clocks": clk}


def run_fp64(args, rank, world, local):
    """--config fp64: the FP64 product mode's record as its own JSON line."""
    import torch

    from p3arsec_gb300 import build as b
    b.build()
    torch.cuda.set_device(local)
    rec = fp64_record(args, local)
    line = {"metric": "FP64 product mode: options/s (double storage)", "value": rec["value"],
            "unit": UNIT, "n_gpus": world, "steps": rec["steps"], "warmup": rec["warmup"],
            "ms_per_step": rec["ms_per_step"], "higher_is_better": True, "dtype": "f64",
            "data": "synthetic (seeded book widened to double)",
            "config": {"workload": rec["workload"], "options": rec["options"],
                       "num_runs": rec["num_runs"]},
            **{k: rec[k] for k in ("roofline", "max_rel_vs_cpu_fp64", "max_rel_above_1e-6_of_max_s_k",
                                   "max_diff_over_max_s_k", "cpu_baseline",
                                   "gpu_launches", "clocks")}}
    if rank == 0:
        print(json.dumps(line), flush=True)


# ---------------------------------------------------------------- file I/O
def io_record(args, n=None):
    """The reference's file formats: parallel parse / write of libbsgpu.so vs
    the reference's sequential fscanf / fprintf loops (oracle restatement),
    same files, results checked byte for byte."""
    import shutil

    import oracle
    from p3arsec_gb300 import abi, books
    oracle.build(ref=False)
    n = args.n if n is None else n
    book = books.generate(n, seed=SEED + 7)
    prices = oracle.price_ref(book.slice(0, min(n, 1 << 20)))
    prices = np.resize(prices, n).astype(np.float32)
    d = tempfile.mkdtemp(prefix="bsg_io_")
    try:
        inp = os.path.join(d, "in.txt")
        t0 = time.perf_counter()
        abi.write_parsec_input(inp, book)
        t_gen = time.perf_counter() - t0
        mb_in = os.path.getsize(inp) / 1e6
        threads = os.cpu_count() or 1
        best = 1e30
        for _ in range(3):
            t0 = time.perf_counter()
            got, _ = abi.read_parsec(inp)
            best = min(best, time.perf_counter() - t0)
        t0 = time.perf_counter()
        ref, _ = oracle.read_parsec_fscanf(inp, n)
        t_ref = time.perf_counter() - t0
        same_in = all(np.array_equal(x.view(np.uint32), y.view(np.uint32))
                      for x, y in zip(got.arrays(), ref.arrays()))
        o1, o2 = os.path.join(d, "o1.txt"), os.path.join(d, "o2.txt")
        bw = 1e30
        for _ in range(3):
            t0 = time.perf_counter()
            abi.write_parsec_prices(o1, prices)
            bw = min(bw, time.perf_counter() - t0)
        t0 = time.perf_counter()
        oracle.write_prices_fprintf(o2, prices)
        t_refw = time.perf_counter() - t0
        mb_out = os.path.getsize(o1) / 1e6
        with open(o1, "rb") as f1, open(o2, "rb") as f2:
            same_out = f1.read() == f2.read()
    finally:
        shutil.rmtree(d, ignore_errors=True)
    return {
        "workload": f"{n} options: parse a {mb_in:.0f} MB input file, write a "
                    f"{mb_out:.0f} MB %.18f output file", "options": n, "threads": threads,
        "value": n / best, "unit": UNIT,
        "parse": {"ours_s": best, "ours_MBps": mb_in / best, "reference_fscanf_s": t_ref,
                  "speedup": t_ref / best, "bit_identical": same_in},
        "write": {"ours_s": bw, "ours_MBps": mb_out / bw, "reference_fprintf_s": t_refw,
                  "speedup": t_refw / bw, "byte_identical": same_out},
        "input_generation_s": t_gen,
        "cpu_baseline": {"value": n / t_ref, "unit": UNIT, "cores": 1, "kind": "port",
                         "sample": "the reference's fscanf loop (blackscholes.c:726-734) on the "
                                   "same file"},
    }


def run_io(args, rank, world, local):
    """--config io: the file-format record as its own JSON line (host code)."""
    from p3arsec_gb300 import build as b
    b.build()
    if rank != 0:
        return
    rec = io_record(args)
    line = {"metric": "PARSEC file I/O: options/s parsed and written (reference formats)",
            "value": rec["value"], "unit": UNIT, "n_gpus": 0, "higher_is_better": True,
            "dtype": "f32", "data": "synthetic (seeded book)",
            "config": {"workload": rec["workload"], "threads": rec["threads"]},
            **{k: rec[k] for k in ("parse", "write", "input_generation_s", "cpu_baseline")}}
    print(json.dumps(line), flush=True)


# --------------------------------------------------------------- swaptions
def swaptions_record(args, local, nsw=None, trials=None, steps=None, warmup=None, sample=None):
    """The swaptions application (P3ARSEC's HJM Monte Carlo,
    HJM_Swaption_Blocking.cpp): nsw swaptions of the reference driver's
    kind, `trials` paths each, priced in one call of bsg_price_swaptions per
    step (host arrays in, prices out, the call synchronises); the CPU oracle
    (the same model and random stream, the whole path matrix as the
    reference simulates it) on every host core over `sample` paths per
    swaption is the CPU baseline, and the GPU's prices on that sample are
    checked against it."""
    import oracle
    from p3arsec_gb300 import Context
    from p3arsec_gb300 import swaptions as S
    oracle.build(ref=False)
    nsw = args.swaptions if nsw is None else nsw
    trials = args.trials if trials is None else trials
    steps = args.steps if steps is None else steps
    warmup = args.warmup if warmup is None else warmup
    sample = min(trials, args.swaption_sample if sample is None else sample)
    sw = S.generate(nsw, seed=1979)
    ctx = Context(local, max_options=1)
    for _ in range(warmup):
        ctx.price_swaptions(sw, trials)
    l0 = ctx.launches
    times = []
    with ClockSampler(local) as clk:
        for _ in range(steps):
            t0 = time.perf_counter()
            price, err = ctx.price_swaptions(sw, trials)
            times.append(time.perf_counter() - t0)
    launches = ctx.launches - l0
    secs = float(np.median(times))
    g_s, _ = ctx.price_swaptions(sw, sample)
    ctx.close()
    threads = os.cpu_count() or 1
    c_s, _, _ = oracle.swaptions_all(sw, sample, threads)  # the checker's build
    _, _, c_secs = oracle.swaptions_all(sw, sample, threads, parsec_flags=True)  # timed
    rel = float(np.max(np.abs(g_s - c_s) / np.maximum(np.abs(c_s), 1e-12)))
    return {
        "workload": f"{nsw} swaptions x {trials} paths, 11-point HJM grid, 3 factors, one "
                    "bsg_price_swaptions call per step (host arrays in, prices out)",
        "swaptions": nsw, "trials": trials, "steps": steps, "warmup": warmup,
        "value": nsw * trials / secs, "unit": "paths/s", "ms_per_step": 1e3 * secs,
        "dtype": "f64",
        "step_time_s": {"median": secs, "min": min(times), "max": max(times)},
        "prices": {"first": price[:4].tolist(), "std_err_first": err[:4].tolist()},
        "gpu_launches": launches,
        "bound": "integer multiply-add issue (the kernel reads no bulk data; ncu: that pipe 71 % busy)",
        "vs_oracle": {"sample_trials": sample, "max_rel_price_diff": rel,
                      "note": "the same paths on the CPU oracle; parity with the reference "
                              "itself is unpinned (its model core is not in its tree)"},
        "cpu_baseline": {"value": nsw * sample / c_secs, "unit": "paths/s", "cores": threads,
                         "kind": "port",
                         "sample": f"{nsw} swaptions x {sample} paths, static partition over "
                                   f"{threads} threads, {c_secs:.2f} s (the oracle simulates every "
                                   "row of each path, as the reference does)"},
        "clocks": clk.summary(),
    }


def run_swaptions(args, rank, world, local):
    """--config swaptions: the swaptions record as its own JSON line."""
    import torch

    from p3arsec_gb300 import build as b
    b.build()
    torch.cuda.set_device(local)
    rec = swaptions_record(args, local)
    line = {"metric": "swaption paths/s (HJM Monte Carlo, FP64)", "value": rec["value"],
            "unit": "paths/s", "n_gpus": world, "steps": rec["steps"], "warmup": rec["warmup"],
            "ms_per_step": rec["ms_per_step"], "higher_is_better": True, "dtype": "f64",
            "data": "synthetic (the reference driver's swaption set, seeded)",
            "config": {"workload": rec["workload"], "swaptions": rec["swaptions"],
                       "trials": rec["trials"]},
            **{k: rec[k] for k in ("step_time_s", "prices", "gpu_launches", "bound", "vs_oracle",
                                   "cpu_baseline", "clocks")}}
    if rank == 0:
        print(json.dumps(line), flush=True)


# ---------------------------------------------------- resident-prefix sweep
def run_prefix_sweep(args, rank, world, local):
    """The map over one book for every (shape, resident prefix size): the
    resident-prefix load path (7) with resident_32nds 32nds of the L2, and
    the same shape with every line evict-first (6) for 0.  Each point is
    `steps` timed steps of NUM_RUNS passes after the warm-up steps.  The
    autotuner searches the same sizes on its best resident-prefix shape."""
    import torch

    from p3arsec_gb300 import Context, books
    from p3arsec_gb300 import build as b
    b.build()
    torch.cuda.set_device(local)
    n, runs = args.n, args.runs
    dev = (books.generate_device(n, SEED, device=f"cuda:{local}") if n > (1 << 24) else
           [torch.from_numpy(a).to(f"cuda:{local}") for a in books.generate(n, seed=SEED).arrays()])
    out = torch.empty(n, dtype=torch.float32, device=f"cuda:{local}")
    ctx = Context(local, max_options=1)
    stream = torch.cuda.ExternalStream(ctx.stream, device=f"cuda:{local}")
    l2 = l2_bytes(local)
    shapes = [tuple(int(x) for x in sh.split(",")) for sh in args.sweep_shapes.split(";")]
    sizes = [int(x) for x in args.sweep_32nds.split(",")]
    rows = []
    for vpt, block, bps in shapes:
        for r32 in sizes:
            tune = (vpt, block, bps, 7 if r32 else 6, 1, r32)
            ctx.set_tune(*tune)

            def step():
                ctx.price_soa(*dev, out, n=n, num_runs=runs, device=True, asynchronous=True)

            secs, _ = time_steps(stream, step, args.steps, args.warmup)
            per_pass = secs / (runs * args.steps)
            t = ctx.get_tune()
            rows.append({"tune": ",".join(str(x) for x in tune),
                         "prefix_bytes": prefix_bytes(t, n, l2),
                         "us_per_pass": round(per_pass * 1e6, 3),
                         "options_per_s": n / per_pass,
                         "frac_of_hbm": BYTES_PER_OPTION * n / per_pass / 1e9 / measured_hbm_peak()[0]})
            print(json.dumps({"sweep_point": rows[-1]}), file=sys.stderr, flush=True)
    best = max(rows, key=lambda r: r["options_per_s"])
    line = {"metric": "resident-prefix sweep: options/s per (shape, prefix size)",
            "value": best["options_per_s"], "unit": UNIT, "n_gpus": 1, "steps": args.steps,
            "warmup": args.warmup, "higher_is_better": True, "dtype": "f32",
            "data": "synthetic (seeded book)",
            "config": {"workload": f"plain map, {n} options, NUM_RUNS={runs} passes per step",
                       "options": n, "num_runs": runs, "l2_bytes": int(l2)},
            "best": best, "points": rows}
    if rank == 0:
        print(json.dumps(line), flush=True)
    ctx.close()


# ---------------------------------------------------------- reference arm
def run_reference(args, rank, world, local):
    """The reference's CPU path (the oracle port of its FastFlow map: its
    arithmetic, static partition, a join per pass, built with PARSEC's
    flags) on every host core.  Rank 0 only; other ranks exit without work."""
    if rank != 0:
        return
    import oracle
    from p3arsec_gb300 import books
    oracle.build(ref=False)
    n = args.n
    book = books.generate(n, seed=SEED)
    threads = os.cpu_count() or 1
    _, t1 = oracle.bs_map(book, threads, 1, parsec_flags=True)
    # each step a bounded sample: ~2 s of CPU work, less when many steps are
    # asked for, so that the whole run stays near a minute
    runs = int(max(1, min(args.runs, round(min(2.0, 60.0 / args.steps) / max(t1, 1e-6)))))
    for _ in range(args.warmup):
        oracle.bs_map(book, threads, runs, parsec_flags=True)
    total = 0.0
    for _ in range(args.steps):
        _, s = oracle.bs_map(book, threads, runs, parsec_flags=True)
        total += s
    value = n * runs * args.steps / total
    sample = (f"each step {n} options x {runs} passes (of {NUM_RUNS}) on {threads} threads")
    line = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": 1e3 * total / args.steps,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
        "data": "synthetic (seeded book, reference config distributions)",
        "config": map_config(n, args.runs, world),
        "impl": "reference",
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": threads, "kind": "port",
                         "sample": sample, "note": PORT_NOTE},
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


def main(argv=None):
    ap = argparse.ArgumentParser(description=__doc__)
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=None,
                    help="timed steps (default: 100 for the map, 10 otherwise)")
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--config", choices=["map", "batch", "precision", "serve", "serve-blocks", "io",
                                         "fp64", "prefix-sweep", "swaptions"],
                    default="map")
    ap.add_argument("--serve-rate", type=float, default=20000.0,
                    help="serve: arrival rate of the specified trace (req/s)")
    ap.add_argument("--serve-seconds", type=float, default=5.0,
                    help="serve: length of the specified trace")
    ap.add_argument("--serve-batched-rates", default="50000,55000,60000,65000,70000,75000,80000",
                    help="serve: arrival rates of the batched loop's equal-p99 sweep")
    ap.add_argument("--serve-plain-rates", default="500,1000,2500,5000,7500,10000,12500,15000",
                    help="serve: arrival rates of the plain loop's equal-p99 sweep")
    ap.add_argument("--serve-repeats", type=int, default=3,
                    help="serve: traces per rate (medians are reported)")
    ap.add_argument("--serve-sizes", default="16,1048576",
                    help="serve config: request sizes log-uniform in [lo, hi] options")
    ap.add_argument("--serve-inflight", type=int, default=8)
    ap.add_argument("--serve-fused", type=int, default=2,
                    help="2: the persistent kernel; 1: one fused kernel per batch; "
                         "0: gather, price, scatter")
    ap.add_argument("--serve-blocks", type=int, default=0,
                    help="serve: blocks of the persistent kernel (0 = SMs x min(occupancy, 3))")
    ap.add_argument("--serve-window", type=int, default=0,
                    help="serve: requests the persistent kernel's blocks share (0 = default)")
    ap.add_argument("--serve-block-list", default="16,32,64,128,0",
                    help="serve-blocks config: the persistent kernel's grid sizes to sweep")
    ap.add_argument("--serve-block-rates", default="20000,60000,70000,80000",
                    help="serve-blocks config: arrival rates per grid size")
    ap.add_argument("--books", type=int, default=4096, help="batch config: number of books")
    ap.add_argument("--batch-tune", default=None,
                    help="batch config: tile_options,blocks_per_sm instead of autotuning")
    ap.add_argument("--n", "--options", dest="n", type=int, default=N_OPTIONS)
    ap.add_argument("--runs", type=int, default=NUM_RUNS)
    ap.add_argument("--no-cpu", action="store_true", help="skip the cpu_baseline leg")
    ap.add_argument("--no-e2e", action="store_true", help="skip the host-buffer leg")
    ap.add_argument("--no-accuracy", action="store_true", help="skip the FP64 error report")
    ap.add_argument("--swaptions", type=int, default=128,
                    help="swaptions config: number of swaptions")
    ap.add_argument("--trials", type=int, default=1_000_000,
                    help="swaptions config: Monte Carlo paths per swaption")
    ap.add_argument("--swaption-sample", type=int, default=200_000,
                    help="swaptions config: paths per swaption of the CPU-oracle sample")
    ap.add_argument("--repeats", type=int, default=3,
                    help="map: extra timed windows of the same steps (their spread is reported)")
    ap.add_argument("--no-nested", action="store_true",
                    help="map: skip the nested 2^28, batch and serve records")
    ap.add_argument("--records", default=None, metavar="FILE",
                    help="map: write the line with every nested record in full to FILE")
    ap.add_argument("--tune", default=None,
                    help="vec_per_thread,block,blocks_per_sm,load_path[,pdl[,resident_32nds]] "
                         "instead of autotuning")
    ap.add_argument("--sweep-shapes", default="1,128,2;1,128,4;1,128,8;1,256,2;1,256,4;1,512,2",
                    help="prefix-sweep: vec_per_thread,block,blocks_per_sm shapes")
    ap.add_argument("--sweep-32nds", default="0,4,8,10,12,14,15,16,18,20,24",
                    help="prefix-sweep: resident prefix sizes in 32nds of the L2 (0: none)")
    args = ap.parse_args(argv)
    if args.steps is None:
        args.steps = 100 if (args.config == "map" and args.impl == "ours") else 10
    if args.warmup < 3:
        ap.error("--warmup must be >= 3")
    rank, world, local = dist_env()
    if args.impl == "reference":
        run_reference(args, rank, world, local)
    elif args.config == "batch":
        run_batch(args, rank, world, local)
    elif args.config == "precision":
        run_precision(args, rank, world, local)
    elif args.config == "serve":
        run_serve(args, rank, world, local)
    elif args.config == "serve-blocks":
        run_serve_blocks(args, rank, world, local)
    elif args.config == "io":
        run_io(args, rank, world, local)
    elif args.config == "fp64":
        run_fp64(args, rank, world, local)
    elif args.config == "prefix-sweep":
        run_prefix_sweep(args, rank, world, local)
    elif args.config == "swaptions":
        run_swaptions(args, rank, world, local)
    else:
        run_ours(args, rank, world, local)


if __name__ == "__main__":
    main()
