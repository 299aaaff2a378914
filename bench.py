#!/usr/bin/env python
"""Benchmark of the MLA-decode hot path.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference] [--workload c1|c2|c3|c4]

One step = one `custom_kernel(data)` call (Q quantisation where the workload has FP8 Q, split-KV
decode, LSE merge) over one batch of seeded synthetic input with the shapes and value
distributions of the BASELINE configuration (default c1: FP8 Q + FP8 KV, batch 32, 16 heads,
KV length 4096, page size 1 behind a shuffled page table).

Prints ONE JSON line (rank 0).  Keys beyond the base contract:
  us_per_call, achieved_gbs   the other two forms of the headline metric
  roofline                    the decode launch (maximum of Q, split-KV decode, merge): algorithmic bytes per
                              launch / its CUDA-event duration, against the measured HBM copy bandwidth;
                              `step`: the same over the duration of a timed step, whose launches overlap
  cpu_baseline                the CPU oracle (torch fp32 dequantise-then-attend) timed on this host
  e2e                         the same call with every input staged from pinned host memory and
                              the output copied back, copies inside the timed region

With N > 1 (torchrun) every rank decodes its own batch (sequences are independent, no
collective): weak scaling.  `--impl reference` times the CPU oracle port (the reference has no
implementation that runs without AMD's aiter library) on rank 0 only.
"""
from __future__ import annotations

import argparse
import ctypes
import json
import math
import os
import statistics
import subprocess
import sys
import tempfile
import time

import torch

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

WORKLOADS = {
    # name: (batch, q_len, heads, kv_len or (lo, hi), kv_format, q_format)
    "c1": dict(batch=32, q_len=1, heads=16, kv_len=4096, kv_format="fp8", q_format="fp8",
               desc="FP8 Q + FP8 KV, B32 H16 q1 S4096, page_size 1 shuffled (BASELINE configs[1])"),
    "c2": dict(batch=64, q_len=1, heads=16, kv_len=8192, kv_format="mxfp4", q_format="bf16",
               desc="bf16 Q + MXFP4 KV, B64 H16 q1 S8192, page_size 1 shuffled (BASELINE configs[2])"),
    "c3": dict(batch=128, q_len=1, heads=128, kv_len=(1024, 16384), kv_format="hybrid", q_format="fp8",
               desc="FP8 Q + hybrid KV, B128 H128 q1 S~U[1024,16384] (BASELINE configs[3])"),
    "c4": dict(batch=8, q_len=2, heads=16, kv_len=131072, kv_format="mxfp4", q_format="bf16",
               desc="bf16 Q + MXFP4 KV, B8 H16 q2 S131072 causal (BASELINE configs[4])"),
}
KV_ROW_BYTES = {"fp8": 576, "mxfp4": 306, "hybrid": 336}
# how a workload uses N > 1 GPUs: independent replicas (weak scaling), a token-balanced split of the
# batch (strong, no collective), or each sequence's keys split over the GPUs (strong, one all-gather)
MODES = {"c1": "replica", "c2": "replica", "c3": "batch_shard", "c4": "split_kv"}
# DRAM bytes read + written by one decode launch, from one ncu capture of that workload's kernel on one GPU
# (profiles/ holds each capture's summary and command; regenerate them together with the kernels).
NCU_TRAFFIC_BYTES = {"c1": 77.8e6, "c2": 190.0e6, "c3": 606.5e6, "c4": 427.9e6}
L2_BYTES = 126 << 20


def algorithmic_bytes(w, total_kv):
    q_elt = 1 if w["q_format"] == "fp8" else 2
    rows = w["batch"] * w["q_len"] * w["heads"]
    return (total_kv * KV_ROW_BYTES[w["kv_format"]] + rows * 576 * q_elt + rows * 512 * 2
            + total_kv * 4 + (w["batch"] + 1) * 8)


def measured_peak_gbs():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            return float(json.load(f)["hbm_gbs"]), "measured"
    except Exception:
        return 6650.0, "fallback"


def measured_peak_tflops():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            return float(json.load(f)["bf16_tflops"]), "measured"
    except Exception:
        return 1590.0, "fallback"


def make_lens(w, seed):
    if isinstance(w["kv_len"], tuple):
        g = torch.Generator().manual_seed(seed)
        lo, hi = w["kv_len"]
        return torch.randint(lo, hi + 1, (w["batch"],), generator=g).tolist()
    return None


class ClockSampler:
    """nvidia-smi sampled every 100 ms while the timed region runs."""
    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index):
        self.idx, self.proc, self.path = gpu_index, None, None

    def __enter__(self):
        try:
            fd, self.path = tempfile.mkstemp(suffix=".csv")
            os.close(fd)
            self.proc = subprocess.Popen(["nvidia-smi", f"--id={self.idx}", f"--query-gpu={self.Q}",
                                          "--format=csv,noheader,nounits", "-lms", "100"],
                                         stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except Exception:
            self.proc = None
        return self

    def __exit__(self, *a):
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                self.proc.kill()

    def summary(self):
        out = {"sm_mhz": None, "sm_max_mhz": None, "reasons": []}
        try:
            rows = [r.split(",") for r in open(self.path).read().strip().splitlines() if r.strip()]
            sm = [float(r[1]) for r in rows]
            out["sm_mhz"] = statistics.median(sm)
            out["sm_max_mhz"] = float(rows[0][2])
            names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
            seen = set()
            for r in rows:
                for n, v in zip(names, r[5:9]):
                    if v.strip().lower().startswith("active"):
                        seen.add(n)
            out["reasons"] = sorted(seen)
            out["samples"] = len(rows)
        except Exception:
            pass
        finally:
            if self.path and os.path.exists(self.path):
                os.unlink(self.path)
        return out


def cpu_oracle_step(host):
    """One full workload call through the CPU oracle (torch fp32, all host threads)."""
    from oracle import mla_oracle as mo
    q, q_scale = host["q"], None
    if host["w"]["q_format"] == "fp8":
        q, q_scale = mo.quantize_fp8_per_tensor(q)
    return mo.decode_from_data(q, q_scale, host["w"]["kv_format"], host["kv"], host["kv_indptr"].numpy(),
                               host["kv_indices"].numpy(), host["sm_scale"], q_len=host["w"]["q_len"])


def time_cpu(host, reps):
    cpu_oracle_step(host)                                   # warm-up
    ts = []
    for _ in range(reps):
        t0 = time.perf_counter()
        cpu_oracle_step(host)
        ts.append(time.perf_counter() - t0)
    return statistics.median(ts)


# ---------------------------------------------------------------------------------------------------
# the two sharded multi-GPU modes, measured inside the default run when it spans more than one GPU
# ---------------------------------------------------------------------------------------------------

def _gpu_time_us(fn, steps, dev, dist=None, world=1, spin_cycles=int(4e7)):
    """Device time per step of `fn`, microseconds, max over ranks.  The steps are queued behind a GPU spin so
    that the host's launch work for all of them is done before the first one runs (the same number of
    steps on every rank, so that collectives inside `fn` pair up)."""
    for _ in range(3):
        fn()
    torch.cuda.synchronize()
    if dist is not None and world > 1:
        dist.barrier()
        torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    torch.cuda._sleep(spin_cycles)
    e0.record()
    for _ in range(steps):
        fn()
    e1.record()
    torch.cuda.synchronize()
    t = torch.tensor([e0.elapsed_time(e1) * 1e3 / steps], device=dev)
    if dist is not None and world > 1:
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def _stage1_us(pkg, fn, reps, dev, dist=None, world=1):
    """Mean duration of the decode launch inside `fn` (events recorded by the library), max over ranks."""
    lib = pkg._cabi.lib
    pairs = []
    for _ in range(reps):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(); b.record()
        pairs.append((a, b))
    torch.cuda.synchronize()
    torch.cuda._sleep(int(2e7))
    for a, b in pairs:
        lib.b200_mla_set_stage1_events(ctypes.c_void_p(a.cuda_event), ctypes.c_void_p(b.cuda_event))
        fn()
    lib.b200_mla_set_stage1_events(None, None)
    torch.cuda.synchronize()
    t = torch.tensor([statistics.mean(a.elapsed_time(b) for a, b in pairs) * 1e3], device=dev)
    if dist is not None and world > 1:
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def sharded_modes(pkg, dist, rank, world, dev, kernel="auto", steps=30):
    """BASELINE configs 3 and 4 in the multi-GPU modes they are defined for, on `world` GPUs, next to the same
    workload on ONE GPU measured in the same process group (every rank runs the whole problem on its own GPU
    with no collective; max over ranks).  Inputs are drawn on the GPU from one seed, so every rank holds the
    identical global problem and takes its shard of it."""
    import amd_optimization_challenge_b200.inputs as gen
    from amd_optimization_challenge_b200.distributed import (PeerSplitKVDecoder, SplitKVDecoder, cuda_partial_fn,
                                                             shard_batch, split_kv_shard, token_balanced_partition)
    out = {}

    # ---- config 3: token-balanced batch sharding, no data-path collective
    w = WORKLOADS["c3"]
    lens = make_lens(w, 1234)
    full = gen.generate_input(w["batch"], 1, max(lens), 1234, num_heads=w["heads"], kv_lens=lens, shuffle_pages=True,
                              formats=("hybrid",), device=dev, generator_device="cuda")
    cfg = dict(full[4], kv_format="hybrid", q_format="fp8", impl=kernel)
    full = (full[0], full[1], full[2], full[3], cfg)
    ids = token_balanced_partition(lens, world)[rank]
    mine = shard_batch(full, ids)
    t1 = _gpu_time_us(lambda: pkg.custom_kernel(full), steps, dev, dist, world)
    tn = _gpu_time_us(lambda: pkg.custom_kernel(mine), steps, dev, dist, world)
    s1 = _stage1_us(pkg, lambda: pkg.custom_kernel(mine), 10, dev, dist, world)
    tokens = w["batch"] * w["q_len"]
    loads = [sum(lens[i] for i in part) for part in token_balanced_partition(lens, world)]
    out["c3"] = {"mode": "token-balanced batch shard, no collective", "us_per_step": tn, "tokens_per_s": tokens / (tn * 1e-6),
                 "stage1_us_max_rank": s1, "n1_us_per_step": t1, "speedup_vs_n1": t1 / tn,
                 "efficiency_vs_n1": t1 / tn / world, "kv_tokens_per_rank": {"min": min(loads), "max": max(loads)},
                 "limiter": "decode launch of the most loaded rank (no exchange step)"}
    del full, mine
    torch.cuda.empty_cache()

    # ---- config 4: each sequence's keys split over the GPUs, one all-gather of (O || LSE), LSE merge
    w = WORKLOADS["c4"]
    B, QL, S = w["batch"], w["q_len"], w["kv_len"]
    full = gen.generate_input(B, QL, S, 4321, num_heads=w["heads"], shuffle_pages=True, formats=("mxfp4",),
                              device=dev, generator_device="cuda")
    q, kvd, _, _, cfg = full
    cfg1 = dict(cfg, kv_format="mxfp4", q_format="bf16", impl=kernel)
    t1 = _gpu_time_us(lambda: pkg.custom_kernel((q, kvd, full[2], full[3], cfg1)), steps, dev, dist, world)
    idx, ip, off, tot, n_loc = split_kv_shard(cfg["kv_indices"], B, S, rank, world)
    dec = SplitKVDecoder(B * QL, w["heads"], dev)
    part = cuda_partial_fn(q, None, "mxfp4", kvd["mxfp4"], ip, sm_scale=cfg["sm_scale"], q_len=QL, kv_indices=idx,
                           kv_pos_offset=off, kv_total_len=tot, total_kv_hint=max(B * n_loc, 1), impl=kernel)
    tn = _gpu_time_us(lambda: dec.step(part), steps, dev, dist, world)
    s1 = _stage1_us(pkg, lambda: dec.step(part), 10, dev, dist, world)
    # the three phases of a step, timed apart on the device
    trip = [tuple(torch.cuda.Event(enable_timing=True) for _ in range(3)) for _ in range(10)]
    torch.cuda.synchronize()
    dist.barrier()
    torch.cuda._sleep(int(2e7))
    for ev in trip:
        dec.step(part, events=ev)
    torch.cuda.synchronize()
    ph = torch.tensor([statistics.mean(e[0].elapsed_time(e[1]) for e in trip) * 1e3,
                       statistics.mean(e[1].elapsed_time(e[2]) for e in trip) * 1e3], device=dev)
    dist.all_reduce(ph, op=dist.ReduceOp.MAX)
    ag_us, merge_us = float(ph[0]), float(ph[1])
    tokens = B * QL
    gathered = world * dec.n * 4
    out["c4"] = {"mode": "cross-GPU split-KV, one NCCL all-gather of (O || LSE), LSE merge", "us_per_step": tn,
                 "tokens_per_s": tokens / (tn * 1e-6), "stage1_us_max_rank": s1, "all_gather_us": ag_us,
                 "merge_us": merge_us, "all_gather_bytes_received": gathered, "n1_us_per_step": t1,
                 "speedup_vs_n1": t1 / tn, "efficiency_vs_n1": t1 / tn / world,
                 "limiter": "stage-1 kernel" if s1 > 2 * (ag_us + merge_us) else "all-gather + merge",
                 "launch": "eager, queued behind a GPU spin; the all-gather is NCCL on the decode stream's order"}

    # ---- config 4 again, the exchange and the merge fused into one kernel over peer memory (no collective call)
    try:
        pdec = PeerSplitKVDecoder(B * QL, w["heads"], dev)
    except RuntimeError as e:                         # raised on every rank or on none
        out["c4"]["peer_memory"] = {"unavailable": str(e)[:300]}
        return out
    ref_out = dec.step(part)
    got = pdec.step(part)
    diff = (got.float() - ref_out.float()).abs().max().reshape(1)
    dist.all_reduce(diff, op=dist.ReduceOp.MAX)
    tp = _gpu_time_us(lambda: pdec.step(part), steps, dev, dist, world)
    pair = [tuple(torch.cuda.Event(enable_timing=True) for _ in range(2)) for _ in range(10)]
    torch.cuda.synchronize()
    dist.barrier()
    torch.cuda._sleep(int(2e7))
    for ev in pair:
        pdec.step(part, events=ev)
    torch.cuda.synchronize()
    pm = torch.tensor([statistics.mean(e[0].elapsed_time(e[1]) for e in pair) * 1e3], device=dev)
    # the rank whose stage 1 ends last does not wait in the merge kernel: its span is signal + peer reads + merge alone
    pm_min = torch.tensor([min(e[0].elapsed_time(e[1]) for e in pair) * 1e3], device=dev)
    dist.all_reduce(pm, op=dist.ReduceOp.MAX)
    dist.all_reduce(pm_min, op=dist.ReduceOp.MIN)
    word = torch.zeros(1, dtype=torch.int32).pin_memory()
    from amd_optimization_challenge_b200 import _cabi
    _cabi.check(_cabi.lib.b200_mla_read_status(None, word.data_ptr(), torch.cuda.current_stream().cuda_stream), "status")
    torch.cuda.synchronize()
    st = torch.tensor([int(word[0])], device=dev)
    dist.all_reduce(st, op=dist.ReduceOp.MAX)
    out["c4"]["peer_memory"] = {
        "mode": "cross-GPU split-KV, one fused signal + wait + merge kernel reading the peers' (O || LSE) over NVLink",
        "us_per_step": tp, "tokens_per_s": tokens / (tp * 1e-6), "exchange_and_merge_us": float(pm[0]),
        "exchange_and_merge_us_without_wait": float(pm_min[0]),
        "nvlink_bytes_read_per_gpu": (world - 1) * dec.n * 4,
        "nvlink_roofline": {"bytes": (world - 1) * dec.n * 4, "peak_gbs": 770.0, "peak_source": "measured peer copy per direction",
                            "floor_us": (world - 1) * dec.n * 4 / 770e9 * 1e6,
                            "frac": ((world - 1) * dec.n * 4 / 770e9 * 1e6) / max(float(pm_min[0]), 1e-9)}, "speedup_vs_n1": t1 / tp, "efficiency_vs_n1": t1 / tp / world,
        "speedup_vs_all_gather_mode": tn / tp, "max_abs_diff_vs_all_gather_mode": float(diff[0]),
        "status_bits_max_rank": int(st[0]),
        # the same partials merged by the same arithmetic: anything but an identical output and a clean status word
        # means the exchange went wrong, and the timings above are then not a result
        "valid": bool(float(diff[0]) == 0.0 and int(st[0]) == 0)}
    pdec.close()
    return out


# ---------------------------------------------------------------------------------------------------
# the reference's own benchmark shapes (task.yml:81-93): contiguous pages, all three caches in the tuple
# ---------------------------------------------------------------------------------------------------

REF8 = [(4, 1024, 4217), (4, 8192, 4220), (32, 1024, 5412), (32, 8192, 5415),
        (64, 1024, 1357), (64, 8192, 1360), (256, 1024, 9823), (256, 8192, 9826)]


def ref8_sweep(pkg, dev, reps=30):
    """custom_kernel on the reference's untouched tuple for its eight benchmark shapes, FP8 route (the
    reference's ref_kernel choice) and MXFP4 route: harness-style (synchronise, flush L2, events around ONE
    eager call: eval.py:225-261) and as a CUDA-graph replay over rotated cache copies."""
    import amd_optimization_challenge_b200.inputs as gen
    flush = torch.empty(256 << 20, dtype=torch.uint8, device=dev)
    rows = []
    for batch, kv_len, seed in REF8:
        data = gen.generate_input(batch, 1, kv_len, seed, device=dev, generator_device="cuda")
        q, kvd, qo, kvp, cfg = data
        cfg.pop("total_kv", None)
        row = {"batch": batch, "kv_len": kv_len}
        for fmt in ("fp8", "mxfp4"):
            c = dict(cfg) if fmt == "fp8" else dict(cfg, kv_format="mxfp4")
            tup = (q, kvd, qo, kvp, c)
            for _ in range(3):
                pkg.custom_kernel(tup)
            ts = []
            for _ in range(reps):
                torch.cuda.synchronize()
                flush.zero_()
                e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                e0.record()
                pkg.custom_kernel(tup)
                e1.record()
                torch.cuda.synchronize()
                ts.append(e0.elapsed_time(e1) * 1e3)
            row[f"{fmt}_eager_us"] = statistics.mean(ts)
            # graph replay over enough distinct copies of the cache to exceed L2
            kv_bytes = sum(t.numel() * t.element_size() for t in kvd[fmt])
            n_rot = min(6, max(2, -(-int(2.4 * L2_BYTES) // kv_bytes)))
            rot = [tup] + [(q, dict(kvd, **{fmt: tuple(t.clone() for t in kvd[fmt])}), qo, kvp, c) for _ in range(n_rot - 1)]
            graph = torch.cuda.CUDAGraph()
            side = torch.cuda.Stream()
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                with torch.cuda.graph(graph, stream=side):
                    for r in rot:
                        pkg.custom_kernel(r)
            torch.cuda.current_stream().wait_stream(side)
            torch.cuda.synchronize()
            for _ in range(3):
                graph.replay()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            for _ in range(10):
                graph.replay()
            e1.record()
            torch.cuda.synchronize()
            row[f"{fmt}_graph_us"] = e0.elapsed_time(e1) * 1e3 / (10 * n_rot)
            del graph, rot
        rows.append(row)
        del data, q, kvd
        torch.cuda.empty_cache()
    geo = lambda k: math.exp(sum(math.log(r[k]) for r in rows) / len(rows))
    return {"shapes": rows, "geomean_us": {k: geo(k) for k in ("fp8_eager_us", "fp8_graph_us", "mxfp4_eager_us", "mxfp4_graph_us")},
            "note": "contiguous pages (no kv_indices), tuple and config exactly as reference.generate_input builds them; "
                    "eager = synchronise, flush L2, CUDA events around one call (the reference harness's timing); B200"}


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=1000)
    ap.add_argument("--warmup", type=int, default=20)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--workload", default="c1", choices=sorted(WORKLOADS) + ["ref8"])
    ap.add_argument("--no-sharded", action="store_true", help="with N > 1: skip the sharded c3 / c4 measurements")
    ap.add_argument("--kernel", default="auto", choices=["auto", "generic", "tcgen05"])
    ap.add_argument("--cpu-reps", type=int, default=5)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-graph", action="store_true", help="time eager API calls instead of a CUDA graph replay")
    args = ap.parse_args()
    if args.workload == "ref8":
        torch.cuda.set_device(int(os.environ.get("LOCAL_RANK", "0")))
        import amd_optimization_challenge_b200 as pkg
        print(json.dumps({"metric": "mla_decode_us_per_call", "unit": "us", "higher_is_better": False, "n_gpus": 1,
                          "data": "synthetic", "config": {"workload": "ref8: the reference's eight benchmark shapes (task.yml:81-93)"},
                          "ref8": ref8_sweep(pkg, torch.device("cuda", torch.cuda.current_device()))}), flush=True)
        return
    w = WORKLOADS[args.workload]
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))
    n_gpus = max(args.gpus, world)
    tokens_per_call = w["batch"] * w["q_len"]

    import amd_optimization_challenge_b200.inputs as gen   # plain torch

    mode = MODES[args.workload] if world > 1 else "replica"

    def build_host(seed, shard_rank=0, shard_world=1, shard_mode="replica"):
        """Seeded host-side inputs of one rank: the whole workload, or this rank's shard of it."""
        lens = make_lens(w, 1234)                                 # the same ragged lengths on every rank
        batch, kv_len, extra = w["batch"], w["kv_len"], {}
        if shard_mode == "batch_shard":
            from amd_optimization_challenge_b200.distributed import token_balanced_partition
            all_lens = lens if lens is not None else [kv_len] * batch
            ids = token_balanced_partition(all_lens, shard_world)[shard_rank]
            lens, batch = [all_lens[i] for i in ids], len(ids)
            extra["global_total_kv"] = sum(all_lens)
        elif shard_mode == "split_kv":
            from amd_optimization_challenge_b200.distributed import kv_range_partition
            a, b = kv_range_partition(kv_len, shard_world)[shard_rank]
            extra.update(kv_pos_offset=a, kv_total_len=kv_len, global_total_kv=batch * kv_len)
            kv_len = b - a
        data = gen.generate_input(batch, w["q_len"], kv_len if lens is None else max(lens), seed,
                                  num_heads=w["heads"], kv_lens=lens, shuffle_pages=True,
                                  formats=(w["kv_format"],), device="cpu")
        q, kvd, qo, kvp, cfg = data
        if shard_mode == "split_kv":                              # Q is replicated: draw it from a rank-independent seed
            q = gen.generate_input(batch, w["q_len"], 1, 4321, num_heads=w["heads"], formats=(), device="cpu")[0]
        h = dict(w=w, q=q, kv=kvd[w["kv_format"]], qo=qo, kv_indptr=kvp, kv_indices=cfg["kv_indices"],
                 sm_scale=cfg["sm_scale"], cfg=cfg, total_kv=cfg["total_kv"], batch=batch)
        h.update(extra)
        return h

    # ------------------------------------------------------------------ reference arm (CPU)
    if args.impl == "reference":
        if rank != 0:
            return
        host = build_host(1234)
        torch.set_num_threads(os.cpu_count() or 1)
        for _ in range(min(max(args.warmup, 1), 2)):
            cpu_oracle_step(host)
        steps = min(args.steps, 20)
        t0 = time.perf_counter()
        for _ in range(steps):
            cpu_oracle_step(host)
        dt = (time.perf_counter() - t0) / steps
        val = tokens_per_call / dt
        abytes = algorithmic_bytes(w, host["total_kv"])
        line = {
            "impl": "reference", "metric": "mla_decode_tokens_per_s", "value": val, "unit": "tokens/s",
            "n_gpus": n_gpus, "steps": steps, "warmup": args.warmup, "ms_per_step": dt * 1e3,
            "us_per_call": dt * 1e6, "achieved_gbs": abytes / dt / 1e9,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
            "config": {"workload": f"{args.workload}: {w['desc']}", "note": "CPU oracle port (torch fp32 "
                       "dequantise-then-attend); the reference's own path needs AMD's aiter and cannot run here; "
                       "each step is one full call, at most 20 steps are timed"},
            "cpu_baseline": {"value": val, "unit": "tokens/s", "cores": torch.get_num_threads(), "kind": "port",
                             "sample": f"{steps} full {args.workload} calls"},
            "e2e": {"value": val, "unit": "tokens/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
            "gpu_launches": 0,
        }
        print(json.dumps(line), flush=True)
        return

    # ------------------------------------------------------------------ our arm (GPU)
    import torch.distributed as dist
    torch.cuda.set_device(local_rank)
    dev = torch.device("cuda", local_rank)
    if world > 1:
        dist.init_process_group("nccl", device_id=dev)
    import amd_optimization_challenge_b200 as pkg

    host = build_host(1234 + rank, rank, world, mode)
    w_rank = dict(w, batch=host["batch"])
    abytes = algorithmic_bytes(w_rank, host["total_kv"])       # this rank's decode launch
    tokens_job = tokens_per_call if mode != "replica" else n_gpus * tokens_per_call
    kv_bytes = sum(t.numel() * t.element_size() for t in host["kv"])
    n_rot = max(2, -(-int(2.4 * L2_BYTES) // kv_bytes))         # rotate > 2.4x L2 worth of cache copies
    n_rot = min(n_rot, 6)

    def to_dev(h):
        cfg = dict(h["cfg"])
        cfg.update(kv_indices=h["kv_indices"].to(dev), kv_format=w["kv_format"], q_format=w["q_format"], impl=args.kernel)
        return (h["q"].to(dev), {w["kv_format"]: tuple(t.to(dev) for t in h["kv"])}, h["qo"].to(dev),
                h["kv_indptr"].to(dev), cfg)

    base = to_dev(host)
    rot = [base]
    for _ in range(n_rot - 1):                                  # same bytes at distinct addresses
        kv = tuple(t.clone() for t in base[1][w["kv_format"]])
        rot.append((base[0], {w["kv_format"]: kv}, base[2], base[3], base[4]))
    torch.cuda.synchronize()

    def barrier():
        if world > 1:
            dist.barrier()
        torch.cuda.synchronize()

    if mode == "split_kv":
        from amd_optimization_challenge_b200.distributed import SplitKVDecoder, cuda_partial_fn
        rows = host["batch"] * w["q_len"]
        decoder = SplitKVDecoder(rows, w["heads"], dev)
        d_off = torch.full((host["batch"],), host["kv_pos_offset"], dtype=torch.int32, device=dev)
        d_tot = torch.full((host["batch"],), host["kv_total_len"], dtype=torch.int32, device=dev)

        def call(data):
            q, kvd, _, kvp, cfg = data
            q_scale = None
            if w["q_format"] == "fp8":
                q, q_scale = pkg.quantize_q_fp8(q)
            return decoder.step(cuda_partial_fn(q, q_scale, w["kv_format"], kvd[w["kv_format"]], kvp,
                                                sm_scale=cfg["sm_scale"], q_len=w["q_len"], kv_indices=cfg["kv_indices"],
                                                kv_pos_offset=d_off, kv_total_len=d_tot, total_kv_hint=host["total_kv"],
                                                impl=args.kernel))
    else:
        call = pkg.custom_kernel

    # ---- launch vehicle: a CUDA graph holding n_rot consecutive steps (one per cache copy), so
    # that the timed region measures the GPU work and not the Python call overhead per step
    for i in range(max(args.warmup, 3)):
        out = call(rot[i % n_rot])
    barrier()
    graph = None
    # the split-KV step contains an NCCL collective: it is launched eagerly (a captured collective has not been
    # validated on this stack), every other mode replays a graph
    if not args.no_graph and mode != "split_kv":
        graph = torch.cuda.CUDAGraph()
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            with torch.cuda.graph(graph, stream=side):
                for i in range(n_rot):
                    out = call(rot[i])
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()

    def run_steps(k):
        if graph is None:
            for i in range(k):
                call(rot[i % n_rot])
            return
        for _ in range(k // n_rot):
            graph.replay()
        for i in range(k % n_rot):
            call(rot[i])

    # ---- clocks are sampled from before the pre-roll (same work, untimed) to after the timed region
    sampler = ClockSampler(local_rank)
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    # The pre-roll and the tail run a FIXED number of steps, the same on every rank (a time-based loop would let
    # the ranks disagree on how many collectives they issue): sized from one probe batch, agreed by a MAX all-reduce.
    t0 = time.perf_counter()
    run_steps(8 * n_rot)
    torch.cuda.synchronize()
    probe = torch.tensor([time.perf_counter() - t0], device=dev)
    if world > 1:
        dist.all_reduce(probe, op=dist.ReduceOp.MAX)
    batch_s = max(float(probe.item()), 1e-4)
    pre_batches = max(1, min(2000, int(0.7 / batch_s)))
    post_batches = max(1, min(700, int(0.25 / batch_s)))
    with sampler:
        for _ in range(pre_batches):
            run_steps(8 * n_rot)
            torch.cuda.synchronize()
        barrier()
        ev0.record()
        run_steps(args.steps)                                   # exactly K steps
        ev1.record()
        barrier()
        ms = ev0.elapsed_time(ev1)
        for _ in range(post_batches):
            run_steps(8 * n_rot)
            torch.cuda.synchronize()
    clocks = sampler.summary()
    if world > 1:
        t = torch.tensor([ms], device=dev)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        ms = float(t.item())
    ms_per_step = ms / args.steps
    value = tokens_job / (ms_per_step * 1e-3)

    # ---- duration of the decode launch (CUDA events recorded by the library around that launch)
    lib = pkg._cabi.lib
    k_ms = []
    pairs = []
    nprof = min(args.steps, 50)
    for i in range(nprof):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(); b.record()                                  # instantiate the handles
        pairs.append((a, b))
    torch.cuda.synchronize()
    torch.cuda._sleep(int(2e7))                                  # ~10 ms of GPU spin: the calls below queue up behind
    for i, (a, b) in enumerate(pairs):                           # it, so no event waits on the host's launch latency
        lib.b200_mla_set_stage1_events(ctypes.c_void_p(a.cuda_event), ctypes.c_void_p(b.cuda_event))
        out = call(rot[i % n_rot])
    lib.b200_mla_set_stage1_events(None, None)
    torch.cuda.synchronize()
    k_ms = [a.elapsed_time(b) for a, b in pairs]
    k_us = statistics.mean(k_ms) * 1e3
    peak, peak_kind = measured_peak_gbs()
    achieved = abytes / (k_us * 1e-6) / 1e9
    hbm = {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s", "frac": achieved / peak,
           "traffic": NCU_TRAFFIC_BYTES.get(args.workload) if mode == "replica" else None,
           "traffic_unit": "bytes per launch (ncu dram read + write, separate capture of this kernel; profiles/)",
           "kernel": "mla_decode (maximum of Q, split-KV decode and merge in one launch)", "kernel_us": k_us,
           "algorithmic_bytes": abytes, "peak_source": f"of {peak_kind}"}
    if mode == "replica":
        # the events around a launch keep it from overlapping with its neighbours, as the launches of the timed steps do
        step = abytes / (ms_per_step * 1e-3) / 1e9
        hbm["step"] = {"us": ms_per_step * 1e3, "achieved": step, "frac": step / peak,
                       "note": "kernel_us stands alone between two events; the timed steps overlap with one another"}
    if w["heads"] >= 128:
        # the H = 128 shape is bound by the tensor pipe, not by HBM: report it against the dense e4m3 rate
        # (twice the measured dense bf16 rate; both operands are e4m3) and keep the HBM view beside it
        flops = 2.0 * w["q_len"] * w["heads"] * host["total_kv"] * (576 + 512)
        tf_peak, tf_kind = measured_peak_tflops()
        tf = flops / (k_us * 1e-6) / 1e12
        roofline = {"bound": "tensor", "achieved": tf, "peak": 2.0 * tf_peak, "unit": "TFLOP/s", "frac": tf / (2.0 * tf_peak),
                    "traffic": hbm["traffic"], "kernel": hbm["kernel"], "kernel_us": k_us, "algorithmic_flops": flops,
                    "peak_source": f"2 x dense bf16 burst, of {tf_kind}", "hbm": hbm}
    else:
        roofline = hbm

    # ---- end to end: host buffers in, host buffer out, every step
    pin = lambda t: t.contiguous().pin_memory()
    h_q, h_kv = pin(host["q"]), tuple(pin(t) for t in host["kv"])
    h_idx, h_ip, h_qo = pin(host["kv_indices"]), pin(host["kv_indptr"]), pin(host["qo"])
    h_out = torch.empty(out.shape, dtype=out.dtype).pin_memory()
    h2d = sum(t.numel() * t.element_size() for t in (h_q, *h_kv, h_idx, h_ip, h_qo))
    d2h = h_out.numel() * h_out.element_size()

    # Two device-side input sets: the copies of step i + 1 run on a copy stream while the kernels of step i run on the
    # compute stream (every step still uploads all of its inputs and reads its output back inside the timed region).
    def dev_set():
        cfg_e = dict(base[4])
        cfg_e["kv_indices"] = torch.empty_like(base[4]["kv_indices"])
        return dict(q=torch.empty_like(base[0]), kv=tuple(torch.empty_like(t) for t in base[1][w["kv_format"]]),
                    ip=torch.empty_like(base[3]), qo=torch.empty_like(base[2]), cfg=cfg_e,
                    ready=torch.cuda.Event(), free=torch.cuda.Event())
    sets = [dev_set(), dev_set()]
    copy_stream = torch.cuda.Stream()

    def stage(s):
        with torch.cuda.stream(copy_stream):
            copy_stream.wait_event(s["free"])                   # the kernels that read this set last have finished
            s["q"].copy_(h_q, non_blocking=True)
            for d, h in zip(s["kv"], h_kv):
                d.copy_(h, non_blocking=True)
            s["cfg"]["kv_indices"].copy_(h_idx, non_blocking=True)
            s["ip"].copy_(h_ip, non_blocking=True); s["qo"].copy_(h_qo, non_blocking=True)
            s["ready"].record(copy_stream)

    def e2e_run(n, start_event=None):
        cur = torch.cuda.current_stream()
        if start_event is not None:
            copy_stream.wait_event(start_event)                 # the first upload starts inside the timed region
        stage(sets[0])
        for k in range(n):
            s = sets[k & 1]
            if k + 1 < n:
                stage(sets[(k + 1) & 1])
            cur.wait_event(s["ready"])
            o = call((s["q"], {w["kv_format"]: s["kv"]}, s["qo"], s["ip"], s["cfg"]))
            h_out.copy_(o, non_blocking=True)
            s["free"].record(cur)

    e_steps = max(3, min(args.steps, 20))
    for st_ in sets:
        st_["free"].record(torch.cuda.current_stream())
    e2e_run(3)
    barrier()
    ev0.record()
    e2e_run(e_steps, ev0)
    ev1.record()
    barrier()
    e_ms = ev0.elapsed_time(ev1) / e_steps
    if world > 1:
        t = torch.tensor([e_ms], device=dev)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        e_ms = float(t.item())
    e2e = {"value": tokens_job / (e_ms * 1e-3), "unit": "tokens/s", "ms_per_step": e_ms,
           "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h,
           "note": "inputs staged from pinned host memory into two device-side sets; the upload of step i+1 overlaps the kernels of step i"}

    # ---- CPU baseline (rank 0, single-GPU runs only)
    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        torch.set_num_threads(os.cpu_count() or 1)
        t_cpu = time_cpu(host, args.cpu_reps)
        cpu = {"value": tokens_per_call / t_cpu, "unit": "tokens/s", "cores": torch.get_num_threads(), "kind": "port",
               "sample": f"median of {args.cpu_reps} full {args.workload} calls ({t_cpu * 1e3:.1f} ms each)",
               "us_per_call": t_cpu * 1e6}

    # the tcgen05 path is one launch (maximum of Q, decode, merge); the warp-level kernel has a combine kernel
    # beside it and, for an FP8-cast Q, an amax kernel; split-KV ranks quantise Q ahead (amax + cast)
    if args.kernel == "generic":
        launches_per_step = 2 + (1 if w["q_format"] == "fp8" else 0)
    else:
        launches_per_step = 1
    if mode == "split_kv" and w["q_format"] == "fp8":
        launches_per_step += 2
    if mode == "split_kv":
        launches_per_step += 1                                        # merge of the gathered partials
    per_gpu = {"replica": "each rank decodes its own batch, no collective",
               "batch_shard": "token-balanced split of the batch over the ranks, no collective",
               "split_kv": "each sequence's keys split over the ranks; (O || LSE) partials exchanged by one NCCL all-gather, then the LSE merge"}[mode]
    sharded = None
    if world > 1 and args.workload == "c1" and not args.no_sharded:
        sharded = sharded_modes(pkg, dist, rank, world, dev, args.kernel)
    if rank == 0:
        line = {
            "metric": "mla_decode_tokens_per_s", "value": value, "unit": "tokens/s", "n_gpus": n_gpus,
            "steps": args.steps, "warmup": max(args.warmup, 3), "ms_per_step": ms_per_step,
            "us_per_call": ms_per_step * 1e3,
            "achieved_gbs": (algorithmic_bytes(w, host.get("global_total_kv", host["total_kv"])) if mode != "replica"
                             else n_gpus * abytes) / (ms_per_step * 1e-3) / 1e9,
            "higher_is_better": True, "scaling": "weak" if mode == "replica" else "strong", "vs_baseline": None,
            "dtype": {"fp8": "e4m3", "mxfp4": "mxfp4(e2m1+e8m0)", "hybrid": "mxfp4+e4m3"}[w["kv_format"]] + " x f32 accumulate",
            "data": "synthetic",
            "config": {"workload": f"{args.workload}: {w['desc']}", "kernel": args.kernel,
                       "launch": "eager custom_kernel calls" if graph is None else f"CUDA graph of {n_rot} custom_kernel steps, replayed",
                       "l2": f"rotating {n_rot} distinct copies of the {kv_bytes / 2**20:.1f} MiB cache (> 2x the 126 MB L2)",
                       "per_gpu": per_gpu},
            "roofline": roofline, "cpu_baseline": cpu, "e2e": e2e, "clocks": clocks,
            "gpu_launches": launches_per_step * args.steps,
        }
        if sharded is not None:
            line["sharded"] = sharded
        print(json.dumps(line), flush=True)
    if world > 1:
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
