#!/usr/bin/env python
"""Benchmarks: edge updates/sec and incremental matches/sec of the per-batch
GPU pipeline, p50/p99 per-batch latency, on one B200.

Headline (the largest single-GPU configuration): R-MAT 4,000,000 vertices /
34,000,000 edges, 32 labels Zipf(1.0), 3,400,000 insertions in batches of
1,000,000, with a 7-vertex tree and a 7-vertex sparse pattern; each pattern
has its own CaLiG index and engine (the plain one-query-per-launch pipeline),
and a step is one batch applied to both (index update + delta lists +
matching per pattern).  Stage 1 (the CaLiG producer that makes the keys)
runs before timing.

  value  keys resident in HBM; step time = sum of the engines' device
         intervals (CUDA events on the engine streams), max over ranks
  e2e    the same batches through the C-ABI call with host buffers
         (cgb_apply_batch: H2D of the keys, compute, D2H of the count)
The stream has 4 batches; steps cycle through them, rebuilding the initial
indexes (untimed) when the cycle restarts, so every cycle sees identical work.

Further workloads ride in the same JSON line under "workloads" (each
guarded: a failure there is reported and leaves the headline intact):
  c2  R-MAT 1M/10M, 16 labels Zipf(1.2), batches of 100,000, 9-vertex dense
      pattern, plain single-query pipeline
  c4  the same stream with 64 registered queries (sizes 4-12; tree, sparse,
      dense; cgbdsm_b200/data/queries_c2.json) in the multi-query engine, one
      launch per batch, against the plain pipeline (CaLiG producer +
      single-query engine per query) on the same batches
  c5  the serving loop (cgbdsm_b200/serve.py) on the R-MAT 4M/34M graph

Usage: python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
                       [--workloads c2,c4,c5] [--quick]
For N > 1 run under torchrun: every rank keeps full index replicas and
applies every batch; the matching of each batch is split by seed group
(rank r expands the groups whose key hashes to r); counts are summed and
step times maxed over ranks (NCCL).  Total work per batch is fixed: scaling
"strong".
"""
from __future__ import annotations

import argparse
import hashlib
import json
import os
import statistics
import subprocess
import sys
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

HEADLINE = ["c3_tree", "c3_sparse"]
L2_FLUSH_BYTES = 256 << 20  # > 126 MB L2
METRIC = "edge updates/sec (and incremental matches/sec, p50/p99 batch latency) on 1 B200"
C3_DESC = ("R-MAT 4,000,000 vertices / 34,000,000 edges, 32 labels Zipf(1.0), 3,400,000 insertions in batches "
           "of 1,000,000, 7-vertex tree and 7-vertex sparse patterns (one engine each)")
C2_DESC = ("R-MAT 1,000,000 vertices / 10,000,000 edges, 16 labels Zipf(1.2), 1,000,000 insertions in batches of "
           "100,000, 9-vertex dense pattern")


def _peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            pk = json.load(f)
        return float(pk["hbm_gbs"]), "measured"
    except Exception:
        return 6650.0, "fallback"


def _engine_source_sha() -> str:
    h = hashlib.sha256()
    for f in ("engine.cu", "multiquery.cuh"):
        with open(os.path.join(ROOT, "cgbdsm_b200", "csrc", f), "rb") as fh:
            h.update(fh.read())
    return h.hexdigest()[:16]


def _profiled(kernel: str, workload: str):
    """Per-launch DRAM bytes and L2 throughput of `kernel` from the committed
    ncu summary profiles/<kernel>_<workload>.md, used only when the summary
    was made from the current kernel sources (its "engine_sha16" line equals
    the sources' hash); else (None, None, reason)."""
    import re

    path = os.path.join(ROOT, "profiles", f"{kernel}_{workload}.md")
    try:
        txt = open(path).read()
    except OSError:
        return None, None, "no ncu summary"
    m = re.search(r"engine_sha16:\s*([0-9a-f]{16})", txt)
    if not m or m.group(1) != _engine_source_sha():
        return None, None, "ncu summary made from other kernel sources"
    t = re.search(r"traffic_bytes_per_launch:\s*(\d+)", txt)
    l2 = re.search(r"l2_throughput_pct:\s*([0-9.]+)", txt)
    return (int(t.group(1)) if t else None), (float(l2.group(1)) if l2 else None), os.path.relpath(path, ROOT)


class ClockSampler:
    """nvidia-smi sampling of SM clocks and throttle reasons during the timed region."""

    def __init__(self, index: int):
        self.index = index
        self.proc = None
        self.path = os.path.join("/tmp", f"cgb_clocks_{os.getpid()}_{index}.csv")

    def __enter__(self):
        q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
             "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
             "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")
        try:
            self.f = open(self.path, "w")
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.index), f"--query-gpu={q}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=self.f, stderr=subprocess.DEVNULL)
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
            self.f.close()

    def summary(self) -> dict:
        rows = []
        try:
            for line in open(self.path):
                t = [x.strip() for x in line.split(",")]
                if len(t) >= 9:
                    rows.append(t)
        except Exception:
            pass
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
        sm = [float(r[1]) for r in rows if r[1].replace(".", "").isdigit()]
        mx = [float(r[2]) for r in rows if r[2].replace(".", "").isdigit()]
        reasons = set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for r in rows:
            for i, n in enumerate(names):
                if r[5 + i].lower() == "active":
                    reasons.add(n)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": sorted(reasons), "samples": len(rows)}


def log(msg: str) -> None:
    print(f"[bench {time.strftime('%H:%M:%S')}] {msg}", file=sys.stderr, flush=True)


def pct(values, p):
    lat = sorted(values)
    return lat[min(len(lat) - 1, int(round(p / 100.0 * (len(lat) - 1))))] if lat else None


# ---------------------------------------------------------------------------
# plain single-query pipeline (CaLiG producer + engine per pattern)
# ---------------------------------------------------------------------------
def produce(spec, rank: int):
    """Stage 1 for every batch: the product's CaLiG producer (keys, vertex counts).
    The workload files are written once, by rank 0, into a directory all
    ranks of the node share; the others wait at a barrier and read them."""
    from cgbdsm_b200 import Producer, dist
    from cgbdsm_b200.workloads import materialize, read_query

    workdir = os.environ.get("CGB_BENCH_DIR", "/tmp/cgb_bench")
    if rank == 0:
        materialize(spec, workdir)
    dist.barrier()
    paths = materialize(spec, workdir)
    t0 = time.perf_counter()
    prod = Producer(paths["query"], paths["data"], paths["update"], spec.cli_batch_size)
    init, dv0 = prod.initial()
    t_init = time.perf_counter() - t0
    batches, s1 = [], []
    for _ in range(prod.num_batches):
        t1 = time.perf_counter()
        batches.append(prod.next())
        s1.append((time.perf_counter() - t1) * 1e3)
    ql, qe = read_query(paths["query"])
    prod.close()
    return {"spec": spec, "paths": paths, "ql": ql, "qe": qe, "init": init, "dv0": dv0, "batches": batches,
            "stage1_init_s": t_init, "stage1_ms": s1}


def run_pipelines(names: list[str], args, rank: int, world: int, local: int, footprint: bool = True) -> dict:
    """Plain pipeline on the patterns `names` (same graph and stream): a step is
    one batch applied to every pattern's engine."""
    import torch

    from cgbdsm_b200 import Engine, dist
    from cgbdsm_b200.engine import FLAG_FOOTPRINT
    from cgbdsm_b200.workloads import SPECS

    t0 = time.perf_counter()
    W = []
    for n in names:
        log(f"stage 1 (CaLiG producer) for {n}")
        W.append(produce(SPECS[n], rank))
    setup_s = time.perf_counter() - t0
    nb = len(W[0]["batches"])
    dev = f"cuda:{local}"

    def new_engine(w, flags=0):
        e = Engine(device=local, dfs_budget_ms=args.budget_ms, shard_index=rank, num_shards=world, flags=flags)
        e.load_query(len(w["ql"]), w["qe"], w["ql"])
        e.build_index(w["init"], w["dv0"])
        return e

    # device-resident keys per pattern and batch: [ins | del | delta]
    dkeys = []
    for w in W:
        row = []
        for b in w["batches"]:
            cat = np.concatenate([b["ins"], b["del"], b["delta"]]).view(np.int64)
            row.append((torch.from_numpy(cat).to(dev), len(b["ins"]), len(b["del"]), len(b["delta"])))
        dkeys.append(row)
    flush = torch.empty(L2_FLUSH_BYTES // 4, dtype=torch.int32, device=dev)
    torch.cuda.synchronize()
    state = {"eng": [new_engine(w) for w in W], "pos": 0}

    def restart():
        for e in state["eng"]:
            e.close()
        state["eng"] = [new_engine(w) for w in W]
        state["pos"] = 0

    def one_step(device_keys: bool):
        if state["pos"] == nb:  # restart the stream: fresh indexes (untimed)
            restart()
        b = state["pos"]
        rec = {"batch": b, "ms": 0.0, "count": 0, "phase": np.zeros(3), "launches": 0, "stats": [], "match_by": []}
        for k, (w, e) in enumerate(zip(W, state["eng"])):
            l0 = e.kernel_launches()
            flush.zero_()  # evict L2 before each engine's batch (outside its timed interval)
            torch.cuda.synchronize()
            if device_keys:
                t, ni, nd, nD = dkeys[k][b]
                base = t.data_ptr()
                c = e.apply_batch_device(w["batches"][b]["dv"], base, ni, base + 8 * ni, nd, base + 8 * (ni + nd), nD)
                ms = float(e.timings()[3])
            else:
                bb = w["batches"][b]
                t1 = time.perf_counter()
                c = e.apply_batch(bb["dv"], bb["ins"], bb["del"], bb["delta"], bb["edge_ok"])
                ms = (time.perf_counter() - t1) * 1e3
            tm = e.timings()
            rec["ms"] += ms
            rec["count"] = (rec["count"] + c) % (1 << 64)
            rec["phase"] += np.array([float(x) for x in tm[:3]])
            rec["match_by"].append(float(tm[2]))
            rec["launches"] += e.kernel_launches() - l0
            rec["stats"].append(e.stats())
        state["pos"] += 1
        log(f"batch {b} ({'device' if device_keys else 'host'} keys): {rec['ms']:.1f} ms, count {rec['count']}, "
            f"phases {[round(x, 2) for x in rec['phase']]}")
        return rec

    for _ in range(args.warmup):
        one_step(True)
    free_b, total_b = torch.cuda.mem_get_info(local)  # after the warm-up: every buffer grown
    device_gb = (total_b - free_b) / 1e9
    log(f"device memory in use: {device_gb:.2f} GB of {total_b / 1e9:.0f} GB")
    dist.barrier()
    torch.cuda.synchronize()
    with ClockSampler(local) as clk:
        recs = [one_step(True) for _ in range(args.steps)]
    torch.cuda.synchronize()
    dist.barrier()
    step_ms = dist.max_values([r["ms"] for r in recs])
    counts = dist.sum_counts([r["count"] for r in recs])
    total_ms = sum(step_ms)
    edges = sum(W[0]["batches"][r["batch"]]["num_edges"] for r in recs)

    restart()
    if args.quick:
        e2e_recs = recs
    else:
        for _ in range(args.warmup):
            one_step(False)
        e2e_recs = [one_step(False) for _ in range(args.steps)]
    e2e_ms = sum(dist.max_values([r["ms"] for r in e2e_recs]))
    e2e_edges = sum(W[0]["batches"][r["batch"]]["num_edges"] for r in e2e_recs)
    h2d = sum(sum(8 * (len(w["batches"][r["batch"]]["ins"]) + len(w["batches"][r["batch"]]["del"])
                       + len(w["batches"][r["batch"]]["delta"])) + len(w["batches"][r["batch"]]["edge_ok"])
                  for w in W) for r in e2e_recs) / len(e2e_recs)

    # roofline: the dominant kernel by device time over the timed steps
    match_ms = sum(r["phase"][2] for r in recs)
    upd_ms = sum(r["phase"][0] for r in recs)
    upd_bytes = sum(st["update_bytes"] for r in recs for st in r["stats"])
    out = {
        "value": edges / (total_ms / 1e3) if total_ms > 0 else 0.0,
        "ms_per_step": total_ms / max(1, len(recs)),
        "matches_per_s": sum(counts) / (total_ms / 1e3) if total_ms > 0 else 0.0,
        "matches_per_batch": sum(counts) / max(1, len(recs)),
        "latency_ms": {"p50": pct(step_ms, 50), "p99": pct(step_ms, 99), "max": max(step_ms)},
        "phase_ms_per_step": {"index_update": upd_ms / len(recs),
                              "delta_lists": sum(r["phase"][1] for r in recs) / len(recs),
                              "matching": match_ms / len(recs)},
        "e2e": {"value": e2e_edges / (e2e_ms / 1e3) if e2e_ms > 0 else 0.0, "unit": "edge updates/s",
                "h2d_bytes_per_step": int(h2d), "d2h_bytes_per_step": 8 * (4 + 16 + 8) * len(W)},
        "gpu_launches": sum(r["launches"] for r in recs),
        "batches_in_stream": nb,
        "patterns": [{"name": w["spec"].name, "query_vertices": len(w["ql"]), "query_edges": len(w["qe"]),
                      "stage1_init_s": round(w["stage1_init_s"], 2),
                      "stage1_ms_per_batch": round(float(np.mean(w["stage1_ms"])), 2)} for w in W],
        "setup_s": round(setup_s, 1),
        "device_memory_gb": round(device_gb, 2),
        "clocks": clk.summary(),
    }
    # the reference's Bottleneck = max(S1, S2) view (main_calig.cpp:435-437):
    # Stage 1 (host producer) of batch b+1 overlaps Stage 2 of batch b
    s1_batch = [sum(w["stage1_ms"][r["batch"]] for w in W) for r in recs]
    bneck_ms = sum(max(a, b) for a, b in zip(s1_batch, step_ms))
    out["with_stage1"] = {"value": edges / (bneck_ms / 1e3) if bneck_ms > 0 else 0.0, "unit": "edge updates/s",
                          "stage1_ms_per_batch": float(np.mean(s1_batch)),
                          "stage2_ms_per_batch": float(np.mean(step_ms)),
                          "view": "sum over batches of max(Stage 1, Stage 2)"}
    peak, peak_kind = _peaks()
    upd_gbs = (upd_bytes / 1e9) / (upd_ms / 1e3) if upd_ms > 0 else 0.0
    if footprint and match_ms >= upd_ms:
        # the dominant launch: the matching of the pattern with the largest
        # matching time; its footprint from one untimed run on batch 0 with the
        # record bit set on (bytes of the distinct records and lists resolved)
        k = int(np.argmax([np.mean([r["match_by"][i] for r in recs]) for i in range(len(W))]))
        w = W[k]
        e = new_engine(w, FLAG_FOOTPRINT)
        t, ni, nd, nD = dkeys[k][0]
        base = t.data_ptr()
        e.apply_batch_device(w["batches"][0]["dv"], base, ni, base + 8 * ni, nd, base + 8 * (ni + nd), nD)
        fp_bytes = e.stats()["match_bytes"]
        e.close()
        fp_ms = float(np.mean([r["match_by"][k] for r in recs if r["batch"] == 0] or
                              [r["match_by"][k] for r in recs]))
        achieved = (fp_bytes / 1e9) / (fp_ms / 1e3) if fp_ms > 0 else 0.0
        kname = "k_dfs_count"
        traffic, l2pct, src = _profiled(kname, w["spec"].name)
        out["roofline"] = {"kernel": f"{kname} (matching, {w['spec'].name})", "bound": "hbm", "achieved": achieved,
                           "peak": peak,
                           "unit": "GB/s", "frac": achieved / peak if peak else None, "peak_source": peak_kind,
                           "algorithmic_bytes": "footprint: 16 B per distinct record resolved + 4 B per entry of "
                                                "its old and delta lists, batch 0",
                           "launch_ms": fp_ms,
                           "algorithmic_bytes_per_launch": fp_bytes, "traffic": traffic, "traffic_source": src,
                           "l2_throughput_pct_ncu": l2pct, "index_update_achieved_gbs": upd_gbs,
                           "index_update_frac": upd_gbs / peak if peak else None}
    else:
        traffic, l2pct, src = _profiled("k_merge", names[0])
        out["roofline"] = {"kernel": "k_merge (index update)", "bound": "hbm",
                           "achieved": upd_gbs, "peak": peak, "unit": "GB/s",
                           "frac": upd_gbs / peak if peak else None, "peak_source": peak_kind,
                           "algorithmic_bytes": "8 B per edit + 4 B per old and new run word + 32 B per record",
                           "algorithmic_bytes_per_step": upd_bytes / len(recs), "traffic": traffic,
                           "traffic_source": src}
    for e in state["eng"]:
        e.close()
    out["_W"] = W
    return out


# ---------------------------------------------------------------------------
# reference CPU path (oracle/_ref): cpu_baseline and the reference arm
# ---------------------------------------------------------------------------
def reference_sample(paths, spec, budget_s: float) -> dict:
    """The reference's own CPU path (oracle/_ref: CaLiG + staging + CPUIndexMirror +
    cpu_dfs) on batch 0 of the stream with all host threads.  Stage 1,
    staging and the index mirror update run fully; the count (the reference
    enumerates every embedding, mask-free seeding) runs for budget_s in a
    supervised child process and is extrapolated by rows counted / rows total.
    When not one row finishes in the budget, the count time is bounded below by
    budget_s x rows_total and the value is an upper bound."""
    from oracle import bind

    threads = os.cpu_count() or 1
    r = bind.supervised_reference_batch(paths["query"], paths["data"], paths["update"], spec.cli_batch_size,
                                        threads, budget_s)
    fixed_ms = r["s1_ms"] + r["staging_ms"] + r["mirror_ms"]
    if r["finished"]:
        count_ms, kind = r["count_ms"], "measured"
    elif r["rows_done"] > 0:
        count_ms, kind = r["count_ms"] * r["rows_total"] / r["rows_done"], "extrapolated"
    else:
        count_ms, kind = r["count_ms"] * max(1, r["rows_total"]), "lower bound (no row finished)"
    return {"batch_ms": fixed_ms + count_ms, "threads": threads, "kind": kind, "r": r, "count_ms": count_ms,
            "spec": spec.name}


def reference_line(names: list[str], budget_s: float, workdir: str) -> dict:
    from cgbdsm_b200.workloads import SPECS, materialize

    parts = []
    for n in names:
        spec = SPECS[n]
        parts.append(reference_sample(materialize(spec, workdir), spec, budget_s))
    spec0 = SPECS[names[0]]
    batch_ms = sum(p["batch_ms"] for p in parts)
    value = spec0.batch_edges / (batch_ms / 1e3) if batch_ms > 0 else 0.0
    sample = "; ".join(
        f"{p['spec']} batch 0: Stage 1 {p['r']['s1_ms']:.0f} ms + staging {p['r']['staging_ms']:.0f} ms + index "
        f"mirror {p['r']['mirror_ms']:.0f} ms measured, mask-free cpu_dfs count {p['r']['rows_done']} of "
        f"{p['r']['rows_total']} seed rows in {p['r']['count_ms'] / 1e3:.1f} s, count time {p['kind']}: "
        f"{p['count_ms'] / 1e3:.3g} s" for p in parts)
    return {"value": value, "unit": "edge updates/s", "cores": parts[0]["threads"], "kind": "reference",
            "sample": sample + ("; value is an upper bound" if any(p["kind"].startswith("lower") for p in parts)
                                else ""),
            "count_time_kind": sorted(set(p["kind"] for p in parts))}


# ---------------------------------------------------------------------------
# extra workloads
# ---------------------------------------------------------------------------
def bench_c2(args, rank, world, local) -> dict:
    r = run_pipelines(["c2"], args, rank, world, local)
    r.pop("_W")
    r["config"] = {"workload": C2_DESC}
    r["unit"] = "edge updates/s"
    return r


def bench_c4(args, rank, world, local) -> dict:
    from cgbdsm_b200 import multiq

    return multiq.bench(args, local, log)


def bench_c5(args, rank, world, local) -> dict:
    from cgbdsm_b200 import serve

    return serve.bench(args, local, log)


def index_layouts(W, local: int) -> dict:
    """The update layouts on the headline's first pattern (R-MAT 4M/34M, 7-vertex
    tree, batches of 1,000,000): per batch, the pool layout's fused merge
    (index update phase of the engine, pending delta + ins - del) against the
    packed-memory array (cgb_gpma_batch_update with the same edits), device
    time of each."""
    import torch

    from cgbdsm_b200 import Engine, Gpma

    w = W[0]
    dev = f"cuda:{local}"
    e = Engine(device=local)
    e.load_query(len(w["ql"]), w["qe"], w["ql"])
    e.build_index(w["init"], w["dv0"])
    gp = Gpma(num_dirs=2 * len(w["qe"]), device=local)
    gp.bulk_load(w["init"])
    pool_ms, gpma_ms, edits = [], [], []
    pending = np.zeros(0, np.uint64)
    for b in w["batches"]:
        e.apply_batch(b["dv"], b["ins"], b["del"], b["delta"], b["edge_ok"])
        pool_ms.append(float(e.timings()[0]))
        ins = np.concatenate([pending, b["ins"]])
        gp.batch_update(ins, b["del"])
        gpma_ms.append(gp.stats()["device_us"] / 1e3)
        edits.append(int(len(ins) + len(b["del"])))
        pending = b["delta"]
    gp.batch_update(pending, np.zeros(0, np.uint64))  # the last batch's delta merge-back (read_index applies it too)
    torch.cuda.synchronize()
    same = bool(np.array_equal(np.sort(e.read_index()), np.sort(np.concatenate(
        [(np.uint64(d) << np.uint64(59)) | gp.extract(d) for d in range(2 * len(w["qe"]))]))))
    e.close()
    gp.close()
    return {"workload": w["spec"].name, "edits_per_batch": edits, "pool_merge_ms": pool_ms, "gpma_update_ms": gpma_ms,
            "gpma_over_pool": float(np.sum(gpma_ms) / max(np.sum(pool_ms), 1e-9)),
            "same_contents_after_stream": same}


def run_ours(args) -> None:
    import torch

    from cgbdsm_b200 import dist

    rank, world, local = dist.env()
    torch.cuda.set_device(local)
    dist.init("nccl", timeout_s=900)
    names = args.headline.split(",")
    head = run_pipelines(names, args, rank, world, local)
    W = head.pop("_W")
    line = {
        "metric": METRIC, "value": head.pop("value"), "unit": "edge updates/s",
        "n_gpus": world, "steps": args.steps, "warmup": args.warmup, "ms_per_step": head.pop("ms_per_step"),
        "higher_is_better": True, "scaling": "strong", "vs_baseline": None,
        "dtype": "u32/u64 integer", "data": "synthetic (seeded R-MAT stand-in for the public graphs)",
        "config": {"workload": C3_DESC if names == HEADLINE else f"{names} (profiling run)",
                   "batch_edges": W[0]["spec"].batch_edges,
                   "batches_in_stream": head.pop("batches_in_stream"), "patterns": head.pop("patterns"),
                   "l2": "flushed before every engine call (256 MiB write); index > 126 MB L2",
                   "parallelism": f"{world} GPU(s): index replicated, seed groups sharded"},
    }
    line.update(head)
    line["stage1_setup_s"] = line.pop("setup_s")
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        from oracle import bind

        if bind.have_ref():
            log("cpu baseline: reference CPU path on batch 0 of each pattern")
            line["cpu_baseline"] = reference_line(names, args.cpu_budget_s,
                                                  os.environ.get("CGB_BENCH_DIR", "/tmp/cgb_bench"))
        else:
            line["cpu_baseline"] = {"unavailable": "oracle/_ref/libcgbref.so was not built (no reference tree)"}
    extras = {}
    if world == 1 and not args.quick:
        try:
            line["index_layouts"] = index_layouts(W, local)
        except Exception as e:
            line["index_layouts"] = {"error": f"{type(e).__name__}: {e}"}
    for name in [w for w in args.workloads.split(",") if w] if world == 1 else []:
        fn = {"c2": bench_c2, "c4": bench_c4, "c5": bench_c5}.get(name)
        if fn is None:
            continue
        log(f"workload {name}")
        try:
            extras[name] = fn(args, rank, world, local)
        except Exception as e:  # reported, the headline stands
            extras[name] = {"error": f"{type(e).__name__}: {e}"}
            log(f"workload {name} failed: {e}")
        torch.cuda.synchronize()
    if extras:
        line["workloads"] = extras
    if rank == 0:
        print(json.dumps(line, default=float), flush=True)
    dist.finish()


def run_reference(args) -> None:
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    from oracle import bind

    if not bind.have_ref():
        print(json.dumps({"impl": "reference", "unavailable": "oracle/_ref/libcgbref.so was not built"}))
        return
    workdir = os.environ.get("CGB_BENCH_DIR", "/tmp/cgb_bench")
    vals, cb = [], None
    per_step_budget = max(2.0, min(args.cpu_budget_s, 150.0 / max(1, args.steps + args.warmup)))
    for i in range(args.warmup + args.steps):
        cb = reference_line(HEADLINE, per_step_budget, workdir)
        if i >= args.warmup:
            vals.append(cb["value"])
    v = statistics.median(vals) if vals else 0.0
    cb["value"] = v
    from cgbdsm_b200.workloads import SPECS

    print(json.dumps({
        "impl": "reference", "metric": METRIC, "value": v, "unit": "edge updates/s", "n_gpus": world,
        "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": (SPECS[HEADLINE[0]].batch_edges / v * 1e3) if v else None, "higher_is_better": True,
        "scaling": "strong", "vs_baseline": None, "dtype": "u32/u64 integer", "data": "synthetic (seeded R-MAT)",
        "config": {"workload": C3_DESC}, "cpu_baseline": cb,
        "e2e": {"value": v, "unit": "edge updates/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }), flush=True)


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=7)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--budget-ms", type=int, default=120000, help="matching time budget per batch")
    ap.add_argument("--cpu-budget-s", type=float, default=8.0)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--workloads", default="c2,c4,c5", help="further workloads in the same JSON line")
    ap.add_argument("--headline", default=",".join(HEADLINE),
                    help="patterns of the timed pipeline (profiling runs use a smaller workload, e.g. c2)")
    ap.add_argument("--quick", action="store_true",
                    help="profiling run: 1 warm-up + 1 step, no e2e leg, no CPU baseline, no further workloads "
                         "(not a benchmark)")
    args = ap.parse_args()
    if args.quick:
        args.steps, args.warmup, args.no_cpu_baseline, args.workloads = 1, 1, True, ""
    elif args.warmup < 3:
        args.warmup = 3
    if args.impl == "reference":
        run_reference(args)
    else:
        run_ours(args)


if __name__ == "__main__":
    main()
