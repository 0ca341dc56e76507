#!/usr/bin/env python
"""SCAN on R-MAT scale 22 (edge factor 16, a/b/c/d = .57/.19/.19/.05, seed 1), eps=0.5, mu=5.

Metric: similarity edges/s -- undirected edges classified (common neighbours counted, eps
tested) and clustered per second.  One step = one full SCAN pass (similarity, predicate,
cores, union-find, attach, hub/outlier) over the graph.

  value     device time, graph resident in HBM (CUDA events on the library's stream)
  e2e       the reference-facing drop-in GPUScan() (scan_gpuscan_compat) from pinned host
            CSR buffers to host labels: H2D, orientation, SCAN, D2H and device allocation
  roofline  the similarity stage's DRAM traffic against the HBM rate, and the words of bitmaps and
            lists that its kernels read (bound by L1 and L2, which supply most of them)
  cpu_baseline  the oracle (a plain OpenMP SCAN: the reference's degree prune, merge or
            binary-search intersection, predicate, union-find, attach, hub/outlier) over the
            whole graph, one pass on every host core
  parity    the last timed step's labels, roles and counters against that oracle pass, and
            the sweep point eps=0.2, mu=2 (cores, clusters, borders, hubs) against another
  sweep     eps in {0.2, 0.4, 0.6, 0.8} x mu in {2, 5, 10} on the same resident graph
  serving / batch   the serving loop and the batched small graphs (their own configs)

  chung_lu  the skewed hub-heavy config (Chung-Lu, exponent 2.1, 50M vertices, ~1.0B
            undirected edges, max degree cap 2M, eps 0.4, mu 5): resident, then streamed
            under a 24 GB device cap, labels compared (--chung-lu-runs resident runs, one
            streamed; --no-chung-lu skips it)
  --chung-lu  only that block, with --steps runs each

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl gb300|reference]
Under torchrun (N > 1) every rank runs an independent replica on its own GPU (the path has
no exchange step); value = all ranks' edges / max-over-ranks time.

--impl reference: GPUSCAN++ has no CPU implementation, so its restatement (the oracle)
runs the same SCAN on the host cores, on the same graph made by the oracle's own generator
(the engine library is not loaded).  The K timed steps are K disjoint edge stripes of one
full pass; the last step adds the predicate and the clustering.  The reference's own GPU
kernels (its cubin, its launch order) are timed on the same graph as a context field.
"""
from __future__ import annotations

import argparse
import gc
import json
import os
import subprocess
import sys
import tempfile
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

WORKLOAD = "rmat-s22-ef16-scan"


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="gb300", choices=["gb300", "reference"])
    ap.add_argument("--scale", type=int, default=22)
    ap.add_argument("--edge-factor", type=int, default=16)
    ap.add_argument("--seed", type=int, default=1)
    ap.add_argument("--eps", default="0.5")
    ap.add_argument("--mu", type=int, default=5)
    ap.add_argument("--predicate", default="ref-f64", choices=["ref-f64", "exact"])
    ap.add_argument("--e2e-steps", type=int, default=20)
    ap.add_argument("--no-cpu-baseline", action="store_true", help="skip the oracle pass (and the parity check)")
    ap.add_argument("--no-reference-kernels", action="store_true",
                    help="with --impl reference: skip the reference's GPU kernels context field")
    ap.add_argument("--no-serving", action="store_true")
    ap.add_argument("--serving-only", action="store_true")
    ap.add_argument("--serving-graphs", type=int, default=64)
    ap.add_argument("--serving-min-scale", type=int, default=12)
    ap.add_argument("--serving-max-scale", type=int, default=24)
    ap.add_argument("--serving-queries", type=int, default=2000)
    ap.add_argument("--no-batch", action="store_true")
    ap.add_argument("--batch-only", action="store_true")
    ap.add_argument("--batch-graphs", type=int, default=4096)
    ap.add_argument("--batch-max-n", type=int, default=100000)
    ap.add_argument("--no-sweep", action="store_true", help="skip the eps x mu sweep on the bench graph")
    ap.add_argument("--no-chung-lu", action="store_true", help="skip the skewed hub-heavy block of the default run")
    ap.add_argument("--chung-lu-runs", type=int, default=2, help="timed runs of the Chung-Lu block in the default run")
    ap.add_argument("--chung-lu", action="store_true",
                    help="instead: the skewed hub-heavy config (Chung-Lu, exponent 2.1, 50M vertices, ~1B edges, "
                         "max degree 2M, eps 0.4, mu 5), resident and streamed under a 24 GB device cap")
    ap.add_argument("--cl-vertices", type=int, default=50_000_000)
    ap.add_argument("--cl-edges", type=int, default=1_100_000_000,
                    help="sampled pairs; about 1.0e9 undirected edges remain after deduplication")
    ap.add_argument("--cl-cap", type=int, default=2_000_000)
    ap.add_argument("--cl-budget-gb", type=float, default=24.0)
    return ap.parse_args()


def dist_env():
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", str(rank)))
    return rank, world, local


class Dist:
    """Barrier and max-reduce across replicas (torch.distributed when WORLD_SIZE > 1)."""

    def __init__(self, world: int, backend: str):
        self.world = world
        self.dist = None
        if world > 1:
            import torch.distributed as dist

            os.environ.setdefault("MASTER_ADDR", "127.0.0.1")
            dist.init_process_group(backend=backend)
            self.dist = dist

    def barrier(self):
        if self.dist:
            self.dist.barrier()

    def max(self, x: float) -> float:
        if not self.dist:
            return x
        import torch

        dev = "cuda" if self.dist.get_backend() == "nccl" else "cpu"
        t = torch.tensor([x], dtype=torch.float64, device=dev)
        self.dist.all_reduce(t, op=self.dist.ReduceOp.MAX)
        return float(t.item())

    def close(self):
        if self.dist:
            self.dist.destroy_process_group()


class ClockSampler:
    """nvidia-smi clocks and throttle reasons, sampled every 50 ms under the timed steps' load.

    The timed steps may be over before the first sample: start() returns once nvidia-smi prints,
    and hold() repeats the step, untimed, until some samples have come in under load."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index: int):
        self.index = index
        self.proc = None
        self.file = None
        self.idle = 0          # samples before the load

    def start(self):
        try:
            self.file = tempfile.NamedTemporaryFile("w+", suffix=".csv", delete=False)
            self.proc = subprocess.Popen(["nvidia-smi", f"--id={self.index}", f"--query-gpu={self.FIELDS}",
                                          "--format=csv,noheader,nounits", "-lms", "50"], stdout=self.file,
                                         stderr=subprocess.DEVNULL)
        except Exception:
            self.proc = None
            return
        limit = time.perf_counter() + 5.0
        while not self.rows() and self.proc.poll() is None and time.perf_counter() < limit:
            time.sleep(0.01)
        self.idle = len(self.rows())

    def rows(self) -> list:
        return [r.split(",") for r in Path(self.file.name).read_text().splitlines() if r.count(",") >= 8]

    def hold(self, step, samples: int = 4, seconds: float = 2.0):
        limit = time.perf_counter() + seconds
        while self.proc and len(self.rows()) < self.idle + samples and time.perf_counter() < limit:
            step()

    def stop(self) -> dict:
        if not self.proc:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        self.proc.wait()
        rows = self.rows()[self.idle:]
        os.unlink(self.file.name)
        sm = [float(r[1]) for r in rows if r[1].strip().replace(".", "").isdigit()]
        mx = [float(r[2]) for r in rows if r[2].strip().replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[i] for r in rows for i in range(4) if r[5 + i].strip().lower() == "active"})
        return {"sm_mhz": float(np.median(sm)) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": reasons, "samples": len(rows)}


def byte_models(off: np.ndarray, adj: np.ndarray, eps: str) -> dict:
    """Algorithmic bytes of one launch of the similarity stage, from the graph alone.

    compulsory: what a run with bitmaps cannot do without but for the bitmaps themselves: each
    edge's endpoints (8 B) and state (1 B), each vertex's rank and degree (8 B).
    prune model: a one-shot run reads only the lists of edges the degree prune leaves at
    this eps (du + 1 >= eps^2 (dv + 1), u the lower endpoint); each such list once (4 du),
    every pivot list staged once (4 d_v), and every edge costs its endpoint, two offsets
    and its count (16 B) plus the zeroing of cn (4 B):  B = 4 sum_counted du + 4 sum_v d_v + 20 E.
    full model: the same with every edge counted (the cached counts of the serving path).
    merge model (what a merge intersection of every edge reads): each edge streams both lists,
      B = sum_e [4 (du + dv) + 16] + 4 E = 4 sum_v d_v^2 + 20 E.
    """
    deg = np.diff(off).astype(np.int64)
    n = deg.size
    src = np.repeat(np.arange(n, dtype=np.int64), deg)
    a = adj.astype(np.int64)
    ds, da = deg[src], deg[a]
    # each undirected edge appears twice; take it at its pivot (the higher endpoint)
    lower = (da < ds) | ((da == ds) & (a < src))
    du, dv = da[lower].astype(np.float64), ds[lower].astype(np.float64)
    E = int(lower.sum())
    e = float(eps)
    counted = ~((du + 1.0) < (dv + 1.0) * e * e)
    staged = 4.0 * float(deg.sum())
    d = deg.astype(np.float64)
    return {"prune": 4.0 * float(du[counted].sum()) + staged + 20.0 * E, "compulsory": 9.0 * E + 8.0 * n,
            "full": 4.0 * float(du.sum()) + staged + 20.0 * E,
            "merge": 4.0 * float((d * d).sum()) + 20.0 * E,
            "counted_edges": int(counted.sum())}


def bench_config(args, n: int, E: int, max_degree: int, world: int) -> dict:
    """The workload, identical in both arms' lines."""
    return {"workload": WORKLOAD, "n": n, "undirected_edges": E, "max_degree": max_degree, "eps": args.eps,
            "mu": args.mu, "predicate": args.predicate, "parallelism": f"replicas{world}",
            "l2": "inputs larger than L2 (adjacency 4*m bytes)"}


STAGE_PROFILE = ROOT / "profiles" / "similarity-stage_rmat-s22.md"


def stage_traffic() -> tuple[float | None, str]:
    """DRAM bytes of one similarity pass on this workload, from the committed ncu summary
    (dram__bytes_read.sum + dram__bytes_write.sum summed over the stage's kernels of one
    pass); None when the summary is absent."""
    import re

    if not STAGE_PROFILE.exists():
        return None, "no ncu summary"
    m = re.search(r"stage_dram_bytes_per_pass\s*=\s*([0-9]+)", STAGE_PROFILE.read_text())
    if not m:
        return None, "no ncu summary"
    return float(m.group(1)), f"{STAGE_PROFILE.relative_to(ROOT)} (ncu, one pass, summed over the stage's kernels)"


def cpu_baseline(off, adj, eps: str, mu: int, mode: int) -> tuple[dict, tuple]:
    """One oracle SCAN pass over the whole graph on every host core: the reference's degree
    prune, intersection, predicate, union-find, attach and hub/outlier.  Returns the
    cpu_baseline record and the oracle's (label, role, counts) for the parity check."""
    from oracle import oracle

    t = time.perf_counter()
    res = oracle.scan_ex(off, adj, eps, mu, mode, prune=True)
    dt = time.perf_counter() - t
    E = int(off[-1]) // 2
    return ({"value": E / dt, "unit": "similarity edges/s", "cores": os.cpu_count(), "kind": "port",
             "sample": f"the whole graph, one pass ({E} edges, eps {eps}, mu {mu}): the reference's degree prune, "
                       f"merge or binary-search intersection, predicate and clustering, OpenMP on "
                       f"{os.cpu_count()} threads, {dt:.1f} s"}, res)


def parity_record(res, want) -> dict:
    """Engine result against the oracle's: labels, roles and every run counter."""
    label, role, counts = want
    st = res.stats
    got = {"cores": st["num_cores"], "clusters": st["num_clusters"], "borders": st["num_borders"],
           "hubs": st["num_hubs"], "outliers": st["num_outliers"], "similar_edges": st["num_similar_edges"],
           "disagreements": st["pred_disagreements"], "multi_borders": st["multi_cluster_borders"]}
    lab_eq = bool(np.array_equal(res.label, label))
    role_eq = bool(np.array_equal(res.role, role))
    return {"oracle_equal": lab_eq and role_eq and got == counts, "labels_equal": lab_eq, "roles_equal": role_eq,
            "counters_equal": got == counts, "labels_differing": int((res.label != label).sum()), "oracle": counts}


def serving_bench(args, device: int) -> dict:
    """Served (graph, eps, mu) queries on a resident pool with cached common-neighbour counts,
    against plain full recompute per query on the same GPU.

    Pool: R-MAT graphs, scales uniform in [min, max] (edge factor 16, seeds 100+i).  Queries:
    graph uniform, eps uniform in {0.1..0.9}, mu uniform in [2, 20], ref-f64.  Poisson
    arrivals at 200 / 2,000 / 20,000 queries/s (native replay), plus a saturated run (every
    query queued at t=0) for the sustainable rate.  Plain recompute: scan_run (similarity +
    cluster stage) per query, one after another, on a sample of the same queries.
    """
    import efficientstructuralgraphclusteringongpus_gb300 as sg

    rng = np.random.default_rng(7)
    scales = rng.integers(args.serving_min_scale, args.serving_max_scale + 1, args.serving_graphs)
    graphs = [sg.Graph.rmat(int(sc), 16, seed=100 + i) for i, sc in enumerate(scales)]
    k = args.serving_queries
    qg = rng.integers(0, len(graphs), k)
    qe = [f"0.{d}" for d in rng.integers(1, 10, k)]
    qm = rng.integers(2, 21, k)
    qp = np.full(k, sg.PRED_REF_F64)
    out = {"pool": f"{len(graphs)} R-MAT graphs, scales {args.serving_min_scale}-{args.serving_max_scale} uniform "
                   f"(edge factor 16), {int(sum(g.num_edges for g in graphs))} undirected edges in total",
           "queries": k, "predicate": "ref-f64", "rates": []}
    with sg.Server(device, 8 << 30, 16) as srv:
        t = time.perf_counter()
        ids = [srv.add_graph(g) for g in graphs]
        out["pool_setup_s"] = time.perf_counter() - t
        gid = [ids[i] for i in qg]
        srv.replay(gid[:200], qe[:200], qm[:200], qp[:200], np.zeros(min(200, k)))   # warm
        for rate in (200, 2000, 20000):
            kk = int(min(k, max(200, rate * 2)))
            arr = np.cumsum(rng.exponential(1000.0 / rate, kk))
            lat, st, wall = srv.replay(gid[:kk], qe[:kk], qm[:kk], qp[:kk], arr)
            ok = st == 0
            out["rates"].append({"offered_qps": rate, "queries": kk, "achieved_qps": kk / (wall / 1e3),
                                 "p50_ms": float(np.percentile(lat[ok], 50)), "p99_ms": float(np.percentile(lat[ok], 99)),
                                 "failed": int((~ok).sum())})
        lat, st, wall = srv.replay(gid, qe, qm, qp, np.zeros(k))
        out["saturated"] = {"queries": k, "qps": k / (wall / 1e3), "p50_ms": float(np.percentile(lat, 50)),
                            "p99_ms": float(np.percentile(lat, 99)), "failed": int((st != 0).sum())}
        out["server_kernel_launches"] = srv.counters()["kernel_launches"]
    # plain full recompute per query, sequential, on a sample of the same queries
    kp = min(k, 200)
    for i in set(int(x) for x in qg[:kp]):
        graphs[i].upload(device)
    graphs[int(qg[0])].run(qe[0], int(qm[0]), sg.PRED_REF_F64, device=device)
    t = time.perf_counter()
    for i in range(kp):
        graphs[int(qg[i])].run(qe[i], int(qm[i]), sg.PRED_REF_F64, device=device)
    plain_s = time.perf_counter() - t
    out["plain_recompute_qps"] = kp / plain_s
    out["speedup_saturated_vs_plain"] = out["saturated"]["qps"] / out["plain_recompute_qps"]
    return out


def batch_bench(args, device: int) -> dict:
    """Many small graphs with their own (eps, mu): one captured pass (scan_batch) against one
    scan_run per graph (each graph resident on the device, cn + cluster stage per run).

    Graphs: stochastic block models, vertex counts log-uniform in [100, max_n], 2-64
    communities, p_in=0.1, p_out=0.001 scaled down to average degree <= 64.  eps uniform in
    {0.3, 0.5, 0.7}, mu uniform in [2, 8], exact predicate.
    """
    import efficientstructuralgraphclusteringongpus_gb300 as sg

    rng = np.random.default_rng(11)
    k = args.batch_graphs
    ns = np.exp(rng.uniform(np.log(100), np.log(args.batch_max_n), k)).astype(int)
    blocks = rng.integers(2, 65, k)
    t = time.perf_counter()
    graphs = [sg.Graph.sbm(int(n), int(min(b, n)), 0.1, 0.001, 64, seed=5000 + i)
              for i, (n, b) in enumerate(zip(ns, blocks))]
    gen_s = time.perf_counter() - t
    eps = [("0.3", "0.5", "0.7")[i] for i in rng.integers(0, 3, k)]
    mus = [int(x) for x in rng.integers(2, 9, k)]
    out = {"graphs": k, "vertices": int(sum(g.n for g in graphs)), "undirected_edges": int(sum(g.num_edges for g in graphs)),
           "n_range": [100, args.batch_max_n], "generate_s": gen_s}
    t = time.perf_counter()
    with sg.Batch(graphs, device, autotune=True) as b:
        out["create_s"] = time.perf_counter() - t
        t = time.perf_counter()
        b.run(eps, mus, sg.PRED_EXACT)                       # tunes the plan, captures the CUDA graph
        out["tune_and_capture_s"] = time.perf_counter() - t
        runs = []
        for _ in range(3):
            labels, _, st = b.run(eps, mus, sg.PRED_EXACT)
            runs.append(st)
    out["batched"] = {"ms_device": float(np.median([r["ms_device"] for r in runs])),
                      "ms_call": float(np.median([r["ms_total"] for r in runs])),
                      "graph_kernels": runs[-1]["graph_kernels"], "long_words": runs[-1]["long_words"],
                      "target_probes": runs[-1]["target_probes"],
                      "tuned_plan": {k: runs[-1][k] for k in ("small_deg", "small_strategy", "hub_min_deg", "chunk_max")}}
    # one scan_run per graph, every graph already resident
    for g in graphs:
        g.upload(device)
    graphs[0].run(eps[0], mus[0], sg.PRED_EXACT, device=device)
    t = time.perf_counter()
    same = True
    for i, g in enumerate(graphs):
        r = g.run(eps[i], mus[i], sg.PRED_EXACT, device=device)
        same &= bool(np.array_equal(r.label, labels[i]))
    per_graph_ms = (time.perf_counter() - t) * 1e3
    out["one_run_per_graph_ms"] = per_graph_ms
    out["speedup_device"] = per_graph_ms / out["batched"]["ms_device"]
    out["speedup_call"] = per_graph_ms / out["batched"]["ms_call"]
    out["identical_to_per_graph_runs"] = same
    for g in graphs:
        g.release_device()
    return out


def reference_arm(args, world: int) -> None:
    """The reference path on the host cores.  GPUSCAN++ has no CPU implementation, so its
    restatement (the oracle) stands in, on the same graph (made by the oracle's generator:
    the engine library is not loaded) and the same eps, mu and predicate.  The K timed steps
    are the K disjoint edge stripes of one full SCAN pass (degree prune and intersection);
    the last one adds the predicate, union-find, attach and hub/outlier over every edge.
    value = E / the K steps' time.  Warm-up steps count stripes of a finer split, untimed.
    Then the reference's own GPU kernels run on the same graph (a context field)."""
    from oracle import oracle

    mode = 1 if args.predicate == "ref-f64" else 0
    off, adj = oracle.rmat(args.scale, args.edge_factor, args.seed)
    deg = np.diff(off)
    E = int(off[-1]) // 2
    sp = oracle.StripedPass(off, adj, args.eps, mode)
    warm = oracle.StripedPass(off, adj, args.eps, mode)
    for w in range(args.warmup):
        warm.count(w, 8 * max(args.steps, args.warmup))
    del warm
    t0 = time.perf_counter()
    for k in range(args.steps):
        sp.count(k, args.steps)
    label, role, counts = sp.finish(args.mu)
    dt = time.perf_counter() - t0
    v = E / dt
    line = {
        "impl": "reference", "metric": "similarity edges/s", "value": v, "unit": "similarity edges/s",
        "n_gpus": world, "steps": args.steps, "warmup": args.warmup, "ms_per_step": dt / args.steps * 1e3,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "u32", "data": "synthetic",
        "config": bench_config(args, off.size - 1, E, int(deg.max()), world),
        "cpu_baseline": {"value": v, "unit": "similarity edges/s", "cores": os.cpu_count(), "kind": "port",
                         "sample": f"one full pass over all {E} edges in {args.steps} edge stripes (one per step): "
                                   f"the reference's degree prune, merge or binary-search intersection, predicate "
                                   f"and clustering, OpenMP on {os.cpu_count()} threads"},
        "e2e": {"value": v, "unit": "similarity edges/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "scan": counts,
        "note": "GPUSCAN++ is GPU-only; its restatement (the oracle) is timed on the host cores",
    }
    if not args.no_reference_kernels:
        line["reference_gpu_kernels"] = reference_kernels(args, off, adj, sp.cn[:E], label)
    print(json.dumps(line))


def reference_kernels(args, off, adj, cn, oracle_label) -> dict:
    """GPUSCAN++'s own kernels (GPUSCAN++/GPUScan.cu compiled unmodified into a cubin) on this
    GPU, replayed by the oracle's harness in GPUScan()'s launch order
    (GPUSCAN++/GPUScan.cu:800-1009), on the bench graph.  kernel_ms = summed kernel time
    (CUDA events); the harness's host-side core/other list compaction between launches is
    outside it.  call_ms = wall time of the whole call (allocation, H2D, kernels, D2H).  The
    host preprocessing GPUScan() expects (getEidAndEdgeList, GPUSCAN++/Graph.cpp:52-141) is
    done once, untimed.  The output is checked against the oracle's counts."""
    from oracle import oracle

    if not oracle.reference_kernels_available():
        return {"unavailable": "the reference's kernel cubin was not built (needs the reference sources)"}
    E = int(off[-1]) // 2
    mode_ok = args.predicate == "ref-f64"
    prep = oracle.reference_gpuscan_prepare(off, adj)
    oracle.reference_gpuscan(off, adj, float(args.eps), args.mu, prepared=prep)   # warm
    ms, walls, out = [], [], None
    for _ in range(3):
        t = time.perf_counter()
        out, k = oracle.reference_gpuscan(off, adj, float(args.eps), args.mu, prepared=prep)
        walls.append((time.perf_counter() - t) * 1e3)
        ms.append(k)
    viol = oracle.check_admissible(off, adj, args.eps, args.mu, 1, out, cn=cn)
    return {"kernel_ms": float(np.mean(ms)), "call_ms": float(np.mean(walls)),
            "edges_per_s": E / (float(np.mean(ms)) / 1e3), "calls": 3,
            "admissible_vs_oracle": mode_ok and viol == {"core": 0, "border": 0, "membership": 0, "hub_rule": 0},
            "violations": viol, "labels_equal_oracle": bool(np.array_equal(out, oracle_label)),
            "note": "reference predicate is ref-f64; a border similar to several clusters may carry any of them"}


def sweep_bench(g, args, mode, device: int) -> list:
    """The eps x mu sweep of the scale-22 config: one warm and two timed one-shot runs each;
    device ms (similarity + cluster stages) and edges/s."""
    out = []
    for eps in ("0.2", "0.4", "0.6", "0.8"):
        for mu in (2, 5, 10):
            g.run(eps, mu, mode, device=device)
            ms = []
            for _ in range(2):
                st = g.run(eps, mu, mode, device=device).stats
                ms.append(st["ms_similarity"] + st["ms_cluster"])
            t = float(np.mean(ms))
            out.append({"eps": eps, "mu": mu, "ms": t, "edges_per_s": g.num_edges / (t / 1e3),
                        "cores": st["num_cores"], "clusters": st["num_clusters"],
                        "similar_edges": st["num_similar_edges"]})
    return out


def chung_lu_bench(args, device: int, runs_resident: int, runs_streamed: int) -> dict:
    """Skewed hub-heavy config: the graph resident in HBM, then streamed (adjacency in pinned
    host memory read over the host link, the rest under a device cap); labels must agree."""
    import efficientstructuralgraphclusteringongpus_gb300 as sg

    mode = sg.PRED_REF_F64 if args.predicate == "ref-f64" else sg.PRED_EXACT
    t = time.perf_counter()
    g = sg.Graph.chung_lu(args.cl_vertices, 2.1, args.cl_edges, args.cl_cap, seed=args.seed)
    gen_s = time.perf_counter() - t
    eps, mu = "0.4", 5
    out = {"workload": f"chung-lu-{args.cl_vertices}v-{args.cl_edges}e-cap{args.cl_cap}", "n": g.n,
           "undirected_edges": g.num_edges, "max_degree": g.max_degree, "eps": eps, "mu": mu,
           "predicate": args.predicate, "generate_s": gen_s}

    def timed(tag, k):
        g.run(eps, mu, mode, device=device)
        runs = [g.run(eps, mu, mode, device=device) for _ in range(max(k, 1))]
        ms = [r.stats["ms_similarity"] + r.stats["ms_cluster"] for r in runs]
        st = runs[-1].stats
        out[tag] = {"ms_per_step": float(np.mean(ms)), "edges_per_s": g.num_edges / (float(np.mean(ms)) / 1e3),
                    "ms_similarity": st["ms_similarity"], "cores": st["num_cores"], "clusters": st["num_clusters"],
                    "similar_edges": st["num_similar_edges"], "device_bytes": g.device_bytes,
                    # each kernel's span on its stream (small pivots, three hash classes, hubs)
                    "ms_cn_kernel": [round(float(x), 3) for x in st["ms_cn_kernel"]],
                    "cn_work_items": [int(x) for x in st["cn_work_items"]], "cn_words": int(st["cn_words"])}
        return runs[-1].label

    t = time.perf_counter()
    g.upload(device)
    out["upload_s"] = time.perf_counter() - t
    lab = timed("resident", runs_resident)
    g.release_device()
    t = time.perf_counter()
    used = g.upload_streamed(device, int(args.cl_budget_gb * (1 << 30)))
    out["streamed_upload_s"] = time.perf_counter() - t
    lab2 = timed("streamed", runs_streamed)
    out["streamed"]["budget_bytes"] = int(args.cl_budget_gb * (1 << 30))
    out["streamed"]["device_bytes_used"] = used
    out["streamed_labels_equal_resident"] = bool(np.array_equal(lab, lab2))
    g.release_device()
    return out


def main():
    args = parse()
    rank, world, local = dist_env()
    if args.impl == "reference":
        if rank == 0:
            reference_arm(args, world)
        return
    import torch

    import efficientstructuralgraphclusteringongpus_gb300 as sg

    torch.cuda.set_device(local)
    dist = Dist(world, "nccl")
    mode = sg.PRED_REF_F64 if args.predicate == "ref-f64" else sg.PRED_EXACT
    if args.chung_lu:
        if rank == 0:
            print(json.dumps({"chung_lu": chung_lu_bench(args, local, args.steps, args.steps)}))
        dist.close()
        return
    if args.serving_only or args.batch_only:
        if rank == 0:
            out = {"serving": serving_bench(args, local)} if args.serving_only else {"batch": batch_bench(args, local)}
            print(json.dumps(out))
        dist.close()
        return

    g = sg.Graph.rmat(args.scale, args.edge_factor, seed=args.seed)
    n, E = g.n, g.num_edges
    off, adj = g.offsets(), g.adjacency()
    g.upload(local)

    # -- device-resident SCAN steps --------------------------------------------------------
    for _ in range(args.warmup):
        g.run(args.eps, args.mu, mode, device=local)
    clocks = ClockSampler(local)
    if rank == 0:
        clocks.start()
    dist.barrier()
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    stats = []
    last_res = None
    for _ in range(args.steps):
        last_res = g.run(args.eps, args.mu, mode, device=local)
        stats.append(last_res.stats)
    torch.cuda.synchronize()
    dist.barrier()
    wall = time.perf_counter() - t0
    clocks.hold(lambda: g.run(args.eps, args.mu, mode, device=local))
    clk = clocks.stop() if rank == 0 else None
    dev_ms = sum(s["ms_similarity"] + s["ms_cluster"] for s in stats)
    dev_ms = dist.max(dev_ms)
    sim_ms = [s["ms_similarity"] for s in stats]
    launches = sum(s["kernel_launches"] for s in stats)
    value = world * E * args.steps / (dev_ms / 1e3)
    last = stats[-1]

    # -- end to end through the drop-in GPUScan with pinned host buffers ----------------------
    off32 = torch.from_numpy(off.astype(np.uint32).view(np.int32)).pin_memory()
    adj32 = torch.from_numpy(adj.view(np.int32)).pin_memory()
    h_off = off32.numpy().view(np.uint32)
    h_adj = adj32.numpy()
    e2e_value, e2e_s, e2e_matches, e2e_step_ms, e2e_cold_ms, e2e_out = None, 0.0, None, [], [], None
    if args.e2e_steps > 0:
        sg.GPUScan(h_off, h_adj, float(args.eps), args.mu)   # warm
        # Python's cyclic collector stays off while the calls are timed, as timeit does: a
        # full collection over torch's and numpy's objects once stalled one call by ~30 ms
        gc.collect()
        gc.disable()
        dist.barrier()
        t = time.perf_counter()
        for _ in range(args.e2e_steps):
            ts = time.perf_counter()
            out = sg.GPUScan(h_off, h_adj, float(args.eps), args.mu)
            e2e_step_ms.append((time.perf_counter() - ts) * 1e3)
        e2e_s = dist.max(time.perf_counter() - t)
        gc.enable()
        e2e_value = world * E * args.e2e_steps / e2e_s
        check = g.run(args.eps, args.mu, sg.PRED_REF_F64, device=local).label
        e2e_matches = bool(np.array_equal(out, check))
        e2e_out = out
        # the same call with an empty device-buffer cache: every call allocates its buffers
        # with cudaMalloc and frees them afterwards (untimed release before each call)
        for _ in range(3):
            sg.release_cached_memory()
            ts = time.perf_counter()
            sg.GPUScan(h_off, h_adj, float(args.eps), args.mu)
            e2e_cold_ms.append((time.perf_counter() - ts) * 1e3)

    # -- roofline of the common-neighbour stage -------------------------------------------
    bm = byte_models(off, adj, args.eps)
    peaks_file = ROOT / "MEASURED_PEAKS.json"
    if peaks_file.exists():
        peak = float(json.loads(peaks_file.read_text())["hbm_gbs"])
        peak_src = "measured"
    else:
        peak, peak_src = 6800.0, "fallback"
    sim_s = float(np.mean(sim_ms)) / 1e3

    def gbs(b):
        return {"achieved": b / sim_s / 1e9, "frac": b / sim_s / 1e9 / peak, "bytes": b}

    words = float(np.mean([s["cn_words"] for s in stats]))
    traffic, traffic_src = stage_traffic() if (args.scale, args.edge_factor, args.seed, args.eps) == (22, 16, 1, "0.5") \
        else (None, "no ncu summary for this configuration")
    compulsory = bm["compulsory"] + g.bitmap_bytes
    hbm_bytes = traffic if traffic else compulsory
    roof = {"bound": "l1/l2", "achieved": hbm_bytes / sim_s / 1e9, "peak": peak, "unit": "GB/s",
            "frac": hbm_bytes / sim_s / 1e9 / peak, "traffic": traffic, "traffic_source": traffic_src,
            "peak_source": peak_src, "bytes": hbm_bytes,
            "bytes_model": "DRAM traffic of the stage (ncu)" if traffic else
                           "9E + 8n + every bitmap once (what DRAM must supply at least)",
            "compulsory_bytes": compulsory, "counted_edges": int(last["cn_edges_counted"]),
            "cache_words": {"words": words, "bytes": 16.0 * words, "gbs": 16.0 * words / sim_s / 1e9,
                            "definition": "16-byte words of bitmaps (the lower endpoints') and lists the kernels report "
                                          "reading; L1 and L2 supply most, so there is no fraction of the HBM rate"},
            "prune_model": dict(gbs(bm["prune"]), counted_edges=bm["counted_edges"],
                                definition="4*sum over edges left by the degree prune of min(du,dv) + 4*sum_v d_v + 20E"),
            "full_model": dict(gbs(bm["full"]), definition="every edge counted (serving cache)"),
            "merge_model": dict(gbs(bm["merge"]), definition="4*sum_v d_v^2 + 20E (both lists per edge)"),
            "kernel_ms": sim_s * 1e3}

    result = None
    if rank == 0:
        cpu, parity = None, None
        if not args.no_cpu_baseline:
            # the oracle pass is the CPU baseline and the checker of the last timed step
            cpu, want = cpu_baseline(off, adj, args.eps, args.mu, mode)
            parity = {"headline": dict(parity_record(last_res, want), eps=args.eps, mu=args.mu)}
            if (args.eps, args.mu) != ("0.2", 2):
                _, want2 = cpu_baseline(off, adj, "0.2", 2, mode)
                parity["sweep_point"] = dict(parity_record(g.run("0.2", 2, mode, device=local), want2),
                                             eps="0.2", mu=2)
            if e2e_out is not None and mode == sg.PRED_REF_F64:
                parity["drop_in_labels_equal_oracle"] = bool(np.array_equal(e2e_out, want[0]))
            parity["oracle_equal"] = all(v["oracle_equal"] for v in parity.values() if isinstance(v, dict)) and \
                parity.get("drop_in_labels_equal_oracle", True)
        sweep = None if args.no_sweep else sweep_bench(g, args, mode, local)
        serving = None if args.no_serving else serving_bench(args, local)
        batch = None if args.no_batch else batch_bench(args, local)
        chung = None if args.no_chung_lu else chung_lu_bench(args, local, args.chung_lu_runs, 1)
        result = {
            "metric": "similarity edges/s", "value": value, "unit": "similarity edges/s", "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": dev_ms / args.steps,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "u32", "data": "synthetic",
            "config": bench_config(args, n, E, g.max_degree, world),
            "e2e": {"value": e2e_value, "unit": "similarity edges/s", "h2d_bytes_per_step": int(4 * (n + 1) + 4 * g.m),
                    "d2h_bytes_per_step": int(4 * n), "api": "GPUScan drop-in (scan_gpuscan_compat)",
                    "ms_per_step": e2e_s / max(args.e2e_steps, 1) * 1e3,
                    "step_ms": [round(x, 3) for x in e2e_step_ms], "labels_match_resident_run": e2e_matches,
                    "cold_cache_step_ms": [round(x, 3) for x in e2e_cold_ms],
                    "python_gc": "collected before the timed calls and disabled during them (as timeit does)",
                    "buffers": "steps reuse the library's cache of freed device buffers (default limit 8 GiB); "
                               "cold_cache_step_ms: the same call after the cache was emptied"},
            "roofline": roof,
            "cpu_baseline": cpu,
            "parity": parity,
            "clocks": clk,
            "gpu_launches": launches,
            "sweep": sweep,
            "serving": serving,
            "batch": batch,
            "chung_lu": chung,
            "stages_ms": {"similarity": float(np.mean(sim_ms)),
                          "cluster": float(np.mean([s["ms_cluster"] for s in stats])),
                          "d2h": float(np.mean([s["ms_d2h"] for s in stats])),
                          "wall_per_step": wall / args.steps * 1e3},
            "scan": {"cores": last["num_cores"], "clusters": last["num_clusters"], "borders": last["num_borders"],
                     "hubs": last["num_hubs"], "outliers": last["num_outliers"],
                     "similar_edges": last["num_similar_edges"],
                     "predicate_disagreements": last["pred_disagreements"]},
        }
        print(json.dumps(result))
    dist.close()


if __name__ == "__main__":
    main()
