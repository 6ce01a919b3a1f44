"""Benchmark of the clique counting path: embeddings/s and time-to-count at k = 4..7.

Workload (one "step"): k-clique counts for k = 4, 5, 6, 7 on the seeded Chung-Lu power-law
graph of the benchmark configuration (18,700 vertices, 198,000 undirected edges, degree
exponent 2.1, max degree 500), each count an exact uint64, from one
dm_count_cliques_upto(kmax = 7) call (one launch walks the clique index to depth 7 and
counts every size on the way). `value` is embeddings/s: the cliques counted per second of
device time per step, with the graph already resident in HBM. `time_to_count_ms` gives
the single-query time of each k (one call per k) beside it. `e2e` is the same metric through the public C ABI with the graph re-uploaded from
host memory every step (device copies released first) and the counts read back.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

With N > 1 (torchrun, one process per GPU) every rank counts its shard of the root tasks
(roots in degree order, dealt round-robin) and the per-rank counts are summed with one
all_reduce; the time is the max over ranks. `--impl reference` times the CPU port of the
reference's plain DFS (OpenMP over roots) on the host cores instead, over the same full
workload per step, reading the graph from the committed edge set.
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import tempfile
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

KS = (4, 5, 6, 7)
WORKLOAD = "chunglu18k"
SEED = 1
FALLBACK_HBM_GBS = 6650.0


def parse_args():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=2000)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--scheduler", choices=["plain", "learned"], default="plain")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-batch", action="store_true", help="skip the batched 256-graph workload")
    return ap.parse_args()


def dist_env():
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return world, rank, local


def measured_peak():
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        try:
            return float(json.loads(p.read_text())["hbm_gbs"]), "measured"
        except Exception:
            pass
    return FALLBACK_HBM_GBS, "fallback"


class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled during the timed region."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index: int):
        self.gpu = gpu_index
        self.proc = None
        self.path = None
        self.out = None

    def __enter__(self):
        fd, self.path = tempfile.mkstemp(prefix="clocks", suffix=".csv")
        os.close(fd)
        try:
            self.out = open(self.path, "w")
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.gpu), f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits",
                 "-lms", "100"], stdout=self.out, stderr=subprocess.DEVNULL)
        except Exception:
            self.proc = None
        time.sleep(0.3)
        return self

    def __exit__(self, *exc):
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                self.proc.kill()
        if self.out is not None:
            self.out.close()

    def summary(self):
        if not self.path or not os.path.exists(self.path):
            return None
        sm, mx, reasons = [], None, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in open(self.path):
            parts = [x.strip() for x in line.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                mx = float(parts[2])
            except ValueError:
                continue
            for nm, flag in zip(names, parts[5:9]):
                if flag.lower() in ("active", "1", "yes"):
                    reasons.add(nm)
        os.unlink(self.path)
        if not sm:
            return None
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": mx, "reasons": sorted(reasons), "samples": len(sm)}


def cpu_baseline(u, v):
    """The oracle's OpenMP port of the reference's plain DFS, timed on this host's cores over
    the full workload (every root, k = 4..7)."""
    import oracle as orc

    og = orc.OracleGraph.from_pairs(u, v)
    threads = os.cpu_count() or 1
    t0 = time.perf_counter()
    total = sum(orc.clique_dfs(og, k, threads=threads) for k in KS)
    dt = time.perf_counter() - t0
    return {"value": total / dt, "unit": "embeddings/s", "cores": threads, "kind": "port",
            "sample": f"full workload: all {og.n} roots, k = 4..7, OpenMP dynamic schedule over roots"}


REF_STEP_BUDGET = 300  # warm-up + timed steps that each run the whole workload


def run_reference(args):
    """The reference's plain DFS (the oracle's OpenMP port of clique_DM_DFS, one dynamic
    task per root) on all host cores, rank 0 only. The graph is read from the committed
    edge set of the same workload, so this process loads no library of this package. One
    step = every root, k = 4..7: the same work as the GPU arm's step. When warm-up + timed
    steps exceed REF_STEP_BUDGET, each step runs one stratum of a seeded random partition
    of the roots instead (strata rotate), which keeps the run within minutes at the same
    per-embedding cost."""
    world, rank, _ = dist_env()
    if rank != 0:
        return 0
    import numpy as np

    import oracle as orc

    z = np.load(ROOT / "tests" / "golden" / f"{WORKLOAD}_s{SEED}.npz")
    og = orc.OracleGraph.from_pairs(z["u"], z["v"])
    threads = os.cpu_count() or 1
    n = og.n
    n_steps = args.warmup + args.steps
    strata = max(1, -(-n_steps // REF_STEP_BUDGET))
    perm = np.random.default_rng(SEED).permutation(n).astype(np.int32)
    parts = [np.sort(perm[s::strata]) for s in range(strata)]
    times, counts = [], []
    for i in range(n_steps):
        t0 = time.perf_counter()
        if strata == 1:
            c = sum(orc.clique_dfs(og, k, threads=threads) for k in KS)
        else:
            c = sum(orc.clique_dfs_roots(og, k, parts[i % strata], threads) for k in KS)
        dt = time.perf_counter() - t0
        if i >= args.warmup:
            times.append(dt)
            counts.append(c)
    value = sum(counts) / sum(times)
    sample = (f"full workload per step: all {n} roots, k = 4..7" if strata == 1 else
              f"1/{strata} of the roots per step (seeded random strata, rotating), k = 4..7") + \
        ", OpenMP dynamic schedule over roots"
    line = {
        "impl": "reference", "metric": "embeddings/s", "value": value, "unit": "embeddings/s",
        "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": 1e3 * sum(times) / len(times), "higher_is_better": True, "scaling": "strong",
        "vs_baseline": None, "dtype": "int64", "data": "synthetic (seeded Chung-Lu power-law graph)",
        "config": {"workload": f"{WORKLOAD} k-cliques k=4..7", "vertices": int(n), "edges": int(og.m),
                   "seed": SEED},
        "cpu_baseline": {"value": value, "unit": "embeddings/s", "cores": threads, "kind": "port",
                         "sample": sample},
        "e2e": {"value": value, "unit": "embeddings/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)
    return 0


LVP_WORKLOADS = ("rmat100k", "rmat317k")
LVP_KS = (6, 7)


def learned_vs_plain(dm, workloads, reps: int = 5):
    """Time-to-count of the learned scheduler against plain device balancing on the skewed
    R-MAT workloads (k = 6, 7). Per workload the predictor is trained on subtree sizes logged
    by the plain engine on two other seeds of the same configuration. Every learned call
    runs its schedule on the device (features, inference, bucketed longest-first order,
    splits) and that time is part of its time-to-count (prep_ms, also reported alone)."""
    import numpy as np

    out = {}
    for wl in LVP_WORKLOADS:
        t0 = time.perf_counter()
        Xs, Ts = [], []
        for s in (2, 3):
            g2 = workloads.make(wl, s)
            for k in (4, 5, 6, 7):
                X, T, m = dm.subtree_log(g2, k)
                Xs.append(X[m])
                Ts.append(T[m])
        pr = dm.Predictor(seed=1)
        loss = pr.train(np.concatenate(Xs), np.concatenate(Ts), epochs=40, batch=512, lr=3e-3)
        train_s = time.perf_counter() - t0
        g = workloads.make(wl, SEED)
        res_wl = {"workload": f"{wl} k-cliques", "train_seeds": [2, 3], "test_seed": SEED, "train_loss": loss,
                  "train_s": train_s, "by_k": {}}
        for k in LVP_KS:
            X, T, m = dm.subtree_log(g, k)
            mae = float(np.mean(np.abs(pr.predict(X[m]) - T[m])))
            res = {}
            for name, opts in (("plain", dm.Options()),
                               ("learned", dm.Options(scheduler=dm.SCHED_LEARNED, predictor=pr.handle))):
                tot, kern, prep, idle, cnt = [], [], [], [], None
                dm.count_cliques(g, k, opts)  # warm-up: graph upload, index build
                for _ in range(reps):
                    c, st = dm.count_cliques(g, k, opts)
                    tot.append(st.kernel_ms + st.prep_ms)
                    kern.append(st.kernel_ms)
                    prep.append(st.prep_ms)
                    idle.append(st.idle_warp_fraction)
                    cnt = c
                res[name] = {"time_to_count_ms": statistics.median(tot), "kernel_ms": statistics.median(kern),
                             "schedule_ms": statistics.median(prep),
                             "idle_warp_fraction": statistics.median(idle), "count": cnt}
            assert res["plain"]["count"] == res["learned"]["count"]
            res["speedup"] = res["plain"]["time_to_count_ms"] / res["learned"]["time_to_count_ms"]
            res["mae_log_subtree"] = mae
            res_wl["by_k"][str(k)] = res
        out[wl] = res_wl
    return out


MOTIF_RUNS = (("chunglu18k", 3), ("chunglu18k", 4), ("rmat100k", 3))


def motifs(dm, workloads, peak, reps: int = 5):
    """Motif counting (connected induced k-subgraphs per class, self-generated dictionaries)
    on the benchmark graphs: count, device time-to-count (median over reps, graph resident),
    embeddings/s and the roofline of the motif kernel against the motif work model (the
    reference's extension unions and per-leaf adjacency probes; this engine counts leaves in
    bulk from adjacency masks, so it can move fewer bytes than the model charges)."""
    out = {}
    for wl, k in MOTIF_RUNS:
        g = workloads.make(wl, SEED)
        d = dm.Dictionary.generate(k)
        dm.count_motifs(g, k, d)  # warm-up: upload
        ms, tot = [], None
        for _ in range(reps):
            h, st = dm.count_motifs(g, k, d)
            ms.append(st.kernel_ms)
            tot = int(h.sum())
        t = statistics.median(ms)
        _, alg = dm.motif_work_model(g, k)
        ach = alg / (t * 1e-3) / 1e9
        # whole graphs of k = 3, 4 are counted from a census, which does not do the model's work: its
        # bytes over that time are no bandwidth
        census = st.mode_used == dm.MODE_BITMAP
        out[f"{wl}_k{k}"] = {"count": tot, "classes": int(d.n_classes), "time_to_count_ms": t,
                             "embeddings_per_s": tot / (t * 1e-3), "algorithmic_bytes": alg,
                             "path": "census" if census else "enumeration",
                             "roofline": None if census else {"bound": "hbm", "achieved": ach, "peak": peak,
                                                              "unit": "GB/s", "frac": ach / peak}}
    return out


def batched(dm, workloads, reps: int = 2):
    """The batched workload (256 Chung-Lu graphs of uneven size, one query each from k-cliques
    k = 3..6 and motifs k = 3..5) in one persistent, CUDA-graph-captured launch, autotuned by
    the cost model. Reports the replay's device time and wall time (host replay + read-back)."""
    t0 = time.perf_counter()
    queries, _graphs, _dicts = workloads.make_batch(seed=SEED, n_graphs=256)
    gen_s = time.perf_counter() - t0
    t0 = time.perf_counter()
    b = dm.Batch(queries)
    create_s = time.perf_counter() - t0
    res, st = b.run()  # warm-up replay
    ks, walls, idle, don = [], [], [], []
    for _ in range(reps):
        t0 = time.perf_counter()
        res, st = b.run()
        walls.append(1e3 * (time.perf_counter() - t0))
        ks.append(st.kernel_ms)
        idle.append(st.idle_warp_fraction)
        don.append(st.donations)
    total = sum(int(r) if isinstance(r, int) else int(r.sum()) for r in res)
    mix = {}
    for q in queries:
        key = f"{'clique' if q.kind == dm.QUERY_CLIQUE else 'motif'}{q.k}"
        mix[key] = mix.get(key, 0) + 1
    vw = {}
    for i in range(len(queries)):
        t = b.tuning(i)
        vw[str(t.vwarp)] = vw.get(str(t.vwarp), 0) + 1
    b.close()
    kms = statistics.median(ks)
    return {"workload": "256 seeded Chung-Lu graphs, V~U[50,5000], avg degree~U[4,40], gamma~U[2.0,2.5]",
            "queries": mix, "vertices": sum(q.graph.info().n_vertices for q in queries),
            "edges": sum(q.graph.info().n_edges for q in queries), "subgraphs": total,
            "kernel_ms": kms, "wall_ms": statistics.median(walls), "embeddings_per_s": total / (kms * 1e-3),
            "launches_per_run": 1, "cuda_graph": True, "autotune": "cost model", "vwarp_chosen": vw,
            "idle_warp_fraction": statistics.median(idle), "donations": int(statistics.median(don)),
            "generate_s": gen_s, "create_s": create_s}


def e2e_upload_bytes(g) -> int:
    """Bytes one e2e step copies host -> device for a clique count on the index: the graph's
    clique image in one copy - the oriented CSR (n row starts, n degrees, rows padded to
    multiples of 4 ints), the descending-degree root order (n ints), the index block offsets
    (n ints) and the task list (16 bytes per entry: one per root, split_parts(d) for roots of
    20..64 out-neighbours), each rounded up to 256 bytes, as engine.cu lays it out - and the
    1,152-byte counter block. The DAG orients every edge from the lower to the higher
    (degree, id) rank."""
    u, v = g.edges()
    n = g.info().n_vertices
    deg = np.bincount(np.concatenate([u, v]), minlength=n)
    rank = np.empty(n, np.int64)
    rank[np.lexsort((np.arange(n), deg))] = np.arange(n)
    lo = np.where(rank[u] < rank[v], u, v)
    od = np.bincount(lo, minlength=n)
    padded = max(int(((od + 3) // 4 * 4).sum()), 4)
    split = (od >= 20) & (od <= 64)
    parts = int(np.where(split, np.maximum(1, (od * od + 128) // 256), 1).sum())
    nn = max(n, 1)
    sizes = [4 * nn, 4 * nn, 4 * padded, 4 * nn, 4 * nn, max(16 * parts, 16)]
    return sum((b + 255) // 256 * 256 for b in sizes) + 1152


def main():
    args = parse_args()
    if args.impl == "reference":
        return run_reference(args)
    import torch

    world, rank, local = dist_env()
    torch.cuda.set_device(local)
    if world > 1:
        from datetime import timedelta

        import torch.distributed as tdist

        tdist.init_process_group("nccl", timeout=timedelta(seconds=120))
    import dumato_b200 as dm
    from dumato_b200 import workloads

    g = workloads.make(WORKLOAD, SEED)
    info = g.info()
    stream = torch.cuda.current_stream()
    sched = dm.SCHED_PLAIN if args.scheduler == "plain" else dm.SCHED_LEARNED
    opts = dm.Options(device=local, stream=stream.cuda_stream, rank=rank, world_size=world, scheduler=sched)
    flush = torch.empty(256 * 1024 * 1024 // 4, dtype=torch.int32, device="cuda")

    def step(collect=None):
        # one call, one launch: the walk to depth 7 counts every smaller clique on the way
        counts, st = dm.count_cliques_upto(g, max(KS), opts)
        if collect is not None:
            collect.append((counts, st))
        return sum(counts[k] for k in KS), st.kernel_launches

    def barrier():
        torch.cuda.synchronize()
        if world > 1:
            torch.distributed.barrier()
            torch.cuda.synchronize()

    for _ in range(args.warmup):
        step()
    # timed: device events around each step on the launching stream; L2 flushed before
    # each step, outside the events
    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(args.steps)]
    fused_ms = []
    fused_idle = []
    emb = 0
    launches = 0
    barrier()
    with ClockSampler(local) as clocks:
        for i in range(args.steps):
            flush.zero_()
            ev[i][0].record(stream)
            coll = []
            c, nl = step(coll)
            ev[i][1].record(stream)
            emb += c
            launches += nl
            fused_ms.append(coll[0][1].kernel_ms)
            fused_idle.append(coll[0][1].idle_warp_fraction)
        barrier()
    t_total = sum(a.elapsed_time(b) for a, b in ev) / 1e3
    if world > 1:
        t = torch.tensor([t_total], dtype=torch.float64, device="cuda")
        torch.distributed.all_reduce(t, op=torch.distributed.ReduceOp.MAX)
        t_total = float(t.item())
        e = torch.tensor([emb], dtype=torch.int64, device="cuda")
        torch.distributed.all_reduce(e)
        emb = int(e.item())
    value = emb / t_total

    # e2e: graph uploaded from host memory each step, counts read back, through the C ABI
    e2e_steps = max(3, min(args.steps, 50))
    e2e_emb = 0
    e2e_ms = 0.0
    barrier()
    t0 = torch.cuda.Event(enable_timing=True)
    t1 = torch.cuda.Event(enable_timing=True)
    upload_ms = []
    for _ in range(e2e_steps):
        g.release_device()
        flush.zero_()
        t0.record(stream)
        coll = []
        c, _ = step(coll)
        t1.record(stream)
        t1.synchronize()
        e2e_ms += t0.elapsed_time(t1)
        e2e_emb += c
        upload_ms.append(coll[0][1].prep_ms)  # the call uploads the graph and builds the index
    n, m = info.n_vertices, info.n_edges
    # padded oriented CSR (row starts, degrees, adjacency padded to 4-int rows), the root
    # order, the clique index's block offsets and task list (the index itself is built on
    # the device), and the per-call counter block; the counter block is read back per call
    h2d = e2e_upload_bytes(g)
    d2h = 1152
    e2e_t = e2e_ms / 1e3
    if world > 1:
        t = torch.tensor([e2e_t], dtype=torch.float64, device="cuda")
        torch.distributed.all_reduce(t, op=torch.distributed.ReduceOp.MAX)
        e2e_t = float(t.item())
        e = torch.tensor([e2e_emb], dtype=torch.int64, device="cuda")
        torch.distributed.all_reduce(e)
        e2e_emb = int(e.item())
    e2e_value = e2e_emb / e2e_t

    # single-query time-to-count per k (one call per k, graph resident), outside the timed region
    per_k = {k: [] for k in KS}
    for _ in range(max(3, min(args.steps, 20))):
        for k in KS:
            flush.zero_()
            per_k[k].append(dm.count_cliques(g, k, opts)[1].kernel_ms)

    # roofline of the fused launch: the walk to depth 7 expands exactly the DFS nodes of the
    # k = 7 work model (no pruning by set size), so its algorithmic bytes are that model's
    peak, peak_kind = measured_peak()
    alg_bytes = dm.clique_work_model(g, max(KS))[1] / max(world, 1)
    kern_s = statistics.mean(fused_ms) / 1e3
    achieved = alg_bytes / kern_s / 1e9
    # DRAM bytes per launch from the committed ncu capture of this kernel and workload
    traffic = None
    l2 = None
    prof = ROOT / "profiles" / "clique_chunglu18k_traffic.json"
    if prof.exists():
        try:
            pj = json.loads(prof.read_text())
            traffic = pj.get("dram_bytes_per_launch")
            l2 = pj.get("l2")
        except Exception:
            traffic = None

    cpu = None
    lvp = None
    bat = None
    mot = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        u, v = g.edges()
        cpu = cpu_baseline(u, v)
        lvp = learned_vs_plain(dm, workloads)
    if rank == 0 and world == 1 and not args.no_batch:
        mot = motifs(dm, workloads, peak)
        bat = batched(dm, workloads)

    if rank == 0:
        line = {
            "metric": "embeddings/s", "value": value, "unit": "embeddings/s", "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1e3 * t_total / args.steps,
            "higher_is_better": True, "scaling": "strong", "vs_baseline": None, "dtype": "int64",
            "data": "synthetic (seeded Chung-Lu power-law graph)",
            "config": {"workload": f"{WORKLOAD} k-cliques k=4..7", "vertices": n, "edges": m,
                       "max_degree": info.max_degree, "max_out_degree": info.max_out_degree, "seed": SEED,
                       "scheduler": args.scheduler, "parallelism": f"root shards x{world}",
                       "step": "one dm_count_cliques_upto(kmax=7) call: one launch counts k = 4..7",
                       "l2": "flushed before every step (256 MB write)"},
            "fused_time_to_count_ms": statistics.mean(fused_ms),
            # the persistent launch's makespan is its duration; idle = warp time spent waiting
            "load_balance": {"makespan_ms": statistics.mean(fused_ms),
                             "idle_warp_fraction": statistics.mean(fused_idle)},
            "time_to_count_ms": {str(k): statistics.mean(per_k[k]) for k in KS},
            "embeddings_per_step": emb // max(args.steps, 1),
            "gpu_launches": launches,
            "roofline": {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s",
                         "frac": achieved / peak, "traffic": traffic, "peak_source": peak_kind,
                         "algorithmic_bytes_per_launch": alg_bytes, "l2": l2,
                         "kernel": "clique_cached_kernel<7, 1, TMA, fused> (one launch per step)"},
            "e2e": {"value": e2e_value, "unit": "embeddings/s", "h2d_bytes_per_step": h2d,
                    "d2h_bytes_per_step": d2h, "steps": e2e_steps,
                    "upload_and_index_ms": statistics.median(upload_ms)},
            "cpu_baseline": cpu,
            "learned_vs_plain": lvp,
            "motifs": mot,
            "batched": bat,
            "clocks": clocks.summary(),
        }
        print(json.dumps(line), flush=True)
    if world > 1:
        torch.distributed.barrier()
        torch.distributed.destroy_process_group()
    return 0


if __name__ == "__main__":
    sys.exit(main())
