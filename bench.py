#!/usr/bin/env python
"""Index-build benchmark: 1M x 128 (SIFT-like mixture), GNN-Descent k=96 with
10 iterations, then the CFS 'path'/'dist' prune (NSG rule) to degree 32, m=64.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

One step builds the whole index once. `value` is seconds per build with the
FP32 base already resident in HBM (timed with CUDA events on the stream the
library launches on, max over ranks); `e2e` is the same build through the C
ABI from host memory to host memory (H2D of the base and D2H of the pruned
rows inside the timed region). Under torchrun every rank builds its own
replica (weak scaling). `--impl reference` times the CPU implementation of the
path (the oracle port: OpenMP NN-Descent + path prune) on a bounded sample.
"""
import argparse
import ctypes as C
import json
import os
import statistics
import sys
import threading
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

import numpy as np  # noqa: E402

METRIC = "1M×128 index build s (GNN-Descent+prune), chosen vs plain FP32 @ equal recall"
K, ITERS, FD, TOPM, THRE = 96, 10, 32, 64, 1.0


def args_():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=3)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--n", type=int, default=1_000_000)
    # 160K points scaled by 6.25 predicts the full 1M run within 1 %; 40K
    # scaled by 25 came out 11 % low (profiles/cpu_baseline_scaling.md)
    ap.add_argument("--cpu-sample", type=int, default=160_000)
    ap.add_argument("--skip-plain", action="store_true")
    ap.add_argument("--skip-e2e", action="store_true")
    ap.add_argument("--skip-cpu", action="store_true")
    ap.add_argument("--skip-recall", action="store_true")
    ap.add_argument("--skip-prunes", action="store_true")
    return ap.parse_args()


def peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            return json.load(f)["hbm_gbs"], "measured"
    except Exception:
        return 6650.0, "fallback"


def tensor_peak():
    """Dense bf16/fp16 tensor peak (TFLOP/s), burst figure: the join is timed alone per launch."""
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            return json.load(f)["bf16_tflops"]
    except Exception:
        return 1590.0


# What limits each kernel, from its ncu captures (profiles/): the roofline
# class stays the HBM roofline of a gather kernel, this names the binding.
BINDING = {
    "prune_select_path": "instruction fetch (no_instruction), then dependent L2-hit row gathers "
                         "(long_scoreboard); DRAM traffic well below the HBM roofline",
    "prune_filter": "gathers of the candidates' rows through L1 (long_scoreboard) and issue; "
                    "mma.sync tiles at a seventh of the tensor pipe",
    "knn_join_tc": "latency and barriers: per-tile TMA gathers from L2 and the consumer "
                   "barriers; tensor pipe lightly used",
    "knn_merge": "latency: dependent pool loads and global atomics per node",
}


class Clocks:
    """Samples SM clock and throttle reasons every 200 ms (read-only NVML)."""

    BITS = {0x4: "sw_power_cap", 0x8: "hw_slowdown", 0x20: "sw_thermal_slowdown",
            0x40: "hw_thermal_slowdown", 0x80: "hw_power_brake_slowdown"}

    def __init__(self, index):
        self.samples, self.reasons, self.stop_ev = [], set(), threading.Event()
        self.max_mhz = None
        try:
            import pynvml
            pynvml.nvmlInit()
            self.nv = pynvml
            self.h = pynvml.nvmlDeviceGetHandleByIndex(index)
            self.max_mhz = pynvml.nvmlDeviceGetMaxClockInfo(self.h, pynvml.NVML_CLOCK_SM)
        except Exception:
            self.nv = None

    def _run(self):
        while not self.stop_ev.is_set():
            try:
                self.samples.append(self.nv.nvmlDeviceGetClockInfo(self.h, self.nv.NVML_CLOCK_SM))
                r = self.nv.nvmlDeviceGetCurrentClocksEventReasons(self.h)
                for bit, name in self.BITS.items():
                    if r & bit:
                        self.reasons.add(name)
            except Exception:
                pass
            self.stop_ev.wait(0.2)

    def __enter__(self):
        if self.nv:
            self.t = threading.Thread(target=self._run, daemon=True)
            self.t.start()
        return self

    def __exit__(self, *a):
        if self.nv:
            self.stop_ev.set()
            self.t.join()

    def summary(self):
        med = statistics.median(self.samples) if self.samples else None
        return {"sm_mhz": med, "sm_max_mhz": self.max_mhz, "reasons": sorted(self.reasons),
                "samples": len(self.samples)}


def stage_stats(capi):
    L = capi.lib()
    arr = (capi.StageStat * 32)()
    cnt = C.c_int(0)
    capi.check(L.tagore_stage_stats(arr, 32, C.byref(cnt)))
    return {arr[i].name.decode(): (arr[i].ms, arr[i].launches, arr[i].bytes, arr[i].items)
            for i in range(min(cnt.value, 32))}


def recall_knn(g, half_t, samp, k=10, batch=2000):
    """kNN recall@k of rows g on the sampled nodes against brute force over the
    FP16 base, in batches of sampled nodes."""
    import torch
    x = half_t.float()
    xx = (x * x).sum(1)
    hits = 0
    for b in range(0, len(samp), batch):
        sb = samp[b:b + batch]
        q = x[sb]
        d2 = (q * q).sum(1, keepdim=True) + xx[None] - 2.0 * (q @ x.T)
        d2[torch.arange(len(sb)), torch.as_tensor(sb, device=x.device)] = float("inf")
        truth = torch.topk(d2, k, largest=False).indices.cpu().numpy()
        hits += sum(len(set(g[s, :k].tolist()) & set(truth[i].tolist())) for i, s in enumerate(sb))
        del d2
    return hits / (k * len(samp))


def index_recall(rows, ep, base, queries, half_t, k=10, L=128, seed=0x5EED):
    """recall@10 of the library's GPU greedy search (tagore_search) over the
    pruned rows: NSG's search with pool L, the entry point's neighbours plus
    seeded random starts."""
    import torch
    from tagore_b200 import capi
    dev = half_t.device
    offs, adj = capi.rows_to_csr(rows)
    xb = torch.as_tensor(np.ascontiguousarray(base, np.float32), device=dev)
    xq = torch.as_tensor(np.ascontiguousarray(queries, np.float32), device=dev)
    found = capi.search(xb, torch.as_tensor(offs.astype(np.int64), device=dev),
                        torch.as_tensor(adj.view(np.int32), device=dev), ep, xq, L, k,
                        seed).cpu().numpy()
    d2 = (xq * xq).sum(1, keepdim=True) + (xb * xb).sum(1)[None] - 2.0 * (xq @ xb.T)
    truth = torch.topk(d2, k, largest=False).indices.cpu().numpy()
    return float(np.mean([len(set(found[i].tolist()) & set(truth[i].tolist())) / k
                          for i in range(len(queries))]))


def cpu_baseline(base, n_total, sample):
    """Oracle port (OpenMP NN-Descent + path prune) on the first `sample`
    points; seconds scaled to the full base by n_total / sample."""
    from oracle import oracle as orc
    xs = np.ascontiguousarray(base[:sample])
    half, center, factor = orc.host_prep(xs)
    t0 = time.perf_counter()
    ids, _ = orc.nndescent(half.astype(np.float32), K, ITERS)
    dis = orc.dist_pairs(half, np.repeat(np.arange(sample, dtype=np.uint32), K), ids.reshape(-1))
    dis = dis.reshape(sample, K)
    order = np.argsort(dis, axis=1, kind="stable")
    buf = orc.Buffers(np.take_along_axis(ids, order, 1), np.take_along_axis(dis, order, 1), half,
                      center)
    orc.prune_cfs(buf, FD, "path", "dist", topm=TOPM, thre=THRE)
    sec = time.perf_counter() - t0
    return {"value": sec * n_total / sample, "unit": "s", "cores": orc.num_threads(),
            "kind": "port",
            "sample": f"first {sample} of the {n_total} base vectors, same K/iterations/prune; "
                      f"{sec:.2f}s measured, scaled by {n_total}/{sample}"}


def max_over_ranks(value, dist, device):
    """The slowest rank's time: every rank takes part (the same collective on
    every rank), and a single process returns its own value."""
    if not dist:
        return float(value)
    import torch
    t = torch.tensor([float(value)], device=device, dtype=torch.float64)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def workload_config(n, dim, world):
    """The workload both arms report (the reference arm runs a bounded CPU sample of it)."""
    return {"workload": "1M x 128 SIFT-like, GNN-Descent k=96 x10 + CFS path/dist 1.0 degree 32 "
                        "m=64", "n": n, "dim": dim, "k": K, "iters": ITERS, "final_degree": FD,
            "topm": TOPM, "storage": "f16 base",
            "screen": "tcgen05 f16 Gram tiles, exact f32 re-rank of every kept pair",
            "index_search": "reference NSG search, L=128, seeded random starts",
            "l2": "inputs larger than L2 (512 MB FP32 + 256 MB FP16 base)",
            "parallelism": f"replicas x{world}"}


def reference_arm(a, rank):
    if rank != 0:
        return
    from tagore_b200 import synth
    base, _ = synth.config(1, n=a.n)
    sample = min(a.cpu_sample, a.n)
    for _ in range(a.warmup):
        cpu_baseline(base, a.n, max(2000, sample // 8))
    vals = []
    for _ in range(a.steps):
        vals.append(cpu_baseline(base, a.n, sample))
    v = statistics.mean(x["value"] for x in vals)
    cb = dict(vals[-1])
    cb["value"] = v
    line = {"impl": "reference", "metric": METRIC, "value": v, "unit": "s", "n_gpus": a.gpus,
            "steps": a.steps, "warmup": a.warmup, "ms_per_step": v * 1000.0,
            "higher_is_better": False, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
            "data": "synthetic SIFT-like mixture (seeded), bounded CPU sample",
            "config": workload_config(a.n, 128, 1),
            "cpu_baseline": cb,
            "e2e": {"value": v, "unit": "s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


def main():
    a = args_()
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if a.impl == "reference":
        reference_arm(a, rank)
        return
    import torch
    from tagore_b200 import capi, synth
    torch.cuda.set_device(local)
    dist = None
    if world > 1:
        import datetime
        import torch.distributed as dist
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=600))
    L = capi.lib()
    base, queries = synth.config(1, n=a.n, nq=1000)
    n, dim = base.shape
    dev = torch.from_numpy(base).cuda()
    stream = torch.cuda.current_stream()
    capi.check(L.tagore_set_stream(C.c_void_p(stream.cuda_stream)))

    def build(mode):
        p = capi.knn_params(K, n, dim, ITERS, mode)
        st = capi.State()
        capi.check(L.tagore_gnn_descent_device(C.byref(p), C.c_void_p(dev.data_ptr()),
                                               base.ctypes.data_as(C.c_void_p), n, dim,
                                               C.byref(st.st)))
        capi.pruning_cfs(st, FD, "path", "dist", topm=TOPM, thre=THRE)
        return st

    def timed(mode, steps, warmup):
        for _ in range(warmup):
            build(mode).free()
        if dist:
            dist.barrier()
        torch.cuda.synchronize()
        capi.check(L.tagore_reset_counters())
        capi.check(L.tagore_set_profiling(1))
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        with Clocks(local) as clk:
            e0.record(stream)
            for _ in range(steps):
                build(mode).free()
            e1.record(stream)
            torch.cuda.synchronize()
        capi.check(L.tagore_set_profiling(0))
        ms = max_over_ranks(e0.elapsed_time(e1) / steps, dist, "cuda")
        launches = capi.last_timings().kernel_launches
        return ms, stage_stats(capi), launches, clk.summary()

    ms, stages, launches, clocks = timed(capi.KNN_CHOSEN, a.steps, a.warmup)
    plain_ms = None
    if not a.skip_plain:
        plain_ms, _, _, _ = timed(capi.KNN_PLAIN, max(1, a.steps // 2), 1)

    # per-kernel rooflines (algorithmic bytes per launch / mean launch time)
    peak, peak_kind = peaks()
    tflops_peak = tensor_peak()
    tf = os.path.join(ROOT, "profiles", "traffic.json")
    traffic_tab = json.load(open(tf)) if os.path.exists(tf) else {}

    def roofline(name):
        s_ms, s_launch, s_bytes, _ = stages[name]
        ms_l = s_ms / max(1, s_launch)
        byt = s_bytes / max(1, s_launch)
        achieved = byt / (ms_l * 1e-3) / 1e9 if s_bytes else None
        traffic = traffic_tab.get(name)
        r = {"bound": "hbm", "kernel": name, "achieved": achieved, "peak": peak, "unit": "GB/s",
             "frac": (achieved / peak) if achieved else None, "peak_source": peak_kind,
             "traffic": traffic, "algorithmic_bytes_per_launch": byt, "ms_per_launch": ms_l,
             "binding": BINDING.get(name, "unmeasured")}
        if traffic:
            r["dram_gbs"] = traffic / (ms_l * 1e-3) / 1e9
            r["dram_frac"] = r["dram_gbs"] / peak
        if name == "knn_join_tc":
            # the joins' 128 x 128 x d FP16 Gram tiles on tcgen05, as the kernels count them
            flops = 2.0 * 128 * 128 * dim * stages["knn_join_tiles"][3] / max(1, s_launch)
            r["tensor_tflops"] = flops / (ms_l * 1e-3) / 1e12
            r["tensor_peak_tflops"] = tflops_peak
            r["tensor_frac"] = r["tensor_tflops"] / tflops_peak
        return r

    ranked = sorted(stages, key=lambda k: stages[k][0], reverse=True)
    name = ranked[0]

    extra = {}
    if rank == 0 and not a.skip_prunes:
        # the configuration's other prunes on one chosen kNN graph, by the stage timers
        p = capi.knn_params(K, n, dim, ITERS, capi.KNN_CHOSEN)
        st = capi.State()
        capi.check(L.tagore_gnn_descent_device(C.byref(p), C.c_void_p(dev.data_ptr()),
                                               base.ctypes.data_as(C.c_void_p), n, dim,
                                               C.byref(st.st)))
        knn_bufs = st.buffers()
        st.free()
        for label, itype, thre in (("vamana_1.2", "Vamana", 1.2), ("cagra", "CAGRA", 1.0),
                                   ("nsg", "NSG", 1.0)):
            for rep in range(2):
                s2 = capi.State.alloc(n, dim, K)
                for i, (nm, _) in enumerate(capi.BUFFERS[:8]):
                    s2.upload(i, knn_bufs[nm])
                torch.cuda.synchronize()
                capi.check(L.tagore_reset_counters())
                capi.check(L.tagore_set_profiling(1))
                capi.pruning(s2, FD, itype, topm=TOPM, thre=thre)
                torch.cuda.synchronize()
                capi.check(L.tagore_set_profiling(0))
                st_ = stage_stats(capi)
                s2.free()
            extra[f"prune_{label}_ms"] = sum(v[0] for k, v in st_.items() if k.startswith("prune"))
            extra[f"prune_{label}_stages_ms"] = {k: v[0] for k, v in st_.items()}
        del knn_bufs
    if not a.skip_recall and rank == 0:
        samp = np.random.default_rng(0).choice(n, min(n, 10_000), replace=False)
        # two search seeds per build, three independent builds per path: the
        # spread between builds (sampling races, the kNN seed) is the larger
        # one, so the standard error is taken over builds
        seeds = [0x5EED + 7 * i for i in range(2)]
        builds = 3

        def seeded(rows, ep, half_t):
            return float(np.mean([index_recall(rows, ep, base, queries, half_t, seed=sd)
                                  for sd in seeds]))

        def mean_se(v):
            return float(np.mean(v)), float(np.std(v, ddof=1) / np.sqrt(len(v)))

        for label, mode in (("chosen", capi.KNN_CHOSEN), ("plain", capi.KNN_PLAIN)):
            if label == "plain" and a.skip_plain:
                continue
            kr, ir, cr, added = [], [], [], []
            for b in range(builds):
                p = capi.knn_params(K, n, dim, ITERS, mode, seed=0x7A6E + 101 * b)
                st = capi.State()
                capi.check(L.tagore_gnn_descent_device(C.byref(p), C.c_void_p(dev.data_ptr()),
                                                       base.ctypes.data_as(C.c_void_p), n, dim,
                                                       C.byref(st.st)))
                g = st.download(0).reshape(n, K)
                half_t = torch.from_numpy(st.download(2).reshape(n, dim)).cuda()
                kr.append(recall_knn(g, half_t, samp))
                ep = capi.pruning_cfs(st, FD, "path", "dist", topm=TOPM, thre=THRE)
                ir.append(seeded(st.download(0).reshape(n, K), ep, half_t))
                # the opt-in connectivity fix (edges appended; not part of the timed build)
                added.append(capi.connect(st, ep))
                cr.append(seeded(st.download(0).reshape(n, K), ep, half_t))
                st.free()
            extra[f"knn_recall10_{label}"], extra[f"knn_recall10_{label}_stderr"] = mean_se(kr)
            extra[f"index_recall10_{label}"], extra[f"index_recall10_{label}_stderr"] = mean_se(ir)
            m, se = mean_se(cr)
            extra[f"index_recall10_{label}_connected"] = m
            extra[f"index_recall10_{label}_connected_stderr"] = se
            extra[f"connect_edges_added_{label}"] = int(np.mean(added))
        extra["index_recall_seeds"] = len(seeds)
        extra["index_recall_builds"] = builds

    e2e = None
    if not a.skip_e2e:
        import torch
        capi.check(L.tagore_set_stream(None))
        # the base and the rows live in pinned host memory, as a caller that
        # streams builds would keep them; both copies are inside the timed call
        host_base = torch.from_numpy(np.ascontiguousarray(base, np.float32)).pin_memory().numpy()
        out = torch.empty((n, K), dtype=torch.int32).pin_memory().numpy().view(np.uint32)
        capi.build_index_host(host_base, K, ITERS, FD, TOPM, THRE, out=out)
        ts = []
        for _ in range(a.steps):
            t0 = time.perf_counter()
            capi.build_index_host(host_base, K, ITERS, FD, TOPM, THRE, out=out)
            ts.append(time.perf_counter() - t0)
        e2e_s = max_over_ranks(statistics.mean(ts), dist, "cuda")
        e2e = {"value": e2e_s, "unit": "s", "h2d_bytes_per_step": int(base.nbytes),
               "d2h_bytes_per_step": int(out.nbytes)}

    cpu = None
    if not a.skip_cpu and rank == 0 and world == 1:
        cpu = cpu_baseline(base, n, min(a.cpu_sample, n))

    if rank == 0:
        value = ms / 1000.0
        line = {"metric": METRIC, "value": value, "unit": "s", "n_gpus": world,
                "steps": a.steps, "warmup": a.warmup, "ms_per_step": ms,
                "higher_is_better": False, "scaling": "weak", "vs_baseline": None,
                "dtype": "f32",
                "data": "synthetic SIFT-like mixture (seeded, 256 components)",
                "config": workload_config(n, dim, world),
                "vectors_per_s": world * n / value,
                "plain_fp32_s": plain_ms / 1000.0 if plain_ms else None,
                "chosen_speedup_vs_plain": (plain_ms / ms) if plain_ms else None,
                "roofline": roofline(name),
                "roofline_next": [roofline(k) for k in ranked[1:3]],
                "stages_ms_per_step": {k: v[0] / a.steps for k, v in stages.items() if v[1]},
                "gpu_launches": launches,
                "clocks": clocks, "e2e": e2e, "cpu_baseline": cpu}
        line.update(extra)
        print(json.dumps(line), flush=True)
    capi.check(L.tagore_set_stream(None))
    if dist:
        dist.barrier()
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
