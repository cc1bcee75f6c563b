"""Benchmark: R-MAT scale-22 multilevel spectral bisection on B200.

One step = one full partition (HEC coarsening, coarse builds, Fiedler power
iteration on every level, median split) of the R-MAT scale-22 graph
(a, b, c, d = 0.57, 0.19, 0.19, 0.05, edge factor 16, seeded; symmetrised,
duplicates merged, self loops dropped, largest connected component kept).

  value  edges/s with the CSR resident in HBM and the partition left on the
         device (FP64 path), whole job over all ranks
  e2e    the same through the public API with pinned host buffers: the CSR
         upload and the partition download are inside the timed region
  mixed  the mixed-precision power iteration on the same graph (FP32
         edge-difference SpMV arithmetic; FP64 iterate, shift, deflation,
         normalisation, dot product and stopping test), its cut and its
         Fiedler value against the FP64 run
  fm     the same partition followed by up to 16 FM passes (cut and time)
  batch  the 2,048-graph batch configuration through the batched entry point
         (FP64 and mixed; edges/s of the whole batch, phase split)

Multi-GPU: the single-graph path does not shard (a row partition would need
halo exchanges per iteration); N ranks run N independent replicas ("weak"),
value = total edges of all replicas / max over ranks of the step time.

`--impl reference` times the reference's own OpenMP path (cmg/sgpar.h built
by oracle/Makefile) on the host cores: the timed steps partition a bounded
sample (R-MAT scale 18 from the same generator; a scale-22 partition takes
minutes there), and one partition of the scale-22 graph itself follows,
reported as `full_size`.

`--workload mtx2csr` measures the MatrixMarket converter instead (the
reference's cmg/mtx2csr.cpp): one step = one conversion of the R-MAT scale-22
graph written as a shuffled symmetric pattern file with 10% repeated entry
lines and 1% extra isolated vertices (symmetrise, dedupe and largest-component
extraction all do work); value = entry lines per second with the text resident
in HBM and the CSR left there, e2e = pinned host text to a host CSR, and the
reference arm times the reference converter binary on the same file.
"""
from __future__ import annotations

import argparse
import json
import os
import subprocess
import sys
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

RMAT = dict(edge_factor=16, a=0.57, b=0.19, c=0.19, seed=1)
SCALE = 22
REF_SAMPLE_SCALE = 18
METRIC = "edges/s partitioned (R-MAT scale 22 bisection, 1 graph per GPU)"


def rmat_graph(scale: int):
    from ipdps_2021_graph_coarsening_b200 import graphs as G
    cache = os.path.join("/tmp", f"sgpb_rmat{scale}_s{RMAT['seed']}.npz")
    if os.path.exists(cache):
        d = np.load(cache)
        return G.CSR(d["rp"], d["col"], None, f"rmat{scale}")
    g = G.rmat(scale, **RMAT)
    try:
        np.savez(cache, rp=g.row_ptr, col=g.col)
    except OSError:
        pass
    return g


def load_peaks():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(p):
        d = json.load(open(p))
        return float(d["hbm_gbs"]), "measured"
    return 6650.0, "fallback"


class Clocks:
    """nvidia-smi sampler running during the timed region."""
    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index: int):
        self.index = index
        self.p = None

    def __enter__(self):
        try:
            self.p = subprocess.Popen(["nvidia-smi", f"--id={self.index}", f"--query-gpu={self.Q}",
                                       "--format=csv,noheader,nounits", "-lms", "100"],
                                      stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
        except OSError:
            self.p = None
        return self

    def __exit__(self, *a):
        self.out = ""
        if self.p:
            self.p.terminate()
            try:
                self.out, _ = self.p.communicate(timeout=5)
            except subprocess.TimeoutExpired:
                self.p.kill()
                self.out, _ = self.p.communicate()

    def summary(self):
        rows = []
        for line in (self.out or "").splitlines():
            f = [x.strip() for x in line.split(",")]
            if len(f) >= 9:
                rows.append(f)
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unavailable"], "samples": 0}
        sm = [float(r[1]) for r in rows if r[1].replace(".", "").isdigit()]
        mx = [float(r[2]) for r in rows if r[2].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[k] for r in rows for k in range(4) if r[5 + k].lower() == "active"})
        return {"sm_mhz": float(np.median(sm)) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": reasons, "samples": len(rows)}


def algorithmic_pi_bytes(n: int, m: int, weighted: bool, s: int) -> int:
    """Bytes one power iteration must move (per-iteration model): offsets,
    destinations, weights (coarse levels), the iterate read and written, the
    degree vector."""
    return 4 * (n + 1) + 4 * m + (4 * m if weighted else 0) + s * n + s * n + 4 * n


def layout_pi_bytes(n: int, m: int, finest: bool) -> int:
    """Bytes an iteration streams at least, by the layout of the kernel that runs
    the level: the finest level's CSR (4-byte destinations and offsets), row
    slices elsewhere (2-byte destinations, weights not counted, a sum per row and
    panel of 25,600 columns written and read), the iterate read and written,
    the degrees."""
    if finest:
        return algorithmic_pi_bytes(n, m, False, 8)
    panels = -(-n // 25600)
    return 2 * m + 3 * 8 * n + (2 * 8 * panels * n if panels > 1 else 0)


def algorithmic_coarsen_bytes(level_n, level_m, level_rounds, wbytes: int = 4) -> int:
    """Bytes the coarsening of a hierarchy must move (the per-level model):
    the heavy-neighbour scan 4(n+1) + 4m + w*m (weighted levels) + 4n, the map
    construction 3*4n per round, and the coarse build 4(n+1) + 4m + w*m + 4n
    (vcmap) + 4(nc+1) + (4 + w)*mc; level 0 is unweighted."""
    total = 0
    for l in range(len(level_n) - 1):
        n, m, nc, mc = level_n[l], level_m[l], level_n[l + 1], level_m[l + 1]
        wm = wbytes * m if l > 0 else 0
        total += 4 * (n + 1) + 4 * m + wm + 4 * n
        total += 12 * n * max(1, level_rounds[l])
        total += 4 * (n + 1) + 4 * m + wm + 4 * n + 4 * (nc + 1) + (4 + wbytes) * mc
    return total


def dist_setup():
    ws = int(os.environ.get("WORLD_SIZE", "1"))
    if ws <= 1:
        return 0, 1, 0, None
    import torch.distributed as dist
    from datetime import timedelta
    rank = int(os.environ["RANK"])
    local = int(os.environ.get("LOCAL_RANK", rank))
    return rank, ws, local, (dist, timedelta)


def reference_arm(args, rank: int, ws: int):
    if rank != 0:
        return
    from oracle import bindings as O
    cores = os.cpu_count() or 1
    if not O.ref_available("omp"):
        print(json.dumps({"impl": "reference", "unavailable": "reference OpenMP build (oracle/_ref) not present"}))
        return
    g = rmat_graph(REF_SAMPLE_SCALE)
    times, cuts = [], []
    for i in range(args.warmup + args.steps):
        t = time.perf_counter()
        _, cut, _ = O.ref_partition_graph(g.row_ptr, g.col, rng_state=1000 + i, kind="omp")
        dt = time.perf_counter() - t
        if i >= args.warmup:
            times.append(dt)
            cuts.append(cut)
    sec = float(np.mean(times))
    value = g.m_undirected / sec
    sample = (f"R-MAT scale {REF_SAMPLE_SCALE} (same generator, {g.n} vertices, {g.m_undirected} edges), "
              f"one partition per step, reference OpenMP build of cmg/sgpar.h with {cores} threads")
    # one partition of the full-size graph, outside the timed steps: a
    # scale-22 partition takes minutes on the host cores, so the steps use
    # the bounded sample above
    full = None
    if not args.no_full_size:
        g22 = rmat_graph(SCALE)
        t = time.perf_counter()
        _, cut22, _ = O.ref_partition_graph(g22.row_ptr, g22.col, rng_state=1000, kind="omp")
        sec22 = time.perf_counter() - t
        full = {"workload": f"rmat{SCALE} bisection ({g22.n} vertices, {g22.m_undirected} edges)",
                "sec_per_partition": sec22, "edges_per_s": g22.m_undirected / sec22, "edgecut": int(cut22),
                "threads": cores, "kind": "reference OpenMP build of cmg/sgpar.h, one partition"}
    line = {"impl": "reference", "metric": METRIC, "value": value, "unit": "edges/s", "n_gpus": args.gpus,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": sec * 1e3, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": {"workload": f"rmat{SCALE} bisection (sampled as rmat{REF_SAMPLE_SCALE} on the CPU)",
                       "cutoff": 50, "tol": 1e-10},
            "cpu_baseline": {"value": value, "unit": "edges/s", "cores": cores, "kind": "reference",
                             "sample": sample},
            "e2e": {"value": value, "unit": "edges/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
            "edgecut_median": float(np.median(cuts)), "full_size": full}
    print(json.dumps(line))


def cpu_baseline():
    from oracle import bindings as O
    cores = os.cpu_count() or 1
    g = rmat_graph(REF_SAMPLE_SCALE)
    if O.ref_available("omp"):
        ts = []
        for i in range(3):
            t = time.perf_counter()
            O.ref_partition_graph(g.row_ptr, g.col, rng_state=500 + i, kind="omp")
            ts.append(time.perf_counter() - t)
        sec = float(np.median(ts))
        return {"value": g.m_undirected / sec, "unit": "edges/s", "cores": cores, "kind": "reference",
                "sample": f"R-MAT scale {REF_SAMPLE_SCALE} ({g.n} v, {g.m_undirected} e), median of 3 partitions, "
                          f"reference OpenMP build of cmg/sgpar.h"}
    t = time.perf_counter()
    O.partition_graph(g.row_ptr, g.col, None, rng_state=500)
    sec = time.perf_counter() - t
    return {"value": g.m_undirected / sec, "unit": "edges/s", "cores": 1, "kind": "port",
            "sample": f"R-MAT scale {REF_SAMPLE_SCALE}, 1 partition, oracle C restatement"}


def batch_graphs_cached():
    from ipdps_2021_graph_coarsening_b200 import graphs as G
    cache = os.path.join("/tmp", "sgpb_batch2048.npz")
    if os.path.exists(cache):
        d = np.load(cache)
        off_r, off_c, rp, col = d["off_r"], d["off_c"], d["rp"], d["col"]   # an npz reads a member on every access
        return [G.CSR(rp[off_r[i]:off_r[i + 1]], col[off_c[i]:off_c[i + 1]]) for i in range(len(off_r) - 1)]
    gs = G.batch_graphs(2048)
    try:
        off_r = np.cumsum([0] + [g.n + 1 for g in gs])
        off_c = np.cumsum([0] + [g.m_directed for g in gs])
        np.savez(cache, rp=np.concatenate([g.row_ptr for g in gs]), col=np.concatenate([g.col for g in gs]),
                 off_r=off_r, off_c=off_c)
    except OSError:
        pass
    return gs


def batch_leg(p, single_value):
    """The batch configuration (2,048 graphs of 10^3..2.5*10^5 vertices,
    grids with holes and Erdos-Renyi graphs, log-uniform sizes): one batched
    call, host graphs in and host partitions out, FP64 and mixed precision,
    after one untimed warm-up call on the whole batch (the first call of this
    size grows the memory pool: 11.0 s against 10.6 s for the next ones);
    wall clock around the call (it synchronises), phases from
    sgp_b200_last_timing."""
    gs = batch_graphs_cached()
    m_und = sum(g.m_undirected for g in gs)
    p.partition_batch(gs, workers=16)
    out = {"workload": "batch2048 (log-uniform 1e3..2.5e5 vertices; grids with 10% holes and ER mean degree 8; "
                       "LCC; unit weights)", "graphs": len(gs), "n": int(sum(g.n for g in gs)),
           "m_undirected": int(m_und), "workers": 16}
    for name, mixed in (("fp64", False), ("mixed", True)):
        t = time.perf_counter()
        rs = p.partition_batch(gs, workers=16, mixed=mixed)
        sec = time.perf_counter() - t
        ph = p.last_timing()
        out[name] = {"value": m_und / sec, "unit": "edges/s", "s": sec,
                     "phases_ms": {"coarsen": ph["coarsen"], "small_and_mid_levels": ph["eigen"],
                                   "large_levels_and_split": ph["split"]},
                     "edgecut_sum": int(sum(r.edgecut for r in rs))}
    out["mixed_speedup_vs_fp64"] = out["fp64"]["s"] / out["mixed"]["s"]
    out["fp64_vs_single_rmat22"] = out["fp64"]["value"] / single_value
    return out


def gpu_arm(args, rank: int, ws: int, local: int, distmod):
    import torch
    from ipdps_2021_graph_coarsening_b200.api import Partitioner
    from ipdps_2021_graph_coarsening_b200 import _lib as L

    torch.cuda.set_device(local)
    dist = None
    if distmod:
        dist, td = distmod
        dist.init_process_group("nccl", timeout=td(seconds=600), device_id=torch.device("cuda", local))
    g = rmat_graph(args.scale)
    n, m = g.n, g.m_directed
    p = Partitioner(local)
    if args.single:
        # one partition of the chosen case (used for profiler captures)
        rp_d = torch.from_numpy(g.row_ptr.view(np.int32)).cuda()
        col_d = torch.from_numpy(g.col.view(np.int32)).cuda()
        r = p.partition({"row_ptr": rp_d, "col": col_d}, rng_state=0x2021, mixed=args.mixed,
                        fm_passes=16 if args.fm else 0, coarsener=args.coarsener)
        if args.repeat:   # the same partition again, warm (pool, caches, modules loaded)
            r = p.partition({"row_ptr": rp_d, "col": col_d}, rng_state=0x2021, mixed=args.mixed,
                            fm_passes=16 if args.fm else 0, coarsener=args.coarsener)
        print(json.dumps({"case": f"rmat{args.scale}", "coarsener": args.coarsener, "n": n,
                          "m_undirected": g.m_undirected,
                          "ms": r.ms_total, "levels": r.level_n, "level_m": r.level_m,
                          "level_iters": r.level_iters, "level_pi_ms": r.level_pi_ms, "edgecut": r.edgecut,
                          "phase_ms": [r.ms_coarsen, r.ms_eigen, r.ms_split], "fm_passes": r.fm_passes,
                          "fm_moves": r.fm_moves}))
        p.close()
        return
    stream = torch.cuda.ExternalStream(L.lib().sgp_b200_stream(p._ctx))
    rp_d = torch.from_numpy(g.row_ptr.view(np.int32)).cuda()
    col_d = torch.from_numpy(g.col.view(np.int32)).cuda()
    part_d = torch.empty(n, dtype=torch.int32, device="cuda")
    dg = {"row_ptr": rp_d, "col": col_d}

    def barrier():
        if dist:
            dist.barrier()

    def timed(fn, steps):
        torch.cuda.synchronize()
        barrier()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        out = [fn() for _ in range(steps)]
        e1.record(stream)
        torch.cuda.synchronize()
        barrier()
        ms = e0.elapsed_time(e1) / steps
        if dist:
            t = torch.tensor([ms], device="cuda")
            dist.all_reduce(t, op=dist.ReduceOp.MAX)
            ms = float(t.item())
        return ms, out

    seed = 0x2021
    for _ in range(args.warmup):
        p.partition(dg, rng_state=seed, part_out=part_d)
    with Clocks(local) as clk:
        ms, res = timed(lambda: p.partition(dg, rng_state=seed, part_out=part_d), args.steps)
    r = res[-1]
    clocks = clk.summary()
    value = ws * g.m_undirected / (ms / 1e3)

    # end to end through the public API with pinned host buffers
    rp_h = torch.from_numpy(g.row_ptr.view(np.int32)).pin_memory().numpy().view(np.uint32)
    col_h = torch.from_numpy(g.col.view(np.int32)).pin_memory().numpy().view(np.uint32)
    part_h = torch.empty(n, dtype=torch.int32).pin_memory().numpy().view(np.uint32)
    from ipdps_2021_graph_coarsening_b200.graphs import CSR
    gh = CSR(rp_h, col_h, None, g.name)
    p.partition(gh, rng_state=seed, part_out=part_h)
    ms_e2e, res_e2e = timed(lambda: p.partition(gh, rng_state=seed, part_out=part_h), args.steps)
    e2e = {"value": ws * g.m_undirected / (ms_e2e / 1e3), "unit": "edges/s",
           "h2d_bytes_per_step": 4 * (n + 1) + 4 * m, "d2h_bytes_per_step": 4 * n, "ms_per_step": ms_e2e}

    # mixed precision on the same graph and seed
    p.partition(dg, rng_state=seed, part_out=part_d, mixed=True)
    ms_mx, res_mx = timed(lambda: p.partition(dg, rng_state=seed, part_out=part_d, mixed=True), args.steps)
    rm = res_mx[-1]
    mixed = {"value": ws * g.m_undirected / (ms_mx / 1e3), "ms_per_step": ms_mx, "edgecut": rm.edgecut,
             "edgecut_fp64": r.edgecut, "cut_rel_diff": abs(rm.edgecut - r.edgecut) / max(1, r.edgecut),
             "lambda_rel_err": abs(rm.lam - r.lam) / abs(r.lam) if r.lam else None,
             "residual": rm.residual, "speedup_vs_fp64": ms / ms_mx, "level_iters": rm.level_iters}

    # FM refinement of the same bisection (fm_passes), timed the same way
    p.partition(dg, rng_state=seed, part_out=part_d, fm_passes=16)
    ms_fm, res_fm = timed(lambda: p.partition(dg, rng_state=seed, part_out=part_d, fm_passes=16), args.steps)
    rf = res_fm[-1]
    fm = {"ms_per_step": ms_fm, "fm_ms": ms_fm - ms, "edgecut": rf.edgecut, "edgecut_spectral": r.edgecut,
          "cut_reduction": 1 - rf.edgecut / max(1, r.edgecut), "passes": rf.fm_passes, "moves": rf.fm_moves,
          "part0_size": rf.part0_size}

    # the batch configuration: 2,048 graphs through the batched entry point
    batch = None
    if ws == 1 and not args.no_batch:
        batch = batch_leg(p, value)

    # roofline of the dominant kernel (power iteration) from this step's levels:
    # the bytes its layouts stream, and beside them the rate of a kernel that
    # reads 8 bytes an entry (CSR with 4-byte weights) and takes the same time
    peak, peak_kind = load_peaks()
    levels = list(enumerate(zip(r.level_n, r.level_m, r.level_iters)))
    byts = sum(it * layout_pi_bytes(nl, ml, l == 0) for l, (nl, ml, it) in levels)
    byts_csr = sum(it * algorithmic_pi_bytes(nl, ml, l > 0, 8) for l, (nl, ml, it) in levels)
    pi_ms = sum(r.level_pi_ms)
    achieved = byts / (pi_ms / 1e3) / 1e9 if pi_ms > 0 else 0.0
    # DRAM bytes (read + write): the ratio of measured to layout bytes from one
    # ncu capture of this graph's largest coarse level, applied to the step
    traffic = None
    tf = os.path.join(ROOT, "profiles", "power_iter_traffic.json")
    if os.path.exists(tf):
        try:
            ratio = json.load(open(tf)).get("dram_to_layout_ratio")
            traffic = ratio * byts if ratio else None
        except (OSError, ValueError):
            traffic = None
    cbytes = algorithmic_coarsen_bytes(r.level_n, r.level_m, r.level_hec_rounds)
    roofline_coarsen = {"bound": "hbm", "algorithmic_bytes_per_step": cbytes, "ms_per_step": r.ms_coarsen,
                        "achieved": cbytes / (r.ms_coarsen / 1e3) / 1e9 if r.ms_coarsen else 0.0,
                        "peak": peak, "unit": "GB/s", "peak_kind": peak_kind,
                        "map_ms": r.ms_map, "build_ms": r.ms_build,
                        "kernels": "HEC scan + map rounds + coarse builds of every level"}
    roofline_coarsen["frac"] = roofline_coarsen["achieved"] / peak
    roofline = {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s", "frac": achieved / peak,
                "traffic": traffic, "kernel": "k_pi_slices (+ k_power_iter on the finest level, k_power_iter_chains on the small levels)",
                "peak_kind": peak_kind,
                "kernel_ms_per_step": pi_ms, "layout_bytes_per_step": byts,
                "csr_model_gbs": byts_csr / (pi_ms / 1e3) / 1e9 if pi_ms > 0 else 0.0,
                "kernel_share_of_step": pi_ms / ms if ms else None}

    line = {"metric": METRIC, "value": value, "unit": "edges/s", "n_gpus": ws, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ms, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": {"workload": f"rmat{SCALE} bisection (a,b,c,d=0.57,0.19,0.19,0.05, ef 16, seed 1, LCC)",
                       "n": n, "m_undirected": g.m_undirected, "cutoff": 50, "tol": 1e-10,
                       "parallelism": f"replicas{ws}", "l2": "inputs larger than L2 (CSR 0.5 GB)"},
            "edgecut": r.edgecut, "lambda": r.lam, "residual": r.residual, "levels": r.level_n,
            "level_m": r.level_m,
            "level_iters": r.level_iters, "level_pi_ms": [round(x, 3) for x in r.level_pi_ms],
            "phase_ms": {"coarsen": r.ms_coarsen, "eigen": r.ms_eigen, "split": r.ms_split},
            "clocks": clocks, "e2e": e2e, "mixed": mixed, "fm": fm, "batch": batch,
            "gpu_launches": r.kernel_launches * args.steps, "roofline": roofline,
            "roofline_coarsen": roofline_coarsen}
    if rank == 0 and ws == 1 and not args.no_cpu_baseline:
        line["cpu_baseline"] = cpu_baseline()
    if rank == 0:
        print(json.dumps(line))
    p.close()
    if dist:
        dist.destroy_process_group()


MTX_METRIC = "MatrixMarket entry lines/s converted to CSR (R-MAT scale 22 file, LCC kept)"
MTX_SAMPLE_SCALE = 20


def mtx_text(scale: int):
    """The converter's input: R-MAT `scale` as a shuffled symmetric pattern
    file with 10% repeated lines and 1% extra isolated vertices."""
    from ipdps_2021_graph_coarsening_b200 import graphs as G
    g = rmat_graph(scale)
    return g, G.mtx_of(g, seed=7, dup_frac=0.1, extra_vertices=g.n // 100)


def mtx_config(g, text, lines, scale):
    return {"workload": f"rmat{scale} as MatrixMarket (symmetric pattern, lower triangle shuffled, "
                        f"10% repeated lines, 1% isolated vertices)",
            "text_bytes": len(text), "entry_lines": lines, "n_out": g.n, "m_out_directed": g.m_directed,
            "l2": "inputs larger than L2 (text 1.2 GB)"}


def mtx_reference_arm(args, rank: int):
    """The reference converter (cmg/mtx2csr.cpp, built by oracle/Makefile) on
    the host: one step converts a file of the same construction at a bounded
    scale, file to file, as its command does."""
    if rank != 0:
        return
    ref = os.path.join(ROOT, "oracle", "_ref", "mtx2csr")
    if not os.path.exists(ref):
        print(json.dumps({"impl": "reference", "unavailable": "reference converter (oracle/_ref/mtx2csr) not built"}))
        return
    import tempfile
    g, text = mtx_text(MTX_SAMPLE_SCALE)
    lines = text.count(b"\n") - 2
    with tempfile.TemporaryDirectory() as d:
        src, dst = os.path.join(d, "g.mtx"), os.path.join(d, "g.csr")
        with open(src, "wb") as f:
            f.write(text)
        times = []
        for i in range(args.warmup + args.steps):
            t = time.perf_counter()
            subprocess.run([ref, src, dst], check=True, capture_output=True)
            if i >= args.warmup:
                times.append(time.perf_counter() - t)
    sec = float(np.mean(times))
    value = lines / sec
    line = {"impl": "reference", "metric": MTX_METRIC, "value": value, "unit": "lines/s", "n_gpus": args.gpus,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": sec * 1e3, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "u32", "data": "synthetic",
            "config": mtx_config(g, text, lines, MTX_SAMPLE_SCALE),
            "cpu_baseline": {"value": value, "unit": "lines/s", "cores": 1, "kind": "reference",
                             "sample": f"R-MAT scale {MTX_SAMPLE_SCALE} file of the same construction, "
                                       f"cmg/mtx2csr.cpp binary (serial), file to file"},
            "e2e": {"value": value, "unit": "lines/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line))


def mtx_arm(args, rank: int, ws: int, local: int, distmod):
    import torch
    from ipdps_2021_graph_coarsening_b200.api import Partitioner
    from ipdps_2021_graph_coarsening_b200 import _lib as L

    torch.cuda.set_device(local)
    dist = None
    if distmod:
        dist, td = distmod
        dist.init_process_group("nccl", timeout=td(seconds=600), device_id=torch.device("cuda", local))
    g, text = mtx_text(args.scale)
    lines = text.count(b"\n") - 2
    p = Partitioner(local)
    stream = torch.cuda.ExternalStream(L.lib().sgp_b200_stream(p._ctx))
    dtext = torch.frombuffer(bytearray(text), dtype=torch.uint8).cuda()
    if args.single:
        # two device-resident conversions (the second is the one to read in a
        # profiler's launch list), then the phase split
        for _ in range(2):
            info = p.mtx_read(dtext, device_out=True)[1]
        print(json.dumps({"case": f"rmat{args.scale} MatrixMarket", "lines": lines, "text_bytes": len(text),
                          **{k: info[k] for k in ("n", "m", "components", "ms_parse", "ms_rows", "ms_components",
                                                   "ms_extract", "kernel_launches")}}))
        p.close()
        return
    htext = torch.frombuffer(bytearray(text), dtype=torch.uint8).pin_memory()

    def barrier():
        if dist:
            dist.barrier()

    def timed(fn, steps):
        torch.cuda.synchronize()
        barrier()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        out = [fn() for _ in range(steps)]
        e1.record(stream)
        torch.cuda.synchronize()
        barrier()
        ms = e0.elapsed_time(e1) / steps
        if dist:
            t = torch.tensor([ms], device="cuda")
            dist.all_reduce(t, op=dist.ReduceOp.MAX)
            ms = float(t.item())
        return ms, out

    def dev_step():
        return p.mtx_read(dtext, device_out=True)[1]

    def host_step():
        return p.mtx_read(htext)[1]

    for _ in range(args.warmup):
        dev_step()
    with Clocks(local) as clk:
        ms, infos = timed(dev_step, args.steps)
    info = infos[-1]
    assert info["n"] == g.n and info["m"] == g.m_directed, "converter output differs from the generated graph"
    clocks = clk.summary()
    value = ws * lines / (ms / 1e3)
    host_step()
    ms_e2e, _ = timed(host_step, args.steps)
    e2e = {"value": ws * lines / (ms_e2e / 1e3), "unit": "lines/s", "h2d_bytes_per_step": len(text),
           "d2h_bytes_per_step": 4 * (g.n + 1) + 4 * g.m_directed, "ms_per_step": ms_e2e}
    # roofline: the parse pass (line starts, ids, degrees) is the byte-bound
    # kernel; the phase split says where the rest of the step goes
    peak, peak_kind = load_peaks()
    parse_bytes = 2 * len(text) + 8 * lines
    # DRAM traffic: the parse kernel's measured bytes per line (one ncu
    # capture on the R-MAT 20 file, profiles/mtx_parse_traffic.json) scaled
    # to this file, plus the count kernel's one streaming read of the text
    traffic = None
    tf = os.path.join(ROOT, "profiles", "mtx_parse_traffic.json")
    if os.path.exists(tf):
        try:
            traffic = json.load(open(tf))["dram_bytes_per_line"] * lines + len(text)
        except (OSError, ValueError, KeyError):
            traffic = None
    roofline = {"bound": "hbm", "kernel": "k_mtx_count + k_mtx_parse (text pass)",
                "algorithmic_bytes": parse_bytes, "kernel_ms": info["ms_parse"],
                "achieved": parse_bytes / (info["ms_parse"] / 1e3) / 1e9, "peak": peak, "unit": "GB/s",
                "peak_kind": peak_kind, "traffic": traffic,
                "note": "phase time incl. two scans and read-backs; the pass is instruction-bound "
                        "(profiles/mtx_parse_rmat20.md); the step's largest kernel is the row sort"}
    roofline["frac"] = roofline["achieved"] / peak
    line = {"metric": MTX_METRIC, "value": value, "unit": "lines/s", "n_gpus": ws, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ms, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "u32", "data": "synthetic",
            "config": mtx_config(g, text, lines, args.scale),
            "phase_ms": {k: info[k] for k in ("ms_parse", "ms_rows", "ms_components", "ms_extract")},
            "components": info["components"], "clocks": clocks, "e2e": e2e, "roofline": roofline,
            "gpu_launches": info["kernel_launches"] * args.steps}
    if rank == 0 and ws == 1 and not args.no_cpu_baseline:
        ref = os.path.join(ROOT, "oracle", "_ref", "mtx2csr")
        if os.path.exists(ref):
            import tempfile
            gs, ts = mtx_text(MTX_SAMPLE_SCALE)
            with tempfile.TemporaryDirectory() as d:
                src, dst = os.path.join(d, "g.mtx"), os.path.join(d, "g.csr")
                with open(src, "wb") as f:
                    f.write(ts)
                t = time.perf_counter()
                subprocess.run([ref, src, dst], check=True, capture_output=True)
                sec = time.perf_counter() - t
            nl = ts.count(b"\n") - 2
            line["cpu_baseline"] = {"value": nl / sec, "unit": "lines/s", "cores": 1, "kind": "reference",
                                    "sample": f"R-MAT scale {MTX_SAMPLE_SCALE} file of the same construction "
                                              f"({nl} lines), cmg/mtx2csr.cpp binary, file to file"}
    if rank == 0:
        print(json.dumps(line))
    p.close()
    if dist:
        dist.destroy_process_group()


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-batch", action="store_true", help="skip the 2,048-graph batch leg")
    ap.add_argument("--no-full-size", action="store_true",
                    help="with --impl reference: skip the one full-size reference partition")
    ap.add_argument("--scale", type=int, default=SCALE, help="R-MAT scale (the benchmark is 22)")
    ap.add_argument("--single", action="store_true",
                    help="one partition (or, with --workload mtx2csr, two conversions) of --scale and exit (profiling)")
    ap.add_argument("--mixed", action="store_true", help="with --single: mixed-precision power iteration")
    ap.add_argument("--fm", action="store_true", help="with --single: FM passes after the split")
    ap.add_argument("--coarsener", type=int, default=0, help="with --single: options.coarsener (0 = HEC)")
    ap.add_argument("--repeat", action="store_true", help="with --single: report a second, warm partition")
    ap.add_argument("--workload", default="partition", choices=["partition", "mtx2csr"],
                    help="partition (the headline) or the MatrixMarket converter")
    args = ap.parse_args()
    if args.warmup < 3:
        args.warmup = 3
    rank, ws, local, distmod = dist_setup()
    if args.impl == "reference":
        os.environ.setdefault("OMP_NUM_THREADS", str(os.cpu_count() or 1))
        if args.workload == "mtx2csr":
            mtx_reference_arm(args, rank)
        else:
            reference_arm(args, rank, ws)
        return
    os.environ.setdefault("OMP_NUM_THREADS", str(os.cpu_count() or 1))
    if args.workload == "mtx2csr":
        mtx_arm(args, rank, ws, local, distmod)
    else:
        gpu_arm(args, rank, ws, local, distmod)


if __name__ == "__main__":
    main()
