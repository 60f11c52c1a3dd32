#!/usr/bin/env python3
"""Throughput of the full hot path on one GB300: all 13 simplex relations plus
critical-point classification, in Mtets/s.

A step = one pass of the path over one mesh: tg_mesh_create (row sort,
validation, VT) + tg_extract(all 13 relations) + tg_critical_points, then the
mesh is destroyed.  The default workload is the large mesh: a 128^3 Kuhn grid
(12,582,912 tets, 2,146,689 vertices), vertex ids permuted, float32 field
sin(ax) sin(by) sin(cz) + N(0, 1e-4).

  value     device-resident inputs (TV and field already in HBM), device
            outputs; CUDA events on the launching stream around each step; L2
            flushed (a 512 MB write) before every step, outside the timed
            window.
  roofline  the whole path against HBM bandwidth: compulsory bytes of a step
            (TV and field read once, every output written once) / step time /
            the measured copy peak; `kernel` inside it is the dominant kernel
            (k_star) on the compulsory bytes it is responsible for, timed
            live with CUDA events on its stream.
  e2e       the same steps through the C ABI with HOST buffers: pinned TV in
            through tg_mesh_create(tv_on_device = 0), the pinned field through
            tg_critical_points(field_on_device = 0), every relation plus the
            classes copied back to pinned host memory
            (tg_copy_relations_async_i32: CSR offsets as int32, narrowed on the
            device by one launch), all inside the timed window.  Steps
            alternate between two streams and two sets of host buffers, so a
            step's copies back overlap the next step's extraction (the host
            link, not the kernels, bounds this number).
  batch     the uneven 512-mesh batch (tet counts log-uniform in [2k, 400k]):
            one batched pipeline run per step against the plain per-mesh loop,
            both timed with CUDA events, and their ratio.

Under torchrun (N > 1) each rank runs an independent replica on its own GPU
(the path does not shard within a mesh); value = tets of all ranks / max time.

--impl reference times the reference's CPU path (the C restatement of it in
oracle/, the only build that exists on the GPU host) on the host cores: one
process per core, each step a bounded sample of the same workload.
"""
from __future__ import annotations

import argparse
import functools
import json
import multiprocessing as mp
import os
import statistics
import subprocess
import sys
import tempfile
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "Mtets/s (13 relations + crit. points), batched vs per-mesh on 1 GB300; p99 ms"
UNIT = "Mtets/s"
WORKLOAD = "kuhn128_permuted_large"
# --workload: the irregular single mesh (the headline), the 128^3 large mesh,
# or the uneven 512-mesh batch (batched path against the per-mesh loop)
WORKLOADS = {"irregular": "kuhn64_coned20_irregular", "large": "kuhn128_permuted_large",
             "batch": "batch512_uneven_2k_400k", "serve": "serve_poisson_70new_30field"}
DEFAULT_STEPS = {"irregular": 300, "large": 20, "batch": 5, "serve": 1}


@functools.lru_cache(maxsize=2)
def load_workload(key: str):
    from tetragpu_gb300 import meshgen
    return WORKLOADS[key], (meshgen.workload_irregular() if key == "irregular"
                            else meshgen.workload_large())
ROOFLINE_KERNEL = "k_star"
# CPU sample for the baseline legs: cells [0, SAMPLE_CELLS) of the same mesh
# (a valid mesh itself), run through the oracle.
SAMPLE_CELLS = 262144


def env_rank():
    return (int(os.environ.get("RANK", 0)), int(os.environ.get("LOCAL_RANK", 0)),
            int(os.environ.get("WORLD_SIZE", 1)))


def max_over_ranks(x: float, dist, torch, device) -> float:
    """The slowest rank's time: replicas share nothing but this reduction."""
    t = torch.tensor([x], device=device, dtype=torch.float64)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def peaks():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(p):
        with open(p) as f:
            d = json.load(f)
        return float(d["hbm_gbs"]), "measured"
    return 6800.0, "fallback"


# ---------------------------------------------------------------------------
# clocks sampling
# ---------------------------------------------------------------------------
class Clocks:
    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index: int):
        self.gpu = gpu_index
        self.proc = None
        self.path = None

    def start(self):
        try:
            fd, self.path = tempfile.mkstemp(suffix=".csv")
            os.close(fd)
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.gpu), f"--query-gpu={self.FIELDS}",
                 "--format=csv,noheader,nounits", "-lms", "100"],
                stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except Exception:
            self.proc = None

    def stop(self) -> dict:
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        sm, smax, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        with open(self.path) as f:
            for line in f:
                parts = [x.strip() for x in line.split(",")]
                if len(parts) < 9:
                    continue
                try:
                    sm.append(float(parts[1]))
                    smax.append(float(parts[2]))
                except ValueError:
                    continue
                for n, val in zip(names, parts[5:9]):
                    if val.lower().startswith("active"):
                        reasons.add(n)
        os.unlink(self.path)
        return {"sm_mhz": statistics.median(sm) if sm else None,
                "sm_max_mhz": max(smax) if smax else None, "reasons": sorted(reasons),
                "samples": len(sm)}


# ---------------------------------------------------------------------------
# algorithmic bytes
# ---------------------------------------------------------------------------
def output_bytes(counts: dict, totals: dict) -> int:
    """Compulsory bytes of the whole path: TV read once (16 B/tet), field read
    once (4 B/vertex), every output written once (int32 entries, int64 CSR
    offsets), classes written once (12 B/vertex)."""
    V, E, F, T = counts["V"], counts["E"], counts["F"], counts["T"]
    b = 16 * T + 4 * V + 12 * V
    b += 4 * (6 * T + 2 * E + 4 * T + 3 * F + 3 * F + 2 * F)          # TE EV TF FV FE FT
    for name, rows in (("ET", E), ("EF", E), ("VT", V), ("TT", T), ("FF", F), ("EE", E),
                       ("VV", V)):
        b += 8 * (rows + 1) + 4 * totals[name]
    return b


def union_sizes(tg, batch) -> dict:
    """Counts and CSR totals of a batch's union mesh (the sum over its
    members), for output_bytes."""
    C = tg._lib.C
    lib = tg.load()
    u = lib.tg_batch_union(batch._h)
    v, e, f, t = (C.c_int64() for _ in range(4))
    tg._lib.check(lib.tg_mesh_counts(u, C.byref(v), C.byref(e), C.byref(f), C.byref(t)))
    totals = {}
    for n in ("ET", "EF", "VT", "TT", "FF", "EE", "VV"):
        off, ent = C.c_void_p(), C.c_void_p()
        rows, cnt, width = C.c_int64(), C.c_int64(), C.c_int32()
        tg._lib.check(lib.tg_get_relation(u, tg.REL[n], C.byref(off), C.byref(ent), C.byref(rows),
                                          C.byref(cnt), C.byref(width)))
        totals[n] = cnt.value
    return {"counts_totals": ({"V": v.value, "E": e.value, "F": f.value, "T": t.value}, totals)}


def kernel_bytes(name: str, c: dict, tot: dict) -> int:
    """Compulsory bytes one launch of a kernel is responsible for: the path's
    inputs it reads once and the final outputs it writes once.  Intermediates
    (first-occurrence bitmaps, edge records, rank words, offsets read back)
    are overhead and not credited.  k_star reads the sorted TV (16 B per cell)
    and VT (16 B per cell, 8 B per vertex); all it writes are intermediates."""
    V, E, F, T = c["V"], c["E"], c["F"], c["T"]
    if name == "k_star":
        return 16 * T + 4 * tot["VT"] + 8 * V
    raise KeyError(name)


def traffic_from_profiles(name: str, workload: str, scale: float,
                          key: str = "dram_bytes_per_launch"):
    """DRAM bytes recorded from an ncu capture (profiles/<name>_<workload>.md,
    a line '<key>: N' and a line 'cells: T'), scaled to this run's cells."""
    p = os.path.join(ROOT, "profiles", f"{name}_{workload}.md")
    if not os.path.exists(p):
        return None
    vals = {}
    with open(p) as f:
        for line in f:
            if ":" in line and line.strip().startswith((key, "cells")):
                k, v = line.split(":", 1)
                try:
                    vals[k.strip()] = float(v.strip().split()[0].replace(",", ""))
                except ValueError:
                    pass
    if key not in vals:
        return None
    b = vals[key]
    if "cells" in vals and vals["cells"] > 0:
        b *= scale / vals["cells"]
    return int(b)


# ---------------------------------------------------------------------------
# CPU legs (oracle = the reference CPU path restated in C)
# ---------------------------------------------------------------------------
def _cpu_sample_worker(args):
    tv, n_verts, field, steps = args
    sys.path.insert(0, ROOT)
    from oracle.oracle import Oracle
    o = Oracle()
    times = []
    for _ in range(steps):
        t0 = time.perf_counter()
        tvs = o.canonicalize(tv, n_verts)
        o.extract(tvs, n_verts)
        o.critical_points(tvs, n_verts, field)
        times.append(time.perf_counter() - t0)
    return times


def cpu_sample(mesh):
    tv = np.ascontiguousarray(mesh.tv[:SAMPLE_CELLS])
    return tv, mesh.n_verts, mesh.field


# the 7 relations the reference's CPU code implements (TE, EV, ET, TF, FV,
# VT, VV: make_TE_and_VE, make_TF_and_VF, elective_make_*)
REF_BUILD_MASK = sum(1 << i for i in (1, 2, 3, 4, 5, 9, 13))


def reference_build_baseline(mesh, workload: str) -> dict | None:
    """The reference's own CPU code (src/cpu_extraction.cpp, compiled
    unmodified into oracle/_ref/libtgref.so where the reference tree was
    present at build time) on the same sample, for the 7 relations it
    implements, beside the port on the same 7; None where that build does
    not exist (the GPU host has no reference tree)."""
    from oracle import oracle as O
    if not O.Reference.available():
        return None
    O.build()
    tv, nv, _ = cpu_sample(mesh)
    orc, ref = O.Oracle(), O.Reference()
    tvs = orc.canonicalize(tv, nv)
    t_ref, t_port = [], []
    for _ in range(2):
        t_ref.append(ref.extract(tvs, nv)["seconds"])
        t0 = time.perf_counter()
        orc.extract(tvs, nv, mask=REF_BUILD_MASK)
        t_port.append(time.perf_counter() - t0)
    n = tv.shape[0]
    return {"value": round(n / min(t_ref) / 1e6, 4), "unit": UNIT, "cores": 1,
            "kind": "reference_build",
            "relations": "TE EV ET TF FV VT VV (the 7 the reference implements on the CPU)",
            "port_same_relations": round(n / min(t_port) / 1e6, 4),
            "sample": f"cells [0, {n}) of the {workload} mesh, row-sorted, single thread, "
                      f"best of 2 ({min(t_ref):.2f} s reference, {min(t_port):.2f} s port)"}


def cpu_baseline(mesh, workload: str = WORKLOAD) -> dict:
    from oracle import oracle as O
    O.build()
    tv, nv, field = cpu_sample(mesh)
    times = _cpu_sample_worker((tv, nv, field, 2))
    t = min(times)
    out = {"value": round(tv.shape[0] / t / 1e6, 4), "unit": UNIT, "cores": 1, "kind": "port",
           "sample": f"cells [0, {tv.shape[0]}) of the {workload} mesh, all 13 relations + "
                     f"critical points, single thread, best of 2 ({t:.2f} s)"}
    rb = reference_build_baseline(mesh, workload)
    out["reference_build"] = rb if rb else \
        "not on this host: the reference's own CPU build needs the reference source tree"
    return out


def run_reference(args):
    rank, _, world = env_rank()
    if rank != 0:
        return
    from oracle import oracle as O
    O.build()
    workload, mesh = load_workload(args.workload)
    tv, nv, field = cpu_sample(mesh)
    cores = os.cpu_count() or 1
    # warm-up + timed steps in every worker process, all cores busy at once
    ctx = mp.get_context("spawn")
    t0 = time.perf_counter()
    with ctx.Pool(cores) as pool:
        per = pool.map(_cpu_sample_worker, [(tv, nv, field, args.warmup + args.steps)] * cores)
    wall = time.perf_counter() - t0
    timed = [sum(t[args.warmup:]) for t in per]
    tmax = max(timed)
    value = cores * args.steps * tv.shape[0] / tmax / 1e6
    line = {
        "impl": "reference", "metric": METRIC, "value": round(value, 4), "unit": UNIT,
        "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": round(1e3 * tmax / args.steps, 3), "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "int32", "data": "synthetic",
        "config": {"workload": workload, "cells_per_step": int(tv.shape[0]),
                   "note": "the reference CPU path (serial) restated in C; one process per core"},
        "cpu_baseline": {"value": round(value, 4), "unit": UNIT, "cores": cores, "kind": "port",
                         "sample": f"cells [0, {tv.shape[0]}) of the {workload} mesh per step, "
                                   f"{cores} processes in parallel, wall {wall:.1f} s"},
        "e2e": {"value": round(value, 4), "unit": UNIT, "h2d_bytes_per_step": 0,
                "d2h_bytes_per_step": 0},
    }
    rb = reference_build_baseline(mesh, workload)
    if rb:
        line["cpu_baseline"]["reference_build"] = rb
    print(json.dumps(line), flush=True)


# ---------------------------------------------------------------------------
# GPU arm
# ---------------------------------------------------------------------------
def run_batch(args, torch, dist, tg, rank, local_rank, world, steps, e2e_steps):
    """The uneven 512-mesh batch: one batched pipeline run (tg_batch_*) per
    step against the plain per-mesh loop (tg_mesh_* per mesh) over the same
    device-resident meshes; both arms time the same step (create, all 13
    relations, critical points, destroy) with CUDA events.  Returns the JSON
    line's fields (rank 0)."""
    from tetragpu_gb300 import meshgen
    meshes = meshgen.workload_batch()
    nc = np.array([m.n_cells for m in meshes], dtype=np.int64)
    nv = np.array([m.n_verts for m in meshes], dtype=np.int64)
    c_off = np.concatenate([[0], np.cumsum(nc)])
    v_off = np.concatenate([[0], np.cumsum(nv)])
    T, V = int(c_off[-1]), int(v_off[-1])
    tv_all = np.concatenate([m.tv for m in meshes])
    f_all = np.concatenate([m.field for m in meshes]).astype(np.float32)
    dev = f"cuda:{local_rank}"
    stream = torch.cuda.Stream()
    s = stream.cuda_stream
    d_tv = torch.from_numpy(tv_all).to(dev)
    d_f = torch.from_numpy(f_all).to(dev)
    d_cls = torch.empty(3 * V, dtype=torch.int32, device=dev)
    flush = torch.empty(512 << 20, dtype=torch.uint8, device=dev)
    torch.cuda.synchronize()

    sizes = {}

    def batch_step():
        with tg.Batch(d_tv.data_ptr(), nv, n_cells=nc, on_device=True, stream=s) as b:
            b.extract(tg.ALL_RELATIONS, options=tg.OPT_LINK_ADJACENCY, stream=s)
            b.critical_points(d_f.data_ptr(), on_device=True, out_ptr=d_cls.data_ptr(), stream=s)
            if not sizes:   # the union's counts and CSR totals: the batch's output bytes
                sizes.update(union_sizes(tg, b))

    def loop_step():
        for i in range(len(meshes)):
            with tg.Mesh(d_tv.data_ptr() + 16 * int(c_off[i]), int(nv[i]), n_cells=int(nc[i]),
                         on_device=True, stream=s) as g:
                g.extract(tg.ALL_RELATIONS, options=tg.OPT_LINK_ADJACENCY, stream=s)
                g.critical_points(d_f.data_ptr() + 4 * int(v_off[i]), on_device=True,
                                  out_ptr=d_cls.data_ptr() + 12 * int(v_off[i]), stream=s)

    def timed(fn, k_steps):
        with torch.cuda.stream(stream):
            for _ in range(max(3, args.warmup)):
                fn()
        torch.cuda.synchronize()
        ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True))
              for _ in range(k_steps)]
        if world > 1:
            dist.barrier()
        torch.cuda.synchronize()
        l0 = tg.kernel_launch_count()
        with torch.cuda.stream(stream):
            for k in range(k_steps):
                flush.fill_(k & 0xff)
                ev[k][0].record(stream)
                fn()
                ev[k][1].record(stream)
        torch.cuda.synchronize()
        total = sum(a.elapsed_time(b) for a, b in ev) / 1e3
        if world > 1:
            total = max_over_ranks(total, dist, torch, dev)
        return total, tg.kernel_launch_count() - l0

    clocks = Clocks(local_rank)
    clocks.start()
    t_batch, launches = timed(batch_step, steps)
    clk = clocks.stop()
    t_loop, loop_launches = timed(loop_step, steps)
    value = world * steps * T / t_batch / 1e6
    loop_value = world * steps * T / t_loop / 1e6
    peak, peak_kind = peaks()
    alg = output_bytes(*sizes["counts_totals"])
    batch_gbs = alg / (t_batch / steps) / 1e9

    # e2e: host TV and fields in, every relation of the union and the classes
    # back to pinned host memory, through the batch API.  As for the single
    # mesh, steps alternate between two streams and two sets of host buffers
    # so one step's copies back overlap the next step's work; inputs go up
    # before the previous step's results come down.
    pin_tv = torch.from_numpy(tv_all).pin_memory()
    pin_f = torch.from_numpy(f_all).pin_memory()
    e2e_value, h2d, d2h = None, pin_tv.numel() * 4 + pin_f.numel() * 4, 12 * V
    lib = tg.load()
    C = tg._lib.C
    if e2e_steps > 0:
        e_streams = [torch.cuda.Stream(), torch.cuda.Stream()]
        d_tv2 = [torch.empty_like(d_tv) for _ in range(2)]
        d_f2 = [torch.empty_like(d_f) for _ in range(2)]
        d_cls2 = [torch.empty(3 * V, dtype=torch.int32, device=dev) for _ in range(2)]
        h_bufs = [{}, {}]
        h_cls = [torch.empty(3 * V, dtype=torch.int32).pin_memory() for _ in range(2)]

        def upload(k):
            with torch.cuda.stream(e_streams[k % 2]):
                d_tv2[k % 2].copy_(pin_tv, non_blocking=True)
                d_f2[k % 2].copy_(pin_f, non_blocking=True)

        def e2e_run(n_steps):
            live = None
            upload(0)
            for k in range(n_steps):
                es = e_streams[k % 2].cuda_stream
                b = tg.Batch(d_tv2[k % 2].data_ptr(), nv, n_cells=nc, on_device=True, stream=es)
                b.extract(tg.ALL_RELATIONS, options=tg.OPT_LINK_ADJACENCY, stream=es)
                tg._lib.check(lib.tg_batch_critical_points(b._h, d_f2[k % 2].data_ptr(),
                                                           tg.FIELD_F32, 1,
                                                           d_cls2[k % 2].data_ptr(), 1, es))
                if k + 1 < n_steps:
                    upload(k + 1)
                u = lib.tg_batch_union(b._h)
                po, pe = (C.c_void_p * 14)(), (C.c_void_p * 14)()
                for n in tg.RELATIONS[1:]:
                    off, ent = C.c_void_p(), C.c_void_p()
                    rows, cnt, width = C.c_int64(), C.c_int64(), C.c_int32()
                    tg._lib.check(lib.tg_get_relation(u, tg.REL[n], C.byref(off), C.byref(ent),
                                                      C.byref(rows), C.byref(cnt),
                                                      C.byref(width)))
                    hb = h_bufs[k % 2]
                    if n not in hb:
                        hb[n] = (torch.empty(max(cnt.value, 1), dtype=torch.int32).pin_memory(),
                                 torch.empty(rows.value + 1, dtype=torch.int32).pin_memory()
                                 if width.value == 0 else None)
                    he, ho = hb[n]
                    pe[tg.REL[n]] = he.data_ptr() if cnt.value else None
                    po[tg.REL[n]] = ho.data_ptr() if ho is not None else None
                tg._lib.check(lib.tg_copy_relations_async_i32(u, tg.ALL_RELATIONS, po, pe, es))
                with torch.cuda.stream(e_streams[k % 2]):
                    h_cls[k % 2].copy_(d_cls2[k % 2], non_blocking=True)
                if live is not None:
                    live.close()    # waits for the previous step's copies
                live = b
            if live is not None:
                live.close()
            torch.cuda.synchronize()

        e2e_run(2)
        d2h += sum(a.numel() * 4 + (bb.numel() * 4 if bb is not None else 0)
                   for a, bb in h_bufs[0].values())
        t0 = time.perf_counter()
        e2e_run(e2e_steps)
        e2e_value = round(world * e2e_steps * T / (time.perf_counter() - t0) / 1e6, 3)

    line = None
    if rank == 0:
        line = {
            "metric": METRIC, "value": round(value, 3), "unit": UNIT, "n_gpus": world,
            "steps": steps, "warmup": max(3, args.warmup),
            "ms_per_step": round(1e3 * t_batch / steps, 3), "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "int32", "data": "synthetic",
            "config": {"workload": WORKLOADS["batch"], "meshes": len(meshes), "cells": T,
                       "vertices": V, "relations": "all 13 + critical points",
                       "parallelism": f"replicas{world}",
                       "l2": "flushed before every step (512 MB write)"},
            "gpu_launches": int(launches),
            "clocks": clk,
            "per_mesh_loop": {"value": round(loop_value, 3), "unit": UNIT,
                              "ms_per_step": round(1e3 * t_loop / steps, 3),
                              "gpu_launches": int(loop_launches)},
            "batched_over_loop": round(value / loop_value, 3),
            "tuning": tg.batch_tuning(),
            "roofline": {"bound": "hbm", "scope": "path (one batched step)",
                         "achieved": round(batch_gbs, 1), "peak": peak, "unit": "GB/s",
                         "frac": round(batch_gbs / peak, 4), "peak_source": peak_kind,
                         "algorithmic_bytes_per_step": alg, "traffic": None},
            "e2e": {"value": e2e_value, "unit": UNIT, "h2d_bytes_per_step": int(h2d),
                    "d2h_bytes_per_step": int(d2h), "steps": e2e_steps},
        }
    return line


def main_batch(args, torch, dist, tg, rank, local_rank, world):
    line = run_batch(args, torch, dist, tg, rank, local_rank, world, args.steps, args.e2e_steps)
    if rank == 0:
        if not args.no_cpu_baseline:
            line["cpu_baseline"] = cpu_baseline(load_workload("large")[1], WORKLOADS["large"])
        print(json.dumps(line), flush=True)


def serve_requests(n_req: int, n_pool: int, seed: int):
    """The request mix, materialised before the stream starts.  Grids: a pool
    of seeded Kuhn grids (the large mesh's generator: ids permuted), tet counts
    lognormal with median 50k and sigma 1, capped at 4M, four Gaussian-mixture
    fields each.  70% of requests are new meshes: a pool grid under a fresh
    seeded vertex relabelling and slot shuffle, so that no two requests share a
    mesh (ids, relations and classes all differ) while sizes follow the pool;
    30% are new fields on the mesh of an earlier request (the field relabelled
    the same way).  Returns the requests as ("mesh", tv, n_verts, field) or
    ("field", index of the mesh request, field), and their tet counts."""
    from tetragpu_gb300 import meshgen
    rng = np.random.default_rng(seed)
    pool = []
    for i in range(n_pool):
        target = float(min(4e6, np.exp(rng.normal(np.log(5e4), 1.0))))
        dims = meshgen._dims_for(max(target, 6.0), rng)
        m = meshgen.kuhn_mesh(dims, 0.0, seed=seed * 1000 + i)
        m.fields = [meshgen.gaussian_mixture_field(m.coords, n_gauss=8, seed=seed * 1000 + i * 7 + k,
                                                   noise=1e-3) for k in range(4)]
        pool.append(m)
    reqs, tets, mesh_reqs = [], [], []
    for r in range(n_req):
        if mesh_reqs and rng.random() < 0.3:
            k = int(rng.choice(mesh_reqs))
            _, perm, pi = reqs[k][1:4]
            m = pool[pi]
            f = np.empty_like(m.fields[0])
            f[perm] = m.fields[int(rng.integers(0, 4))]
            reqs.append(("field", k, f))
            tets.append(m.n_cells)
        else:
            pi = int(rng.integers(0, n_pool))
            m = pool[pi]
            perm = rng.permutation(m.n_verts).astype(np.int32)
            tv = rng.permuted(perm[m.tv], axis=1).astype(np.int32)
            f = np.empty_like(m.fields[0])
            f[perm] = m.fields[int(rng.integers(0, 4))]
            reqs.append(("mesh", tv, perm, pi, m.n_verts, f))
            tets.append(m.n_cells)
            mesh_reqs.append(r)
    return pool, reqs, tets


def fifo_latencies(arrivals, service):
    """Latencies of one server taking requests in arrival order, one at a
    time: completion_i = max(completion_{i-1}, arrival_i) + service_i."""
    done, out = 0.0, []
    for t, sv in zip(arrivals, service):
        done = max(done, t) + sv
        out.append(done - t)
    return out


def main_serve(args, torch, tg, rank):
    """Serving: Poisson arrivals at swept rates into tg_server (continuous
    batching, 150 GB budget), against the plain per-request path (each request
    alone through tg_mesh_*, resident meshes kept under the same budget).
    Server latency = submission to result ready, measured (queueing
    included).  Plain path: each request's service time measured back to
    back, and its latency under the same arrivals computed as one server taking
    requests in arrival order (queueing included, the same definition)."""
    n_req = args.serve_requests
    t_gen = time.perf_counter()
    pool, reqs, tets = serve_requests(n_req, 256, 2468)
    t_gen = time.perf_counter() - t_gen
    total_tets = int(sum(tets))
    rates = [float(x) for x in args.serve_rates.split(",")]
    results = {}
    arrivals = {}
    for rate in rates:
        rng = np.random.default_rng(int(rate))
        gaps = rng.exponential(1.0 / rate, size=n_req)
        arrivals[rate] = np.cumsum(gaps)
        with tg.Server(n_slots=4, hbm_budget_bytes=150 * 10**9) as srv:
            rid, mid = [None] * n_req, [None] * n_req
            t0 = time.perf_counter()
            t_next = t0
            for k, q in enumerate(reqs):
                t_next += gaps[k]
                while time.perf_counter() < t_next:
                    pass
                if q[0] == "mesh":
                    rid[k], mid[k] = srv.submit_mesh(q[1], q[4], q[5])
                else:
                    rid[k] = srv.submit_field(mid[q[1]], q[2])
            lat = []
            for k in range(n_req):
                lat.append(srv.wait(rid[k])[1])
            wall = time.perf_counter() - t0
            st = srv.stats()
        results[str(int(rate))] = {
            "offered_req_per_s": rate, "p50_ms": round(float(np.percentile(lat, 50)), 3),
            "p99_ms": round(float(np.percentile(lat, 99)), 3),
            "mtets_per_s": round(total_tets / wall / 1e6, 3), "wall_s": round(wall, 3),
            "batches": st["batches"], "meshes_built": st["meshes_built"],
            "evictions": st["evictions"], "peak_gb": round(st["peak_bytes"] / 1e9, 2)}

    # plain per-request path: one request at a time, back to back (service times)
    budget = 150 * 10**9
    resident, used, order = {}, 0, []
    service = []
    stream = torch.cuda.Stream()
    s = stream.cuda_stream
    t0 = time.perf_counter()
    for k, q in enumerate(reqs):
        t1 = time.perf_counter()
        if q[0] == "mesh":
            g = tg.Mesh(q[1], q[4], stream=s)
            g.extract(tg.ALL_RELATIONS, options=tg.OPT_LINK_ADJACENCY, stream=s)
            g.critical_points(q[5], stream=s)
            b = g.device_bytes()
            while order and used + b > budget:
                old = order.pop(0)
                used -= resident[old][1]
                resident[old][0].close()
                resident[old] = None
            resident[k] = (g, b)
            order.append(k)
            used += b
        else:
            mq = reqs[q[1]]
            if resident.get(q[1]) is None:  # evicted: rebuild
                g = tg.Mesh(mq[1], mq[4], stream=s)
                g.extract(tg.ALL_RELATIONS, options=tg.OPT_LINK_ADJACENCY, stream=s)
                resident[q[1]] = (g, g.device_bytes())
                order.append(q[1])
                used += resident[q[1]][1]
            resident[q[1]][0].critical_points(q[2], stream=s)
        service.append(time.perf_counter() - t1)
    plain_wall = time.perf_counter() - t0
    for v in resident.values():
        if v is not None:
            v[0].close()
    svc_ms = [x * 1e3 for x in service]
    plain = {"service_p50_ms": round(float(np.percentile(svc_ms, 50)), 3),
             "service_p99_ms": round(float(np.percentile(svc_ms, 99)), 3),
             "mtets_per_s": round(total_tets / plain_wall / 1e6, 3),
             "wall_s": round(plain_wall, 3), "under_arrivals": {}}
    for rate in rates:
        fl = [x * 1e3 for x in fifo_latencies(arrivals[rate], service)]
        plain["under_arrivals"][str(int(rate))] = {
            "p50_ms": round(float(np.percentile(fl, 50)), 3),
            "p99_ms": round(float(np.percentile(fl, 99)), 3)}
    if rank == 0:
        top = results[str(int(rates[-1]))]
        line = {
            "metric": METRIC, "value": top["mtets_per_s"], "unit": UNIT, "n_gpus": 1,
            "steps": 1, "warmup": 0, "ms_per_step": round(top["wall_s"] * 1e3, 3),
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "int32",
            "data": "synthetic",
            "config": {"workload": WORKLOADS["serve"], "requests": n_req,
                       "mesh_requests": sum(1 for q in reqs if q[0] == "mesh"),
                       "grid_pool": len(pool), "tets_requested": total_tets, "budget_gb": 150,
                       "slots": 4, "generation_s": round(t_gen, 1),
                       "meshes": "every mesh request a distinct mesh: a pool grid relabelled "
                                 "and slot-shuffled with its own seed",
                       "latency": "server: submission to result ready (queueing included); "
                                  "plain: measured service times, latency under the same "
                                  "arrivals as one server in arrival order"},
            "serving": results, "plain_per_request": plain,
            "p99_ms": top["p99_ms"], "p50_ms": top["p50_ms"],
        }
        if not args.no_cpu_baseline:
            line["cpu_baseline"] = cpu_baseline(load_workload("large")[1], WORKLOADS["large"])
        print(json.dumps(line), flush=True)


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=None)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="tetragpu", choices=["tetragpu", "reference"])
    ap.add_argument("--e2e-steps", type=int, default=8)
    ap.add_argument("--workload", default="large", choices=sorted(WORKLOADS))
    ap.add_argument("--batch-steps", type=int, default=3,
                    help="timed steps of the 512-mesh batch leg beside the large mesh (0: skip)")
    ap.add_argument("--serve-requests", type=int, default=10000)
    ap.add_argument("--serve-rates", default="500,2000,8000,32000",
                    help="offered request rates (per second) for --workload serve")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    args = ap.parse_args()
    if args.steps is None:
        args.steps = 20 if args.impl == "reference" else DEFAULT_STEPS[args.workload]
    if args.impl == "reference":
        if args.workload in ("batch", "serve"):
            args.workload = "large"
        run_reference(args)
        return

    import torch
    import torch.distributed as dist

    rank, local_rank, world = env_rank()
    torch.cuda.set_device(local_rank)
    if world > 1:
        dist.init_process_group("nccl", device_id=torch.device("cuda", local_rank))

    import tetragpu_gb300 as tg
    from tetragpu_gb300 import _build
    if not os.path.exists(_build.LIB):
        _build.build()
    tg.load()

    if args.workload == "serve":
        main_serve(args, torch, tg, rank)
        if world > 1:
            dist.destroy_process_group()
        return
    if args.workload == "batch":
        main_batch(args, torch, dist, tg, rank, local_rank, world)
        if world > 1:
            dist.destroy_process_group()
        return
    # the batch leg first: its per-mesh loop makes thousands of small
    # allocations and launches, which the single-mesh e2e leg's pinned
    # buffers would slow down
    b = None
    if args.workload == "large" and args.batch_steps > 0:
        b = run_batch(args, torch, dist, tg, rank, local_rank, world, args.batch_steps, 0)
        torch.cuda.synchronize()
    line = run_single(args, torch, dist, tg, rank, local_rank, world)
    if b is not None:
        if rank == 0:
            line["batch"] = {
                "workload": b["config"]["workload"], "meshes": b["config"]["meshes"],
                "cells": b["config"]["cells"], "value": b["value"], "unit": UNIT,
                "ms_per_step": b["ms_per_step"], "steps": b["steps"],
                "gpu_launches": b["gpu_launches"], "per_mesh_loop": b["per_mesh_loop"],
                "batched_over_loop": b["batched_over_loop"], "tuning": b["tuning"],
                "roofline": b["roofline"], "clocks": b["clocks"]}
            line["gpu_launches_batch_leg"] = b["gpu_launches"] + \
                b["per_mesh_loop"]["gpu_launches"]
    if rank == 0:
        if not args.no_cpu_baseline:
            _, mesh = load_workload(args.workload)
            line["cpu_baseline"] = cpu_baseline(mesh, line["config"]["workload"])
        print(json.dumps(line), flush=True)
    if world > 1:
        dist.destroy_process_group()


def run_single(args, torch, dist, tg, rank, local_rank, world):
    """One mesh per step (device-resident value, host-buffer e2e); returns the
    JSON line (rank 0) without the CPU baseline."""
    workload, mesh = load_workload(args.workload)
    T, V = mesh.n_cells, mesh.n_verts
    dev = f"cuda:{local_rank}"
    stream = torch.cuda.Stream()
    s = stream.cuda_stream
    d_tv = torch.from_numpy(mesh.tv).to(dev)
    d_field = torch.from_numpy(mesh.field).to(dev)
    d_classes = torch.empty(3 * V, dtype=torch.int32, device=dev)
    flush = torch.empty(512 << 20, dtype=torch.uint8, device=dev)
    torch.cuda.synchronize()

    def step():
        with tg.Mesh(d_tv.data_ptr(), V, n_cells=T, on_device=True, stream=s) as g:
            g.extract(tg.ALL_RELATIONS, options=tg.OPT_LINK_ADJACENCY, stream=s)
            g.critical_points(d_field.data_ptr(), on_device=True, out_ptr=d_classes.data_ptr(),
                              stream=s)
            info = {"counts": g.counts()}
            for n in ("ET", "EF", "VT", "TT", "FF", "EE", "VV"):
                info[n] = g.device_relation(n)["n_entries"]
        return info

    with torch.cuda.stream(stream):
        for _ in range(max(3, args.warmup)):
            info = step()
    torch.cuda.synchronize()
    Vc, E, F, Tc = info["counts"]
    counts = {"V": Vc, "E": E, "F": F, "T": Tc}
    totals = {n: info[n] for n in ("ET", "EF", "VT", "TT", "FF", "EE", "VV")}

    # ---- timed region: device-resident inputs ----
    clocks = Clocks(local_rank)
    tg.profile_kernel(ROOFLINE_KERNEL)
    tg.profile_read(reset=True)
    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True))
          for _ in range(args.steps)]
    if world > 1:
        dist.barrier()
    torch.cuda.synchronize()
    clocks.start()
    launches0 = tg.kernel_launch_count()
    wall0 = time.perf_counter()
    with torch.cuda.stream(stream):
        for k in range(args.steps):
            flush.fill_(k & 0xff)          # evict L2 (outside the timed window)
            ev[k][0].record(stream)
            step()
            ev[k][1].record(stream)
    torch.cuda.synchronize()
    wall = time.perf_counter() - wall0
    launches = tg.kernel_launch_count() - launches0
    clk = clocks.stop()
    kern_ms, kern_n = tg.profile_read(reset=True)
    tg.profile_kernel(None)
    ms = [a.elapsed_time(b) for a, b in ev]
    total_s = sum(ms) / 1e3
    t_max = total_s
    if world > 1:
        t_max = max_over_ranks(total_s, dist, torch, dev)
        dist.barrier()
    value = world * args.steps * T / t_max / 1e6

    # ---- e2e: host buffers through the C ABI ----
    # Each step: tg_mesh_create from the pinned host TV (the library copies it
    # in), tg_extract, tg_critical_points from the pinned host field (copied
    # in by the library) into device classes, then every relation and the
    # classes out to pinned host memory.  Steps alternate between two streams
    # and two sets of host buffers, so one step's copies back (host-link
    # bound) overlap the next step's extraction, the way a caller processing
    # many meshes would run; the timed region covers every copy of every step.
    pin_tv = torch.from_numpy(mesh.tv).pin_memory()
    pin_field = torch.from_numpy(mesh.field).pin_memory()
    names = tg.RELATIONS[1:]
    fixed_rows = {"TE": (Tc, 6), "EV": (E, 2), "TF": (Tc, 4), "FV": (F, 3), "FE": (F, 3),
                  "FT": (F, 2)}
    csr_rows = {"ET": E, "EF": E, "VT": Vc, "TT": Tc, "FF": F, "EE": E, "VV": Vc}
    lib = tg.load()
    Cc = tg._lib.C
    e2e_value, h2d, d2h = None, 0, 0
    if args.e2e_steps > 0:
        bufs = []
        for _ in range(2):
            h_ent = {n: torch.empty(max(r * w, 1), dtype=torch.int32).pin_memory()
                     for n, (r, w) in fixed_rows.items()}
            h_ent.update({n: torch.empty(max(totals[n], 1), dtype=torch.int32).pin_memory()
                          for n in csr_rows})
            h_off = {n: torch.empty(r + 1, dtype=torch.int32).pin_memory()
                     for n, r in csr_rows.items()}
            h_cls = torch.empty(3 * V, dtype=torch.int32).pin_memory()
            bufs.append((h_ent, h_off, h_cls))
        ptr_off, ptr_ent = [], []
        for h_ent, h_off, _ in bufs:
            po, pe = (Cc.c_void_p * 14)(), (Cc.c_void_p * 14)()
            for n in names:
                pe[tg.REL[n]] = h_ent[n].data_ptr()
                if n in h_off:
                    po[tg.REL[n]] = h_off[n].data_ptr()
            ptr_off.append(po)
            ptr_ent.append(pe)
        h2d = pin_tv.numel() * 4 + pin_field.numel() * 4
        d2h = sum(r * w * 4 for r, w in fixed_rows.values()) + \
            sum(totals[n] * 4 for n in csr_rows) + sum((r + 1) * 4 for r in csr_rows.values()) + \
            V * 12
        e_streams = [torch.cuda.Stream(), torch.cuda.Stream()]
        d_cls2 = [torch.empty(3 * V, dtype=torch.int32, device=dev) for _ in range(2)]

        def e2e_run(n_steps):
            live = None
            for k in range(n_steps):
                es = e_streams[k % 2].cuda_stream
                h_ent, h_off, h_cls = bufs[k % 2]
                h = Cc.c_void_p()
                tg._lib.check(lib.tg_mesh_create(pin_tv.data_ptr(), T, V, 0, es, Cc.byref(h)))
                tg._lib.check(lib.tg_extract(h, tg.ALL_RELATIONS, tg.OPT_LINK_ADJACENCY, es))
                tg._lib.check(lib.tg_critical_points(h, pin_field.data_ptr(), tg.FIELD_F32, 0,
                                                     d_cls2[k % 2].data_ptr(), 1, es))
                # every relation through one call: CSR offsets narrowed to
                # int32 by one launch, then the copies back to back
                tg._lib.check(lib.tg_copy_relations_async_i32(h, tg.ALL_RELATIONS,
                                                              ptr_off[k % 2], ptr_ent[k % 2], es))
                with torch.cuda.stream(e_streams[k % 2]):
                    h_cls.copy_(d_cls2[k % 2], non_blocking=True)
                if live is not None:
                    lib.tg_mesh_destroy(live)   # waits for the previous step's copies
                live = h
            if live is not None:
                lib.tg_mesh_destroy(live)
            torch.cuda.synchronize()

        e2e_run(2)
        if world > 1:
            dist.barrier()
        t0 = time.perf_counter()
        e2e_run(args.e2e_steps)
        e2e_s = time.perf_counter() - t0
        if world > 1:
            e2e_s = max_over_ranks(e2e_s, dist, torch, dev)
        e2e_value = round(world * args.e2e_steps * T / e2e_s / 1e6, 3)

    if rank != 0:
        return None
    peak, peak_kind = peaks()
    step_s = t_max / args.steps
    alg = output_bytes(counts, totals)
    path_gbs = alg / step_s / 1e9
    kb = kernel_bytes(ROOFLINE_KERNEL, counts, totals)
    per_launch_s = (kern_ms / 1e3) / max(kern_n, 1)
    k_gbs = kb / per_launch_s / 1e9 if kern_n else None
    return {
        "metric": METRIC, "value": round(value, 3), "unit": UNIT, "n_gpus": world,
        "steps": args.steps, "warmup": max(3, args.warmup),
        "ms_per_step": round(1e3 * step_s, 4), "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "int32", "data": "synthetic",
        "config": {"workload": workload, "cells": T, "vertices": V, "edges": E, "faces": F,
                   "relations": "all 13 + critical points", "parallelism": f"replicas{world}",
                   "l2": "flushed before every step (512 MB write)",
                   "step": "tg_mesh_create + tg_extract(all 13, link adjacency) + "
                           "tg_critical_points + tg_mesh_destroy"},
        "gpu_launches": int(launches),
        "wall_s": round(wall, 3),
        "clocks": clk,
        "e2e": {"value": e2e_value, "unit": UNIT, "h2d_bytes_per_step": int(h2d),
                "d2h_bytes_per_step": int(d2h), "steps": args.e2e_steps,
                "path": "C ABI with host buffers: tg_mesh_create(host TV), tg_extract, "
                        "tg_critical_points(host field), tg_copy_relations_async_i32"},
        "roofline": {
            "bound": "hbm", "scope": "path (one step: every kernel of create + extract + "
                                     "critical points)",
            "achieved": round(path_gbs, 1), "peak": peak, "unit": "GB/s",
            "frac": round(path_gbs / peak, 4), "peak_source": peak_kind,
            "algorithmic_bytes_per_step": alg,
            "traffic": traffic_from_profiles("path", workload, T, "dram_bytes_per_step"),
            "kernel": {"name": ROOFLINE_KERNEL, "achieved": round(k_gbs, 1) if k_gbs else None,
                       "frac": round(k_gbs / peak, 4) if k_gbs else None,
                       "algorithmic_bytes_per_launch": kb,
                       "launch_ms": round(per_launch_s * 1e3, 4), "launches": kern_n,
                       "traffic": traffic_from_profiles(ROOFLINE_KERNEL, workload, T)},
        },
    }


if __name__ == "__main__":
    main()
