"""Benchmark: closest-hit Mrays/s of the BVH hot path on one B200 (or N replicas).

Workload (the reference's soup configuration): LBVH + 3 treelet rounds over a seeded
1,000,000-triangle FP32 soup; each step traces 4,194,304 closest-hit rays (origins
uniform in [-0.1,1.1]^3, directions uniform on the sphere, tmax = inf) against the
resident BVH, in the exact mode, traced in the Morton order of the ray origins
(CAV_TRACE_REORDER: the sort and the write-back of every ray's results to its own index
are inside the timed step; the hits equal those of the given order, which is timed too).
`value` is device-timed closest-hit Mrays/s with rays already in HBM (L2 flushed between
steps); `e2e` is the same metric through the C ABI's host-buffer entry point (pinned host
rays in, hits out, copies inside the timed region).

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

N > 1 runs under torchrun: every rank builds its own replica and traces its own rays
(the path has no exchange step), time is the max over ranks.  `--impl reference` times
the reference algorithm on the host cores (the C oracle port of BVH::build and
BVH::intersect, all OpenMP threads) on a bounded sample of the same workload.
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

N_TRI = 1_000_000
N_RAYS = 4 * 1024 * 1024
ROUNDS = 3
METRIC = "closest-hit Mrays/s"
UNIT = "Mrays/s"
WORKLOAD = "soup_1M_tris_3_treelet_rounds_4M_closest_rays"
RAY_BYTES = 32
HIT_BYTES = 16  # prim id 4 + t 4 + uv 8
# algorithmic traversal bytes per ray: ray 32 B + hit 16 B, plus 64 B per node visited and
# 36 B (three float3 vertices) per triangle tested, counted by the instrumented kernel
NODE_BYTES = 64
TRI_BYTES = 36
WIDE_NODE_BYTES = 96  # node of the compressed 8-wide view (the fast mode)


def parse():
    p = argparse.ArgumentParser()
    p.add_argument("--gpus", type=int, default=1)
    p.add_argument("--steps", type=int, default=20)
    p.add_argument("--warmup", type=int, default=5)
    p.add_argument("--impl", default="ours", choices=["ours", "reference"])
    p.add_argument("--no-cpu-baseline", action="store_true")
    p.add_argument("--launch-shape", default=None,
                   help="soup workload: BLOCK,CHUNK[,SMEM_STACK] for the exact traversal instead of the "
                        "autotuner's pick")
    p.add_argument("--no-reference-cuda", action="store_true",
                   help="soup workload: skip the reference CUDA timings and the config-1 block")
    p.add_argument("--workload", default="soup",
                   choices=["soup", "render", "serve", "guided", "mlp", "capture", "batch"],
                   help="soup: BVH + 4M closest-hit rays (default); render: the 5.24M-triangle path-traced scene; "
                        "serve: a Poisson stream of render and ray-query jobs, merged server vs sequential loop")
    p.add_argument("--jobs", type=int, default=256, help="jobs in the served stream (serve workload)")
    p.add_argument("--serve-trace", default="fast", choices=["fast", "exact"], help="serve workload: traversal mode")
    p.add_argument("--serve-loaders", type=int, default=8, help="serve workload: the server's scene loader threads")
    p.add_argument("--serve-lanes", default="8",
                   help="serve workload: the server's lanes; a comma list runs the server arm once per value "
                        "(the first value is the bench's `value`)")
    p.add_argument("--bounce", type=int, default=1, help="capture workload: which bounce's extend rays")
    p.add_argument("--ref-spp", type=int, default=16384, help="guided workload: spp of the reference render")
    p.add_argument("--no-reference", action="store_true", help="render workload: skip the reference's CUDA build")
    p.add_argument("--render-steps", type=int, default=1, help="timed full renders (render workload)")
    p.add_argument("--small", action="store_true", help="render workload at 1/16 size (smoke runs)")
    p.add_argument("--tris", type=int, default=None, help="soup size (default: the 1M-triangle workload)")
    p.add_argument("--rays", type=int, default=None, help="rays per step (default: 4M)")
    a = p.parse_args()
    g = globals()
    if a.tris or a.rays:  # a smaller case of the same kernels (profiling)
        g["N_TRI"] = a.tris or N_TRI
        g["N_RAYS"] = a.rays or N_RAYS
        g["WORKLOAD"] = f"soup_{g['N_TRI']}_tris_3_treelet_rounds_{g['N_RAYS']}_closest_rays"
    return a


class ClockSampler:
    """nvidia-smi clocks/throttle reasons sampled every 200 ms during the timed region."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device: int):
        self.device = device
        self.proc = None
        self.path = Path(os.environ.get("TMPDIR", "/tmp")) / f"cav_clocks_{os.getpid()}.csv"

    def start(self):
        try:
            self.f = open(self.path, "w")
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--id={self.device}", f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits",
                 "-lms", "200"], stdout=self.f, stderr=subprocess.DEVNULL)
        except (FileNotFoundError, OSError):
            self.proc = None

    def stop(self):
        if self.proc is None:
            return None
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        self.f.close()
        rows = [r.split(",") for r in self.path.read_text().splitlines() if r.strip()]
        self.path.unlink(missing_ok=True)
        if not rows:
            return None
        sm = [float(r[1]) for r in rows if r[1].strip().replace(".", "").isdigit()]
        smax = [float(r[2]) for r in rows if r[2].strip().replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = set()
        for r in rows:
            for k, name in enumerate(names):
                if len(r) > 5 + k and r[5 + k].strip() == "Active":
                    reasons.add(name)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(smax) if smax else None,
                "reasons": sorted(reasons), "samples": len(rows)}


def measured_peaks():
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        d = json.loads(p.read_text())
        return float(d["hbm_gbs"]), "measured"
    return 6650.0, "fallback"


def committed_profile():
    """The committed ncu summary of the closest-hit kernel on this workload ({} if absent)."""
    p = ROOT / "profiles" / "trace_closest_soup1m.json"
    return json.loads(p.read_text()) if p.exists() else {}


# ------------------------------------------------------------------------- ours
def run_ours(args):
    import torch
    import torch.distributed as dist

    import cavalry_b200 as cav
    from cavalry_b200 import scenes

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if world > 1:
        from datetime import timedelta

        torch.cuda.set_device(local)
        dist.init_process_group("nccl", timeout=timedelta(seconds=120), device_id=torch.device("cuda", local))
    else:
        torch.cuda.set_device(0)
    dev = torch.device("cuda", local if world > 1 else 0)

    def barrier():
        if world > 1:
            dist.barrier()

    ctx = cav.Context(dev.index)
    pos, idx = scenes.soup(N_TRI, seed=2)
    d_pos = torch.from_numpy(pos).to(dev)
    d_idx = torch.from_numpy(idx).to(dev)

    # build throughput (secondary): full build incl. 3 treelet rounds, device events
    builds_ms = []
    stage = None
    for k in range(4):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        b = ctx.build(d_pos, d_idx, rounds=ROUNDS)
        e1.record()
        torch.cuda.synchronize()
        if k > 0:
            builds_ms.append(e0.elapsed_time(e1))
            stage = b.stage_times()
        b.free()
    bvh = ctx.build(d_pos, d_idx, rounds=ROUNDS)
    torch.cuda.synchronize()
    ctx.sync_check()

    rays_np = scenes.closest_rays(N_RAYS, seed=20 + rank)
    rays = torch.from_numpy(rays_np).to(dev)
    prim = torch.empty(N_RAYS, dtype=torch.int32, device=dev)
    tt = torch.empty(N_RAYS, dtype=torch.float32, device=dev)
    uv = torch.empty((N_RAYS, 2), dtype=torch.float32, device=dev)
    out = (prim, tt, uv)
    # launch shape picked by the project's autotuner on a separate 4M-ray sample
    if args.launch_shape:
        vals = [int(x) for x in args.launch_shape.split(",")]
        blk, chunk, smem = vals[0], vals[1], (vals[2] if len(vals) > 2 else 0)
        ctx.set_trace_config(blk, 0, chunk)
        ctx.set_trace_stack(128, smem, flags=cav.TRACE_EXACT)
        tuned = {"block_threads": blk, "batch": chunk, "stack": 128, "smem_stack": smem, "picked_by": "--launch-shape"}
    else:
        # tuned on a separate sample of the step's size in the given order: a 1M-ray sample,
        # whose launches end in a relatively longer tail, picked shapes 0.2-4 % slower on the
        # 4M step (the local-memory stack, or 128 x 16 when tuned on reordered rays)
        tune_rays = torch.from_numpy(scenes.closest_rays(N_RAYS, seed=90 + rank)).to(dev)
        tuned = bvh.autotune(tune_rays)
        del tune_rays
    nodes_v, tris_t = bvh.trace_stats(rays)
    nodes_per_ray = nodes_v / N_RAYS
    tris_per_ray = tris_t / N_RAYS
    flush = torch.empty(256 * 1024 * 1024 // 4, dtype=torch.float32, device=dev)  # 256 MiB > 126 MB L2

    # The batch is traced in the Morton order of its ray origins (CAV_TRACE_REORDER: key,
    # sort, gather, traversal and scatter back, all inside each timed step); the results are
    # those of the given order, which is also timed below.
    flags = cav.TRACE_EXACT | cav.TRACE_REORDER
    for _ in range(args.warmup):
        bvh.trace_closest(rays, flags=flags, out=out)
    torch.cuda.synchronize()

    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(args.steps)]
    clocks = ClockSampler(dev.index)
    barrier()
    torch.cuda.synchronize()
    clocks.start()
    t_wall0 = time.perf_counter()
    for k in range(args.steps):
        flush.fill_(float(k))
        ev[k][0].record()
        bvh.trace_closest(rays, flags=flags, out=out)
        ev[k][1].record()
    torch.cuda.synchronize()
    barrier()
    wall = time.perf_counter() - t_wall0
    clk = clocks.stop()
    step_ms = [a.elapsed_time(b) for a, b in ev]
    total_ms = sum(step_ms)
    if world > 1:
        tm = torch.tensor([total_ms], dtype=torch.float64, device=dev)
        dist.all_reduce(tm, op=dist.ReduceOp.MAX)
        total_ms = float(tm.item())
    ctx.sync_check()
    ms_per_step = total_ms / args.steps
    value = N_RAYS * world / (ms_per_step * 1e-3) / 1e6
    # the same rays in the given order (secondary)
    out_g = (torch.empty_like(prim), torch.empty_like(tt), torch.empty_like(uv))
    bvh.trace_closest(rays, out=out_g)
    given_ms = []
    for k in range(3):
        flush.fill_(float(k))
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        bvh.trace_closest(rays, out=out_g)
        b.record()
        torch.cuda.synchronize()
        given_ms.append(a.elapsed_time(b))
    assert all(torch.equal(x, y) for x, y in zip(out, out_g)), "reordered and given-order results differ"
    given_value = N_RAYS / (statistics.mean(given_ms) * 1e-3) / 1e6

    # any-hit (secondary)
    srays_np, lim_np = scenes.shadow_rays(N_RAYS, seed=21 + rank)
    srays = torch.from_numpy(srays_np).to(dev)
    lim = torch.from_numpy(lim_np).to(dev)
    occ = torch.empty(N_RAYS, dtype=torch.uint8, device=dev)
    for _ in range(2):
        bvh.trace_any(srays, lim, out=occ)
    any_ms = []
    for k in range(max(3, args.steps // 2)):
        flush.fill_(float(k))
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        bvh.trace_any(srays, lim, out=occ)
        b.record()
        torch.cuda.synchronize()
        any_ms.append(a.elapsed_time(b))

    # the compressed 8-wide fast mode on the same rays (secondary): same closest-hit
    # distances, a different triangle only at an equal-distance tie
    tuned_fast = bvh.autotune(torch.from_numpy(scenes.closest_rays(N_RAYS, seed=90 + rank)).to(dev),
                              flags=cav.TRACE_FAST)
    fnodes, ftris = bvh.trace_stats(rays, flags=cav.TRACE_FAST)
    fout = (torch.empty_like(prim), torch.empty_like(tt), torch.empty_like(uv))
    for _ in range(2):
        bvh.trace_closest(rays, flags=cav.TRACE_FAST, out=fout)
    fast_ms = []
    for k in range(args.steps):
        flush.fill_(float(k))
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        bvh.trace_closest(rays, flags=cav.TRACE_FAST, out=fout)
        b.record()
        torch.cuda.synchronize()
        fast_ms.append(a.elapsed_time(b))
    same_id = float((fout[0] == prim).float().mean().item())
    same_t = bool(torch.equal(fout[1][prim >= 0], tt[prim >= 0]))
    # the fast mode with the rays traced in the Morton order of their origins: the same hits
    fro = (torch.empty_like(prim), torch.empty_like(tt), torch.empty_like(uv))
    for _ in range(2):
        bvh.trace_closest(rays, flags=cav.TRACE_FAST | cav.TRACE_REORDER, out=fro)
    fast_ro_ms = []
    for k in range(args.steps):
        flush.fill_(float(k))
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        bvh.trace_closest(rays, flags=cav.TRACE_FAST | cav.TRACE_REORDER, out=fro)
        b.record()
        torch.cuda.synchronize()
        fast_ro_ms.append(a.elapsed_time(b))
    assert all(torch.equal(x, y) for x, y in zip(fro, fout)), "reordered fast-mode hits differ"
    del fro
    fany_ms = []
    for k in range(max(3, args.steps // 2)):
        flush.fill_(float(k))
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        bvh.trace_any(srays, lim, flags=cav.TRACE_FAST, out=occ)
        b.record()
        torch.cuda.synchronize()
        fany_ms.append(a.elapsed_time(b))
    ctx.sync_check()
    fast_ms_step = statistics.mean(fast_ms)
    fast_bytes = RAY_BYTES + HIT_BYTES + WIDE_NODE_BYTES * fnodes / N_RAYS + TRI_BYTES * ftris / N_RAYS

    # e2e through the host-buffer C-ABI entry point (pinned host memory)
    h_rays = torch.from_numpy(rays_np).pin_memory()
    h_prim = torch.empty(N_RAYS, dtype=torch.int32).pin_memory()
    h_t = torch.empty(N_RAYS, dtype=torch.float32).pin_memory()
    h_uv = torch.empty((N_RAYS, 2), dtype=torch.float32).pin_memory()
    hout = (h_prim, h_t, h_uv)
    for _ in range(2):
        bvh.trace_closest_host(h_rays, flags=flags, out=hout)
    barrier()
    torch.cuda.synchronize()
    e2e_ms = []
    for k in range(args.steps):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        bvh.trace_closest_host(h_rays, flags=flags, out=hout)
        b.record()
        torch.cuda.synchronize()
        e2e_ms.append(a.elapsed_time(b))
    e2e_total = sum(e2e_ms)
    if world > 1:
        tm = torch.tensor([e2e_total], dtype=torch.float64, device=dev)
        dist.all_reduce(tm, op=dist.ReduceOp.MAX)
        e2e_total = float(tm.item())
    assert np.array_equal(h_prim.numpy(), prim.cpu().numpy()), "host-buffer path disagrees with device path"
    e2e_value = N_RAYS * world / (e2e_total / args.steps * 1e-3) / 1e6

    peak, peak_kind = measured_peaks()
    # so many closest hits on so dense a tree take the binary traversal (wide.cu, view_use)
    bytes_per_ray = RAY_BYTES + HIT_BYTES + NODE_BYTES * nodes_per_ray + TRI_BYTES * tris_per_ray
    achieved = bytes_per_ray * N_RAYS / (ms_per_step * 1e-3) / 1e9
    prof = committed_profile()
    traffic = prof.get("dram_bytes_per_launch")

    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        cpu = cpu_baseline(bvh, pos, idx, rays_np)
    ref_cuda = cfg1 = None
    if rank == 0 and world == 1 and not args.no_reference_cuda:
        try:
            ref_cuda = reference_cuda_block(ctx, d_pos, d_idx, pos, idx, bvh, rays_np, round(value, 2), tuned,
                                            round(given_value, 2))
        except Exception as e:  # a reported baseline: note the failure, keep the bench line
            ref_cuda = {"error": str(e)[:300]}
        cfg1 = config1_block(ctx)

    result = {
        "metric": METRIC,
        "value": round(value, 2),
        "unit": UNIT,
        "n_gpus": world,
        "steps": args.steps,
        "warmup": args.warmup,
        "ms_per_step": round(ms_per_step, 4),
        "higher_is_better": True,
        "scaling": "weak",
        "vs_baseline": None,
        "dtype": "f32",
        "data": "synthetic (seeded triangle soup and rays, generated in-process)",
        "config": {
            "workload": WORKLOAD,
            "triangles": N_TRI,
            "rays_per_step": N_RAYS,
            "treelet_rounds": ROUNDS,
            "trace_mode": "exact (reference order and pruning)",
            "ray_order": "Morton order of the ray origins (CAV_TRACE_REORDER): keys, sort, gather, traversal and "
                         "scatter of the results back to each ray's index inside every timed step",
            "launch_shape": {"block": tuned["block_threads"], "queue_chunk": tuned["batch"], "stack": tuned["stack"],
                             "smem_stack": tuned.get("smem_stack", 0),
                             "picked_by": tuned.get("picked_by", "cav_trace_autotune on a separate 4M-ray sample")},
            "l2": "flushed between timed steps (256 MiB write); rays 128 MiB > L2",
            "parallelism": f"replicas x{world}",
        },
        "gpu_launches": args.steps * 9,  # per step: keys, histogram, 4 sort passes, gather, traversal, scatter
        "given_order_mrays_s": round(given_value, 2),
        "e2e": {"value": round(e2e_value, 2), "unit": UNIT, "h2d_bytes_per_step": N_RAYS * RAY_BYTES,
                "d2h_bytes_per_step": N_RAYS * HIT_BYTES},
        "roofline": {
            # The node-fetch stream is measured against the HBM copy peak (the algorithmic
            # bytes of the scope table), but with the rays in Morton order nearly all of it is
            # served by L2 and DRAM carries well under a percent of the peak: the kernel is
            # bound by the L1 data pipe's wavefronts (one per lane per 32-byte node half,
            # ncu), not by HBM, and that pipe's rate is the fraction to read.  The time is the
            # whole step's (sort included).
            "bound": "l1/l2",
            "achieved": round(achieved, 1),
            "peak": peak,
            "unit": "GB/s",
            "frac": round(achieved / peak, 4),
            "traffic": traffic,
            "peak_kind": peak_kind,
            "dram_frac": (round(traffic / (ms_per_step * 1e-3) / 1e9 / peak, 4) if traffic else None),
            "l1_data_pipe_wavefronts_pct": prof.get("l1_data_pipe_lsu_wavefronts_pct"),
            "l1tex_throughput_pct": prof.get("l1tex_throughput_pct"),
            "lts_throughput_pct": prof.get("lts_throughput_pct"),
            "l2_hit_rate_pct": prof.get("l2_hit_rate_pct"),
            "algorithmic_bytes_per_ray": round(bytes_per_ray, 2),
            "nodes_per_ray": round(nodes_per_ray, 3),
            "tris_per_ray": round(tris_per_ray, 3),
            "kernel": "k_closest (binary nodes, 64 B)",
        },
        "clocks": clk,
        "anyhit_mrays_s": round(N_RAYS / (statistics.mean(any_ms) * 1e-3) / 1e6, 2),
        "fast_mode": {
            "closest_mrays_s": round(N_RAYS / (fast_ms_step * 1e-3) / 1e6, 2),
            "closest_reordered_mrays_s": round(N_RAYS / (statistics.mean(fast_ro_ms) * 1e-3) / 1e6, 2),
            "anyhit_mrays_s": round(N_RAYS / (statistics.mean(fany_ms) * 1e-3) / 1e6, 2),
            "same_prim_frac": round(same_id, 6), "same_t_on_hits": same_t,
            "wide_nodes_per_ray": round(fnodes / N_RAYS, 3), "tris_per_ray": round(ftris / N_RAYS, 3),
            "algorithmic_bytes_per_ray": round(fast_bytes, 2),
            "achieved_gbs": round(fast_bytes * N_RAYS / (fast_ms_step * 1e-3) / 1e9, 1),
            "launch_shape": {"block": tuned_fast["block_threads"], "queue_chunk": tuned_fast["batch"],
                             "smem_stack": tuned_fast.get("smem_stack", 0)},
            "kernel": "k_trace_wide<closest> (compressed 8-wide nodes, 96 B)",
        },
        "build": {
            "ms": round(statistics.mean(builds_ms), 3),
            "builds_per_s": round(1000.0 / statistics.mean(builds_ms), 2),
            # algorithmic bytes: ~390 B per triangle for the LBVH stages (vertices in, codes,
            # 6 sort passes, radix tree, refit, node write) plus, per treelet round, every
            # node read and written once (2N-1 x 128 B); latency-bound, so far below HBM
            "algorithmic_bytes": int(390 * N_TRI + ROUNDS * (2 * N_TRI - 1) * 128),
            "achieved_gbs": round((390 * N_TRI + ROUNDS * (2 * N_TRI - 1) * 128)
                                  / (statistics.mean(builds_ms) * 1e-3) / 1e9, 1),
            "stage_ms": {k: round(v, 4) for k, v in zip(
                ["boxes_morton", "sort", "radix_tree", "refit", "treelet_rounds", "layout"], stage)},
        },
        "wall_s_timed_region": round(wall, 3),
    }
    if cpu is not None:
        result["cpu_baseline"] = cpu
    if ref_cuda is not None:
        result["reference_cuda"] = ref_cuda
    if cfg1 is not None:
        result["config1_mini_room"] = cfg1
    if rank == 0:
        print(json.dumps(result))
    bvh.free()
    ctx.close()
    if world > 1:
        dist.destroy_process_group()


def _oracle_nodes_from_export(nodes):
    from oracle import pyoracle as po

    o = np.zeros(len(nodes), po.ONODE_DTYPE)
    for f in ("bmin", "bmax", "left", "right", "is_leaf"):
        o[f] = nodes[f]
    o["begin"] = nodes["prim_begin"]
    o["end"] = nodes["prim_end"]
    return o


def cpu_baseline(bvh, pos, idx, rays_np, target_s: float = 10.0):
    """The C oracle's BVH::intersect port on all host threads, over the same tree."""
    from oracle import pyoracle as po

    onodes = _oracle_nodes_from_export(bvh.export_nodes())
    m = 1 << 16
    t0 = time.perf_counter()
    po.trace_closest(onodes, pos, idx, rays_np[:m])
    dt = time.perf_counter() - t0
    m2 = int(min(len(rays_np), max(m, m * target_s / max(dt, 1e-3))))
    t0 = time.perf_counter()
    po.trace_closest(onodes, pos, idx, rays_np[:m2])
    dt = time.perf_counter() - t0
    return {"value": round(m2 / dt / 1e6, 3), "unit": UNIT, "cores": po.num_threads(), "kind": "port",
            "sample": f"{m2} of the step's {len(rays_np)} closest-hit rays on the same tree, "
                      f"{dt:.1f} s wall, OpenMP"}


# ------------------------------------------------------- reference CUDA build, config 1
def _median(xs):
    return float(statistics.median(xs))


def reference_cuda_block(ctx, d_pos, d_idx, pos, idx, bvh, rays_np, value, closest_shape, given_value=None):
    """The reference's own CUDA code on this B200 beside ours (a reported baseline, like
    cpu_baseline): its BVH::build (BVH/BVH.cu:317-370, replayed stage by stage with CUDA events
    by oracle/ref_harness.cu, 0 treelet rounds: its treelet kernel faults on the B200) against
    our LBVH build of the same 1M soup; its BVH::intersect (BVH/BVH.h:23-107) on this step's
    rays over our 3-round tree; and, on the 5.24M-triangle icosphere scene at 0 rounds (its
    own LBVH, bit-exact topology with ours), its BVH::intersect against ours on the renderer's
    bounce-0 and bounce-1 extend rays.  Beside them, config 3 as this renderer renders it
    (the whole 1920 x 1080 x 64-spp film of that scene)."""
    import os as _os
    import tempfile

    import torch

    import cavalry_b200 as cav
    from cavalry_b200 import scenes
    from oracle import pyoracle as po

    if not po.ref_available():
        return {"unavailable": "reference harness not built (oracle/_ref/libcavref.so)"}
    out = {}
    # (1) LBVH build of the 1M soup
    ref_ms, ours_ms = [], []
    for k in range(4):
        R = po.RefScene(pos, idx, rounds=0, id_mode=0, dump=False)
        if k > 0:
            ref_ms.append(float(np.sum(R.stage_ms)))
        R.free()
        b = ctx.build(d_pos, d_idx, rounds=0)
        torch.cuda.synchronize()
        if k > 0:
            ours_ms.append(float(np.sum(b.stage_times())))
        b.free()
    out["soup_1M_lbvh_build"] = {
        "ref_ms": round(_median(ref_ms), 3), "ours_ms": round(_median(ours_ms), 3),
        "ref_builds_per_s": round(1e3 / _median(ref_ms), 1), "ours_builds_per_s": round(1e3 / _median(ours_ms), 1),
        "speedup": round(_median(ref_ms) / _median(ours_ms), 2),
        "timing": "device stage times (CUDA events), median of 3; 0 treelet rounds"}
    # (2) closest hit on this step's rays over the 3-round tree, ours loaded into the reference
    R = po.RefScene(pos, idx, rounds=0, id_mode=0, dump=False)
    R.load_nodes(bvh.export_nodes())
    R.trace_closest(rays_np[: 1 << 20], reps=1)
    _, _, ms = R.trace_closest(rays_np, reps=2)
    ref_mrays = len(rays_np) / (ms * 1e-3) / 1e6
    R.free()
    out["soup_1M_closest_3_rounds"] = {"ref_mrays_s": round(ref_mrays, 2), "ours_mrays_s": value,
                                       "ours_given_order_mrays_s": given_value,
                                       "speedup": round(value / ref_mrays, 2), "rays": len(rays_np)}
    # (3) the 5.24M-triangle scene at 0 rounds: closest hit against the reference on its own LBVH
    sc_np = scenes.sphere_scene(64, 6, seed=9)
    tmp = tempfile.mkdtemp()
    path = _os.path.join(tmp, "spheres.pbrt")
    scenes.write_pbrt(path, sc_np, width=1920, height=1080, spp=64, max_depth=8)
    sc = ctx.load_pbrt(path, bvh_rounds=0)
    sc_r = ctx.load_pbrt(path, bvh_rounds=3)  # the same file as this renderer renders it
    _os.remove(path)
    sb = sc.bvh()
    R = po.RefScene(sc_np["positions"], sc_np["indices"], sc_np["mesh_ids"], rounds=0, id_mode=0, dump=False)
    ref_nodes = R.nodes()
    ours_nodes = sb.export_nodes()
    topo = bool(np.array_equal(ref_nodes["left"], ours_nodes["left"]) and
                np.array_equal(ref_nodes["right"], ours_nodes["right"]) and
                np.array_equal(ref_nodes["is_leaf"], ours_nodes["is_leaf"]))
    leaves = ours_nodes["is_leaf"] == 1
    topo = topo and bool(np.array_equal(ref_nodes["begin"][leaves], ours_nodes["prim_begin"][leaves]))
    del ref_nodes, ours_nodes
    rows = {}
    for depth in (0, 1):
        r = sc.capture_rays(depth, capacity=1 << 22)
        r_np = r.cpu().numpy()
        R.trace_closest(r_np[: 1 << 18], reps=1)
        _, _, rms = R.trace_closest(r_np, reps=2)
        ref_v = len(r_np) / (rms * 1e-3) / 1e6
        mine = {}
        for name, fl in (("exact", cav.TRACE_EXACT), ("fast", cav.TRACE_FAST)):
            sb.autotune(r[: 1 << 20].contiguous(), flags=fl)
            for _ in range(2):
                sb.trace_closest(r, flags=fl)
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(3):
                sb.trace_closest(r, flags=fl)
            b.record()
            torch.cuda.synchronize()
            mine[name] = 3 * len(r_np) / (a.elapsed_time(b) * 1e-3) / 1e6
        rows[f"bounce{depth}"] = {"rays": len(r_np), "ref_mrays_s": round(ref_v, 2),
                                  "ours_exact_mrays_s": round(mine["exact"], 2),
                                  "ours_fast_mrays_s": round(mine["fast"], 2),
                                  "speedup_exact": round(mine["exact"] / ref_v, 2),
                                  "speedup_fast": round(mine["fast"] / ref_v, 2)}
    R.free()
    sc.free()
    out["spheres_5M_closest_0_rounds"] = {"triangles": int(len(sc_np["indices"])), "topology_bit_exact": topo, **rows}
    # (4) config 3 rendered whole by this renderer: 1920 x 1080 x 64 spp, depth 8, 3 treelet
    # rounds, fast traversal (device time of the render, median of 2 after a short warm-up)
    sc_r.render(spp=2, fast_trace=True)
    times = [sc_r.render(fast_trace=True)[2] for _ in range(2)]
    ms3 = statistics.median(times)
    samples = 1920 * 1080 * 64
    out["config3_render"] = {"workload": "spheres_5M_1920x1080_64spp_depth8_path", "treelet_rounds": 3,
                             "trace_mode": "fast", "render_s": round(ms3 / 1e3, 4),
                             "samples_per_s": round(samples / (ms3 * 1e-3), 1)}
    sc_r.free()
    # the soup bench's own launch shape is restored for anything measured after this block
    ctx.set_trace_config(closest_shape["block_threads"], 0, closest_shape["batch"])
    ctx.set_trace_stack(closest_shape["stack"], closest_shape.get("smem_stack", 0), flags=cav.TRACE_EXACT)
    return out


def config1_block(ctx):
    """Config 1: the mini room (36 triangles with the light quad), 256x256, 16 spp, depth 5,
    path integrator, 0 treelet rounds: paths/s of whole renders (device time, median of 5);
    and the LBVH build + 2 treelet rounds of its 34 non-light triangles alone (device stage
    times, median of 20 builds)."""
    import os as _os
    import tempfile

    import torch

    from cavalry_b200 import scenes

    room = scenes.mini_room()
    tmp = tempfile.mkdtemp()
    path = _os.path.join(tmp, "room.pbrt")
    scenes.write_pbrt(path, room, width=256, height=256, spp=16, max_depth=5)
    sc = ctx.load_pbrt(path, bvh_rounds=0)
    ms = []
    for k in range(6):
        _, _, m = sc.render()
        if k > 0:
            ms.append(m)
    st = sc.stats().as_dict()
    sc.free()
    paths = 256 * 256 * 16
    light = {i for i, m in enumerate(room["meshes"]) if m[0].startswith("light")}
    keep = np.array([int(m) not in light for m in room["mesh_ids"]])
    idx34 = np.ascontiguousarray(room["indices"][keep])
    d_pos = torch.from_numpy(np.ascontiguousarray(room["positions"])).cuda()
    d_idx = torch.from_numpy(idx34).cuda()
    bms = []
    for k in range(21):
        b = ctx.build(d_pos, d_idx, rounds=2)
        torch.cuda.synchronize()
        if k > 0:
            bms.append(float(np.sum(b.stage_times())))
        b.free()
    return {"render": {"workload": "mini_room_256x256_16spp_depth5_path", "ms": round(_median(ms), 3),
                       "paths_per_s": round(paths / (_median(ms) * 1e-3), 1), "closest_rays": st["closest_rays"],
                       "shadow_rays": st["shadow_rays"], "timing": "cav_render_to_host device time, median of 5"},
            "build_34_tris_2_rounds": {"triangles": int(len(idx34)), "ms": round(_median(bms), 4),
                                       "builds_per_s": round(1e3 / _median(bms), 1),
                                       "timing": "device stage times (CUDA events), median of 20"}}


# -------------------------------------------------------------------- reference
def run_reference(args):
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    from cavalry_b200 import scenes
    from oracle import pyoracle as po

    pos, idx = scenes.soup(N_TRI, seed=2)
    o = po.build(pos, idx, rounds=ROUNDS)
    rays = scenes.closest_rays(N_RAYS, seed=20)
    m = 1 << 16
    t0 = time.perf_counter()
    po.trace_closest(o["final"], pos, idx, rays[:m])
    dt = time.perf_counter() - t0
    sample = int(min(N_RAYS, max(m, m * 4.0 / max(dt, 1e-3))))  # ~4 s per step
    for _ in range(args.warmup):
        po.trace_closest(o["final"], pos, idx, rays[:min(sample, 1 << 16)])
    times = []
    for k in range(args.steps):
        off = (k * sample) % max(1, N_RAYS - sample + 1)
        t0 = time.perf_counter()
        po.trace_closest(o["final"], pos, idx, rays[off:off + sample])
        times.append(time.perf_counter() - t0)
    ms = statistics.mean(times) * 1e3
    value = sample / (ms * 1e-3) / 1e6
    cores = po.num_threads()
    print(json.dumps({
        "impl": "reference",
        "metric": METRIC, "value": round(value, 3), "unit": UNIT, "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": round(ms, 3), "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f32", "data": "synthetic (seeded triangle soup and rays)",
        "config": {"workload": WORKLOAD, "triangles": N_TRI, "rays_per_step": sample, "treelet_rounds": ROUNDS},
        "cpu_baseline": {"value": round(value, 3), "unit": UNIT, "cores": cores, "kind": "port",
                         "sample": f"{sample} of {N_RAYS} closest-hit rays per step (C port of BVH::build "
                                   f"+ BVH::intersect, OpenMP)"},
        "e2e": {"value": round(value, 3), "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }))


# ------------------------------------------------------------------------ render workload
def run_render(args):
    """The 5.24M-triangle path-traced scene: 64 icospheres (level 6) in a 20x10x20 room, 4
    materials, 3 area lights, 1920x1080, 64 spp, max depth 8, path integrator, treelet
    rounds 0 and 3.  Reports the extend stage's closest-hit Mrays/s (rays traced by the
    closest-hit stage / that stage's device time) and samples/s of whole renders, beside the
    reference's CUDA build on the same B200: its BVH::intersect on the renderer's own
    bounce-0 and bounce-1 rays (same trees), and its CLI render of the same .pbrt."""
    import tempfile

    import torch

    import cavalry_b200 as cav
    from cavalry_b200 import scenes
    from oracle import pyoracle as po
    from oracle import ref_cli

    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    if args.small:
        n_sph, level, W, H, spp = 16, 5, 480, 270, 16
    else:
        n_sph, level, W, H, spp = 64, 6, 1920, 1080, 64
    depth = 8
    workload = f"spheres_{n_sph}x{20 * 4 ** level}_tris_{W}x{H}_{spp}spp_depth{depth}_path"
    # seed 9: LBVH depth 44, inside the reference's fixed 64-entry traversal stack (seeds 3
    # and 4 give depth 64 and 69, which the reference's unchecked stack could overrun)
    scene = scenes.sphere_scene(n_sph, level, seed=9)
    tmp = tempfile.mkdtemp()
    pbrt = os.path.join(tmp, "spheres.pbrt")
    scenes.write_pbrt(pbrt, scene, width=W, height=H, spp=spp, max_depth=depth)
    ctx = cav.Context(0)
    out = {"metric": "closest-hit Mrays/s (render extend stage)", "unit": "Mrays/s", "n_gpus": 1,
           "higher_is_better": True, "dtype": "f32", "data": "synthetic (seeded icosphere scene written as .pbrt)",
           "config": {"workload": workload, "triangles": int(len(scene["indices"])), "width": W, "height": H,
                      "spp": spp, "max_depth": depth}}
    sampler = ClockSampler(0)
    runs = {}
    captured = {}
    for rounds in (0, 3):
        t0 = time.time()
        sc = ctx.load_pbrt(pbrt, bvh_rounds=rounds)
        load_s = time.time() - t0
        for _ in range(max(args.warmup, 1)):  # warm-up: full-resolution 1-spp renders
            sc.render(spp=1)
        # the project's autotuner picks the traversal launch shape on the renderer's own
        # bounce-0 and bounce-1 rays (a 1M-ray sample of each)
        bvh = sc.bvh()
        tune_rays = torch.cat([sc.capture_rays(d, capacity=1 << 20) for d in (0, 1)])
        tuned = bvh.autotune(tune_rays)
        tuned_fast = bvh.autotune(tune_rays, flags=cav.TRACE_FAST)
        fs = torch.empty(H * W * 3, device="cuda")
        fw = torch.empty(H * W, device="cuda")
        sc.render_into(fs, fw, fast_trace=True)  # builds the fast mode's layout
        if rounds == 3:
            sampler.start()
        totals, totals_fast = [], []
        for _ in range(args.render_steps):
            torch.cuda.synchronize()
            sc.render_into(fs, fw)
            totals.append(sc.stats().as_dict())
            torch.cuda.synchronize()
            sc.render_into(fs, fw, fast_trace=True)
            totals_fast.append(sc.stats().as_dict())
        if rounds == 3:
            clocks = sampler.stop()
        st = totals[-1]
        samples = W * H * spp
        runs[rounds] = {
            "load_s": round(load_s, 2),
            "ms_render": round(statistics.median(t["ms_total"] for t in totals), 2),
            "samples_per_s": round(samples / (statistics.median(t["ms_total"] for t in totals) * 1e-3), 1),
            "extend_mrays_s": round(st["closest_rays"] / (st["ms_closest"] * 1e-3) / 1e6, 2),
            "shadow_mrays_s": round(st["shadow_rays"] / max(st["ms_any"], 1e-9) * 1e-3, 2),
            "closest_rays": st["closest_rays"], "shadow_rays": st["shadow_rays"],
            "ms_closest": round(st["ms_closest"], 2), "ms_any": round(st["ms_any"], 2),
            "ms_shade": round(st["ms_shade"], 2), "bounces": st["bounces"],
        }
        runs[rounds]["launch_shape"] = {k: tuned[k] for k in ("block_threads", "batch", "stack")}
        # the renderer's own bounce-0 and bounce-1 rays, traced alone by ours (same tree),
        # with the launch shape tuned for each bounce's rays
        caps = [sc.capture_rays(d, capacity=1 << 22) for d in (0, 1)]
        ours = []
        shapes = []
        for r in caps:
            t_b = bvh.autotune(r)
            shapes.append({k: t_b[k] for k in ("block_threads", "batch", "stack")})
            for _ in range(3):
                bvh.trace_closest(r)
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(5):
                bvh.trace_closest(r)
            b.record()
            torch.cuda.synchronize()
            ours.append(len(r) * 5 / (a.elapsed_time(b) * 1e-3) / 1e6)
        # the same rays in the compressed 8-wide fast mode (same hit distances; ties may pick
        # another triangle), its launch shape tuned for each bounce's rays
        fast = []
        for r in caps:
            bvh.autotune(r, flags=cav.TRACE_FAST)
            for _ in range(3):
                bvh.trace_closest(r, flags=cav.TRACE_FAST)
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(5):
                bvh.trace_closest(r, flags=cav.TRACE_FAST)
            b.record()
            torch.cuda.synchronize()
            fast.append(len(r) * 5 / (a.elapsed_time(b) * 1e-3) / 1e6)
        runs[rounds]["ours_fast_captured_mrays_s"] = [round(x, 2) for x in fast]
        # whole renders with the fast traversal (timed beside the exact ones above)
        stf = sorted(totals_fast, key=lambda t: t["ms_total"])[len(totals_fast) // 2]
        runs[rounds]["fast_render"] = {
            "ms_render": round(stf["ms_total"], 2),
            "samples_per_s": round(samples / (stf["ms_total"] * 1e-3), 1),
            "extend_mrays_s": round(stf["closest_rays"] / (stf["ms_closest"] * 1e-3) / 1e6, 2),
            "shadow_mrays_s": round(stf["shadow_rays"] / max(stf["ms_any"], 1e-9) * 1e-3, 2),
            "ms_closest": round(stf["ms_closest"], 2), "ms_any": round(stf["ms_any"], 2),
            "launch_shape": {k: tuned_fast[k] for k in ("block_threads", "batch")}}
        runs[rounds]["captured_rays"] = [int(len(r)) for r in caps]
        runs[rounds]["captured_launch_shapes"] = shapes
        runs[rounds]["ours_captured_mrays_s"] = [round(x, 2) for x in ours]
        captured[rounds] = ([r.cpu().numpy() for r in caps], bvh.export_nodes())
        if rounds == 0:
            s_np, w_np = fs.view(H, W, 3).cpu().numpy(), fw.view(H, W).cpu().numpy()
            ours_img = cav.film_to_rgb8(s_np, w_np)
        sc.free()
    out["value"] = runs[3]["fast_render"]["extend_mrays_s"]
    out["config"]["trace_mode"] = ("fast: compressed 8-wide traversal (closest hits identical to the exact mode "
                                   "except at equal-distance ties); exact-mode figures in render.roundsN")
    out["render"] = {f"rounds{k}": v for k, v in runs.items()}
    out["clocks"] = clocks
    # reference CUDA build on the same B200
    ref = {}
    if po.ref_available() and not args.no_reference:
        try:
            R = po.RefScene(scene["positions"], scene["indices"], scene["mesh_ids"], rounds=0, dump=False)
            for rounds in (0, 3):
                rays, nodes = captured[rounds]
                if rounds == 3:
                    R.load_nodes(nodes)
                mr = []
                for r in rays:
                    R.trace_closest(r, reps=1)
                    _, _, ms = R.trace_closest(r, reps=3)
                    mr.append(round(len(r) / (ms * 1e-3) / 1e6, 2))
                ref[f"rounds{rounds}_bvh_intersect_mrays_s"] = mr
                ref[f"rounds{rounds}_speedup"] = [round(a / b, 2) for a, b in
                                                  zip(runs[rounds]["ours_captured_mrays_s"], mr)]
                ref[f"rounds{rounds}_speedup_fast"] = [round(a / b, 2) for a, b in
                                                       zip(runs[rounds]["ours_fast_captured_mrays_s"], mr)]
            R.free()
        except Exception as e:  # the harness is test infrastructure: report, do not fail the bench
            ref["harness_error"] = str(e)[:300]
    if ref_cli.available() and not args.no_reference:
        try:
            t0 = time.time()
            img, text = ref_cli.render(pbrt, os.path.join(tmp, "ref.png"), spp=spp, timeout=1500)
            ref["cli_wall_s"] = round(time.time() - t0, 2)
            for line in text.splitlines():
                if line.startswith("Rendering took"):
                    ms = float(line.split()[2].rstrip("ms"))
                    ref["cli_rendering_ms"] = ms
                    ref["cli_samples_per_s"] = round(W * H * spp / (ms * 1e-3), 1)
            d = np.abs(img.astype(int) - ours_img.astype(int)).max(2)
            ref["image_vs_ours_rounds0"] = {"exact": round(float((d == 0).mean()), 4),
                                            "le2": round(float((d <= 2).mean()), 4), "max": int(d.max())}
        except Exception as e:
            ref["cli_error"] = str(e)[:300]
    out["reference_cuda"] = ref or {"unavailable": "reference build not present (oracle/_ref)"}
    # CPU baseline: the path-tracing oracle on a bounded sample of the same render
    if not args.no_cpu_baseline:
        n = 4096 if not args.small else 2048
        t0 = time.time()
        po.render_path(scene, width=W, height=H, spp=spp, max_depth=depth, first=0, count=n)
        dt = time.time() - t0
        out["cpu_baseline"] = {"value": round(n / dt, 1), "unit": "samples/s", "cores": po.num_threads(),
                               "kind": "port", "sample": f"first {n} camera samples (pixel-major), OpenMP"}
    print(json.dumps(out))


# ------------------------------------------------------------------------ captured-ray workload
def run_capture(args):
    """The renderer's own extend rays of one bounce on the icosphere scene (64 spheres,
    level 6, or level 5 with --small; seed 9; 3 treelet rounds), traced alone by the exact
    and the fast (compressed 8-wide) modes with default launch shapes: one warm-up and three
    timed launches each (CUDA events), then the instrumented visit counts."""
    import tempfile

    import torch

    import cavalry_b200 as cav
    from cavalry_b200 import scenes

    level = 5 if args.small else 6
    W, H = (640, 360) if args.small else (1920, 1080)
    tmp = tempfile.mkdtemp()
    pbrt = os.path.join(tmp, "spheres.pbrt")
    scenes.write_pbrt(pbrt, scenes.sphere_scene(64, level, seed=9), width=W, height=H, spp=8, max_depth=8)
    ctx = cav.Context(0)
    sc = ctx.load_pbrt(pbrt, bvh_rounds=3)
    sc.render(spp=1)
    rays = sc.capture_rays(args.bounce, capacity=1 << 22)
    bvh = sc.bvh()
    out = {"metric": "closest-hit Mrays/s (captured extend rays)", "unit": "Mrays/s", "n_gpus": 1,
           "higher_is_better": True, "dtype": "f32", "data": "synthetic (seeded icosphere scene, renderer's rays)",
           "config": {"workload": f"spheres_64x{20 * 4 ** level}_tris_bounce{args.bounce}_rays",
                      "rays": int(len(rays)), "treelet_rounds": 3}}
    for name, fl in (("fast", cav.TRACE_FAST), ("exact", cav.TRACE_EXACT)):
        bvh.trace_closest(rays, flags=fl)
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(3):
            bvh.trace_closest(rays, flags=fl)
        b.record()
        torch.cuda.synchronize()
        out[name] = {"mrays_s": round(3 * len(rays) / (a.elapsed_time(b) * 1e-3) / 1e6, 1)}
    for name, fl in (("fast", cav.TRACE_FAST), ("exact", cav.TRACE_EXACT)):
        nodes, tris = bvh.trace_stats(rays, flags=fl)
        out[name]["nodes_per_ray"] = round(nodes / len(rays), 3)
        out[name]["tris_per_ray"] = round(tris / len(rays), 3)
    out["value"] = out["fast"]["mrays_s"]
    ctx.sync_check()
    print(json.dumps(out))


# ------------------------------------------------------------------------ serve workload
def run_serve(args):
    """Served stream (config 4): `--jobs` jobs (256) arriving as a Poisson process (mean gap
    20 ms, seed 4), each with its OWN seeded scene of the soup type (scenes.soup_scene: a
    config-2-type soup, triangle counts log-uniform in [1k, 2M], seed 1000 + job) written
    before the stream starts as a .pbrt file with its mesh in binary PLY.  3 of 4 jobs render
    their scene (resolution uniform in {64^2, 256^2, 512^2, 1024^2}, spp uniform in {1, 4, 16,
    64}, depth 6, path integrator); 1 of 4 are ray queries of 256k-4M rays (log-uniform; half
    closest hit, half any hit with limits) against their scene's tree.  Treelet rounds follow
    the reference's default (3, or 10 when spp >= 64) in both arms.

    Server arm: cav_server_submit_scene per job at its arrival: loader threads parse, the
    job is admitted under an 80 GB HBM budget, the trees of scenes admitted together are
    built in one batched build on the lane's stream, renders join the merged traversal
    launches (or, for small ones, are replayed as one CUDA graph), the scene is freed at the
    end.  Plain loop: per job in arrival order, what a user writes with the public calls:
    cav_scene_load_pbrt (parse, upload, build), cav_render_to_host or the host-buffer trace
    calls, cav_scene_free.  Both arms trace in the same mode (`--serve-trace`, default fast)
    and render the same samples, so every job's result is compared between them (relMSE of
    films, equality of hits).  Latency = completion - arrival."""
    import shutil
    import tempfile
    import threading

    import cavalry_b200 as cav
    from cavalry_b200 import scenes

    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    flags = cav.TRACE_FAST if args.serve_trace == "fast" else cav.TRACE_EXACT
    rng = np.random.default_rng(4)
    resolutions = [64, 256, 512, 1024]
    jobs = []
    t = 0.0
    for i in range(args.jobs):
        t += rng.exponential(0.020)
        n = int(np.exp(rng.uniform(np.log(1e3), np.log(2e6))))
        if rng.random() < 0.25:
            nr = int(np.exp(rng.uniform(np.log(2 ** 18), np.log(2 ** 22))))
            kind = "any" if rng.random() < 0.5 else "closest"
            jobs.append(dict(at=t, kind=kind, tris=n, rays=nr, seed=1000 + i))
        else:
            jobs.append(dict(at=t, kind="render", tris=n, res=resolutions[int(rng.integers(0, 4))],
                             spp=[1, 4, 16, 64][int(rng.integers(0, 4))], seed=1000 + i))
    tmp = tempfile.mkdtemp(prefix="cav_serve_")
    t0 = time.time()
    ray_inputs = {}
    for i, j in enumerate(jobs):
        j["path"] = os.path.join(tmp, f"job{i}.pbrt")
        res = j.get("res", 64)
        scenes.write_pbrt(j["path"], scenes.soup_scene(j["tris"], seed=j["seed"]), width=res, height=res,
                          spp=j.get("spp", 1), max_depth=6, ply=True)
        if j["kind"] == "closest":
            ray_inputs[i] = (scenes.closest_rays(j["rays"], seed=j["seed"]), None)
        elif j["kind"] == "any":
            ray_inputs[i] = scenes.shadow_rays(j["rays"], seed=j["seed"])
    setup_s = time.time() - t0
    ctx = cav.Context(0)

    def summarize(lat, makespan, service):
        lat = np.array(lat)
        return {"jobs_per_s": round(len(jobs) / makespan, 3), "makespan_s": round(makespan, 3),
                "p50_latency_ms": round(float(np.percentile(lat, 50)) * 1e3, 2),
                "p99_latency_ms": round(float(np.percentile(lat, 99)) * 1e3, 2),
                "mean_latency_ms": round(float(lat.mean()) * 1e3, 2),
                "service_s_by_class": dict(sorted((k, round(v, 3)) for k, v in service.items()))}

    def serve(lanes):
        sv = cav.Server(ctx, hbm_budget_bytes=80 << 30, mode=cav.SERVE_MERGED, trace_flags=flags,
                        loaders=args.serve_loaders, lanes=lanes)
        ids = [None] * len(jobs)
        outs = [None] * len(jobs)
        wall0 = time.perf_counter()
        clock0 = sv.stats().now_s

        def submitter():
            for i, j in enumerate(jobs):
                delay = j["at"] - (time.perf_counter() - wall0)
                if delay > 0:
                    time.sleep(delay)
                if j["kind"] == "render":
                    jid, fs, fw = sv.submit_scene_render(j["path"], j["res"], j["res"], spp=j["spp"], max_depth=6)
                    outs[i] = (fs, fw)
                else:
                    r, lim = ray_inputs[i]
                    res = sv.submit_scene_rays(j["path"], r, any_hit=j["kind"] == "any", limit=lim)
                    jid = res[0]
                    outs[i] = res[1:]
                ids[i] = jid

        th = threading.Thread(target=submitter)
        th.start()
        th.join()
        stats = [sv.wait(jid, timeout_s=3600).as_dict() for jid in ids]
        st = sv.stats().as_dict()
        sv.close()
        # arrival = submission on the server's clock (the submitter keeps the schedule)
        lat = [s["t_done"] - (clock0 + j["at"]) for s, j in zip(stats, jobs)]
        makespan = max(s["t_done"] for s in stats) - (clock0 + jobs[0]["at"])
        service = {}
        for j, s in zip(jobs, stats):
            cls = f"render_{j['res']}" if j["kind"] == "render" else f"rays_{j['kind']}"
            service[cls] = service.get(cls, 0.0) + s["t_done"] - s["t_start"]
        out = summarize(lat, makespan, service)
        out.update({"ticks": st["ticks"], "closest_launches": st["closest_launches"],
                    "any_launches": st["any_launches"], "max_segments_per_launch": st["max_segments"],
                    "server_busy_s": round(st["busy_s"], 3)})
        return out, outs

    def plain_loop():
        """The plain sequential loop: each job, in arrival order, through the public one-shot
        calls; results back in host memory."""
        fast = flags == cav.TRACE_FAST
        outs = [None] * len(jobs)
        lat, service = [], {}
        wall0 = time.perf_counter()
        for i, j in enumerate(jobs):
            delay = j["at"] - (time.perf_counter() - wall0)
            if delay > 0:
                time.sleep(delay)
            t0 = time.perf_counter()
            sc = ctx.load_pbrt(j["path"])
            if j["kind"] == "render":
                fs, fw, _ = sc.render(spp=j["spp"], max_depth=6, width=j["res"], height=j["res"], integrator="path",
                                      fast_trace=fast)
                outs[i] = (fs, fw)
                cls = f"render_{j['res']}"
            else:
                bvh = sc.bvh()
                r, lim = ray_inputs[i]
                if j["kind"] == "closest":
                    outs[i] = tuple(bvh.trace_closest_host(r, flags=flags))
                else:
                    outs[i] = (bvh.trace_any_host(r, limit=lim, flags=flags),)
                cls = f"rays_{j['kind']}"
            sc.free()
            t1 = time.perf_counter()
            service[cls] = service.get(cls, 0.0) + t1 - t0
            lat.append(t1 - wall0 - j["at"])
        makespan = time.perf_counter() - wall0 - jobs[0]["at"]
        return summarize(lat, makespan, service), outs

    # warm-up: one small job through each arm (first-use costs: module load, Halton tables)
    sc = ctx.load_pbrt(jobs[0]["path"])
    sc.render(spp=1, max_depth=2, width=16, height=16, fast_trace=flags == cav.TRACE_FAST)
    sc.free()
    plain, out_p = plain_loop()
    lane_list = [int(x) for x in str(args.serve_lanes).split(",")]
    sweep = {}
    for k, lanes in enumerate(lane_list):
        res, outs = serve(lanes)
        sweep[f"lanes{lanes}"] = res
        if k == 0:
            merged, out_m = res, outs
    # each job's result alone (plain loop) against the same job in the mix (server)
    rel, ray_same = [], []
    for i, j in enumerate(jobs):
        a, b = out_m[i], out_p[i]
        if j["kind"] == "render":
            ra = a[0] / np.maximum(a[1], 1e-30)[..., None]
            rb = b[0] / np.maximum(b[1], 1e-30)[..., None]
            rel.append(float(np.mean((ra - rb) ** 2 / (rb ** 2 + 1e-2))))
        else:
            ray_same.append(all(np.array_equal(x, y) for x, y in zip(a, b)))
    shutil.rmtree(tmp, ignore_errors=True)
    renders = sum(1 for j in jobs if j["kind"] == "render")
    out = {
        "metric": "served jobs/s (server vs plain sequential loop, jobs bring their own scenes)",
        "value": merged["jobs_per_s"], "unit": "jobs/s", "n_gpus": 1, "higher_is_better": True, "dtype": "f32",
        "data": "synthetic (seeded soups written as .pbrt + binary PLY per job; seeded Poisson job stream)",
        "config": {"workload": f"served_stream_{len(jobs)}_jobs_own_scenes_poisson_20ms", "jobs": len(jobs),
                   "render_jobs": renders, "ray_jobs": len(jobs) - renders,
                   "triangles_total": int(sum(j["tris"] for j in jobs)),
                   "triangles_range": [int(min(j["tris"] for j in jobs)), int(max(j["tris"] for j in jobs))],
                   "resolutions": resolutions, "spp": [1, 4, 16, 64], "depth": 6, "hbm_budget_gib": 80,
                   "trace_mode": args.serve_trace, "loaders": args.serve_loaders, "lanes": lane_list[0]},
        "server": merged, "plain_loop": plain,
        "server_by_lanes": {k: {"jobs_per_s": v["jobs_per_s"], "p50_latency_ms": v["p50_latency_ms"],
                                "p99_latency_ms": v["p99_latency_ms"]} for k, v in sweep.items()},
        "speedup_vs_plain_loop": round(merged["jobs_per_s"] / plain["jobs_per_s"], 3),
        "p99_latency_ratio_plain_over_server": round(plain["p99_latency_ms"] / merged["p99_latency_ms"], 3),
        "relmse_server_vs_alone": {"max": max(rel) if rel else None, "mean": float(np.mean(rel)) if rel else None,
                                   "renders": len(rel)},
        "ray_jobs_identical": int(sum(ray_same)), "setup_s": round(setup_s, 1),
    }
    print(json.dumps(out))


# ------------------------------------------------------------------------ guided workload
def run_guided(args):
    """Config 5 (scenes.aperture_scene: a room lit only through a 0.3 x 0.3 aperture, 80 %
    plastic spheres at roughness 0.05), 1280 x 720 (--small: 256 x 192), depth 10.  relMSE
    against a 16384-spp plain path render of the same film (`--ref-spp`) for plain path,
    rlpath (Q-table) and the MLP-guided integrator at 16-256 spp, with device times; relMSE
    at equal time is interpolated (log-log) at the guided render's time for each spp."""
    import tempfile

    import cavalry_b200 as cav
    from cavalry_b200 import scenes

    if int(os.environ.get("RANK", "0")) != 0:
        return
    W, H = (256, 192) if args.small else (1280, 720)
    tmp = tempfile.mkdtemp()
    path = os.path.join(tmp, "aperture.pbrt")
    scenes.write_pbrt(path, scenes.aperture_scene(), width=W, height=H, spp=4, max_depth=10)
    ctx = cav.Context(0)
    sc = ctx.load_pbrt(path, bvh_rounds=3)
    s, w, ref_ms = sc.render(spp=args.ref_spp, integrator="path", fast_trace=True)
    ref = s / w[..., None]

    def relmse(x):
        return float(np.mean((x - ref) ** 2 / (ref ** 2 + 1e-2)))

    sc.render(spp=1, integrator="path")  # warm-up
    rows = {"path": [], "rlpath": [], "guided": []}

    def best_of_two(fn):
        # each render runs twice and keeps the first film with the faster time (path is
        # deterministic; rlpath and the guided render relearn from the same start, so their
        # two films differ only by the order of float atomics)
        r0 = fn()
        r1 = fn()
        return r0[0], r0[1], min(r0[2], r1[2])

    # the baselines run to 1024 spp so that every guided time lies inside their sweep
    for spp in (16, 32, 64, 128, 256, 512, 1024):
        s, w, ms = best_of_two(lambda: sc.render(spp=spp, integrator="path"))
        rows["path"].append((spp, ms, relmse(s / w[..., None])))
        s, w, ms = best_of_two(lambda: sc.render(spp=spp, integrator="rlpath"))
        rows["rlpath"].append((spp, ms, relmse(s / w[..., None])))
        if spp <= 256:
            s, w, ms = best_of_two(lambda: sc.render_guided(spp=spp, steps_per_pass=64, lr=5e-3)[:3])
            rows["guided"].append((spp, ms, relmse(s / w[..., None])))

    def at_time(rs, t):
        ts = np.log([r[1] for r in rs])
        es = np.log([r[2] for r in rs])
        return float(np.exp(np.interp(np.log(t), ts, es)))

    equal_time = [{"spp_guided": g[0], "ms": round(g[1], 2), "guided": round(g[2], 6),
                   "path": round(at_time(rows["path"], g[1]), 6), "rlpath": round(at_time(rows["rlpath"], g[1]), 6)}
                  for g in rows["guided"]]
    out = {"metric": f"relMSE at equal spp and equal time vs a {args.ref_spp}-spp path render", "unit": "relMSE",
           "higher_is_better": False, "n_gpus": 1, "dtype": "f32 (network bf16, fp32 accumulate)",
           "data": "synthetic (seeded aperture scene written as .pbrt)",
           "config": {"workload": f"aperture_{W}x{H}_depth10", "triangles": int(sc.info().triangles),
                      "reference_spp": args.ref_spp, "reference_ms": round(ref_ms, 1),
                      "reference_trace": "fast (same hit distances; an equal-distance tie may pick another "
                                         "triangle)"},
           "equal_spp": {k: [{"spp": r[0], "ms": round(r[1], 2), "relmse": round(r[2], 6)} for r in v]
                         for k, v in rows.items()},
           "equal_time": equal_time}
    print(json.dumps(out))


# ------------------------------------------------------------------------ batched builds
def run_batch(args):
    """Many scenes built at once: `cav_bvh_build_batch` (one launch per LBVH stage over all
    scenes, treelet rounds per group of scenes, one shared arena) against one `cav_bvh_build`
    per scene, for three mixes of seeded soups with log-uniform triangle counts, at 0 and 3
    treelet rounds.  Wall time of the whole build (host call to device completion), min of
    3 repetitions after a warm-up, inputs resident on the device."""
    import torch

    import cavalry_b200 as cav
    from cavalry_b200 import scenes

    if int(os.environ.get("RANK", "0")) != 0:
        return
    ctx = cav.Context(0)
    mixes = [(256, 1_000, 30_000), (64, 1_000, 100_000), (16, 10_000, 2_000_000)]
    rows = []
    for k, lo, hi in mixes:
        rng = np.random.default_rng(k)
        sizes = np.exp(rng.uniform(np.log(lo), np.log(hi), k)).astype(int)
        data = []
        for i, nt in enumerate(sizes):
            pos, idx = scenes.soup(int(nt), seed=100 + i)
            data.append((torch.from_numpy(pos).cuda(), torch.from_numpy(idx).cuda()))
        for rounds in (0, 3):
            def batched():
                return ctx.build_batch(data, rounds=rounds)

            def single():
                return [ctx.build(p, i, rounds=rounds) for p, i in data]

            best = {}
            for name, fn in (("batched", batched), ("one_by_one", single)):
                t = []
                for rep in range(4):
                    torch.cuda.synchronize()
                    t0 = time.perf_counter()
                    trees = fn()
                    torch.cuda.synchronize()
                    t.append(time.perf_counter() - t0)
                    ctx.sync_check()
                    for tr in trees:
                        tr.free()
                best[name] = min(t[1:]) * 1e3  # the first repetition warms the allocator
            rows.append({"scenes": k, "triangles": int(sizes.sum()), "range": [lo, hi], "rounds": rounds,
                         "batched_ms": round(best["batched"], 2), "one_by_one_ms": round(best["one_by_one"], 2),
                         "ratio": round(best["one_by_one"] / best["batched"], 2)})
    print(json.dumps({"metric": "batched BVH build speed-up over one build per scene", "unit": "x",
                      "higher_is_better": True, "n_gpus": 1, "data": "synthetic (seeded soups)",
                      "config": {"workload": "batched_builds_3_mixes", "timing": "wall, min of 3 after one warm-up"},
                      "rows": rows}))


# ------------------------------------------------------------------------ mlp workload
def run_mlp(args):
    """The learned proposal's kernels alone: forward passes over 4M vertices (--small: 1M)
    and Adam steps at batch 16,384, device-timed, for the tcgen05 kernel (the value) and
    the mma.sync kernel beside it; FLOP/s counts the 41 kFLOP of one forward pass per
    vertex (160x64 + 2 x 64x64 + 64x32 multiply-adds x 2).  The forward reads 20 bytes and
    writes 128 bytes per vertex, so its HBM floor is also reported."""
    import torch

    import cavalry_b200 as cav

    if int(os.environ.get("RANK", "0")) != 0:
        return
    ctx = cav.Context(0)
    n = 1 << 20 if args.small else 1 << 22
    g = torch.Generator("cuda").manual_seed(1)
    x = torch.rand((n, 5), device="cuda", generator=g)
    d = torch.nn.functional.normalize(torch.randn((n, 3), device="cuda", generator=g), dim=1).contiguous()
    w = torch.rand(n, device="cuda", generator=g)
    flop = 2 * (160 * 64 + 2 * 64 * 64 + 64 * 32)
    steps = max(args.steps, 1)
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    peaks = json.loads((ROOT / "MEASURED_PEAKS.json").read_text()) if (ROOT / "MEASURED_PEAKS.json").exists() else {}
    peak = float(peaks.get("bf16_tflops", 1590.0))
    hbm = float(peaks.get("hbm_gbs", 6650.0))

    def measure(kernel):
        net = cav.Mlp(ctx, seed=1, kernel=kernel)
        for _ in range(max(args.warmup, 3)):
            net.forward(x)
        torch.cuda.synchronize()
        a.record()
        for _ in range(steps):
            net.forward(x)
        b.record()
        torch.cuda.synchronize()
        fwd_ms = a.elapsed_time(b) / steps
        bs = 16384
        for _ in range(3):
            net.train_step(x[:bs], d[:bs], w[:bs], lr=1e-3)
        torch.cuda.synchronize()
        a.record()
        for k in range(steps):
            o = (k * bs) % (n - bs)
            net.train_step(x[o:o + bs], d[o:o + bs], w[o:o + bs], lr=1e-3)
        b.record()
        torch.cuda.synchronize()
        train_ms = a.elapsed_time(b) / steps
        ctx.sync_check()
        net.free()
        ach = flop * n / (fwd_ms * 1e-3) / 1e12
        return {"forward_ms": round(fwd_ms, 4), "train_step_ms": round(train_ms, 4),
                "g_samples_s": round(n / (fwd_ms * 1e-3) / 1e9, 3), "tflops": round(ach, 1),
                "frac": round(ach / peak, 4)}

    tc = measure(cav.MLP_KERNEL_TCGEN05)
    ms = measure(cav.MLP_KERNEL_MMA_SYNC)
    floor_ms = n * (20 + 128) / (hbm * 1e9) * 1e3
    print(json.dumps({"metric": "MLP forward samples/s", "value": tc["g_samples_s"],
                      "unit": "G samples/s", "n_gpus": 1, "steps": steps, "higher_is_better": True,
                      "dtype": "bf16 (fp32 accumulate)", "data": "synthetic",
                      "config": {"workload": f"mlp_forward_{n}_vertices", "batch": n, "train_batch": 16384},
                      "forward_ms": tc["forward_ms"], "train_step_ms": tc["train_step_ms"],
                      "roofline": {"bound": "tensor", "achieved": tc["tflops"], "peak": peak, "unit": "TFLOP/s",
                                   "frac": tc["frac"], "peak_kind": "measured" if peaks else "fallback",
                                   "instruction": "tcgen05.mma.cta_group::1.kind::f16 M128 bf16, TMEM accumulators",
                                   "hbm_floor_ms": round(floor_ms, 4)},
                      "mma_sync": ms}))


def main():
    args = parse()
    if args.workload == "mlp":
        run_mlp(args)
    elif args.workload == "batch":
        run_batch(args)
    elif args.workload == "guided":
        run_guided(args)
    elif args.workload == "serve":
        run_serve(args)
    elif args.workload == "capture":
        run_capture(args)
    elif args.workload == "render":
        run_render(args)
    elif args.impl == "reference":
        run_reference(args)
    else:
        run_ours(args)


if __name__ == "__main__":
    main()
