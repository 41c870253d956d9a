"""Benchmark: exact min-cut segmentation throughput on GB300.

Prints ONE JSON line (rank 0) of at most 2,800 characters (headline()); the
full record of every leg, some 20,000, goes to standard error as one line that
begins with "detail: ".  A step = the full hot path over one batch of
synthetic images: colour-histogram t-links, contrast-sensitive n-links,
graph build, exact max-flow, both canonical cuts.

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
                  [--workload batch256|batch64|plain1080|plain256|plain4096|n8_640x480]
                  [--no-single] [--no-serve] [--no-plain]

Default workload (batch256): 256 images of uneven sizes (side log-uniform
64..1024, aspect uniform 0.5..2, the 256x256 ellipse generator scaled to each
image, per-image seeds 1000+i, lambda 50) solved as ONE batch: one data-term
pass, one build, one persistent solver launch, one extraction.  The same
images solved one at a time by the plain per-image path are timed beside it
("plain_per_image"), and the single-image workloads (256x256, three
1920x1080 images at lambda 10/50/200, 4096x4096 with 2000 blobs, and the
8-neighbourhood 640x480 graph) are measured the same way under
"single_image" (skipped with --no-single).

value : Mpixel/s with the images already resident in HBM (CUDA events per
        step; a 256 MB buffer is written before every step to flush L2).
e2e   : the same metric through the host entry points: images and scribbles
        copied in from pinned host memory and both label maps copied back
        inside the timed region, every step.  Batched workloads stream the
        steps through gcfg_batch_submit_host / gcfg_batch_wait with two
        batches in flight (wall clock over all steps, the first upload and
        the last download included; no L2 flush, the inputs uploaded anew
        every step being larger than L2); per-image workloads call
        gcfg_seg_run_host.  "e2e_sync" is one blocking gcfg_batch_run_host
        call per step.
roofline: the kernel with the largest device time in a profiled step;
        achieved = its algorithmic bytes (work counters x bytes per pixel)
        / its CUDA-event time; peak = MEASURED_PEAKS.json hbm_gbs.
        roofline.solve_phases: the solver's first global relabel and the push
        rounds after it run as two separate launches (gcfg_batch_phase_split,
        inside an NVTX range "phase_split" for ncu), each with its device
        time, its algorithmic bytes, the bytes it really moves and the DRAM
        traffic of its ncu capture (profiles/solve_gr_*.md, solve_push_*.md).
cpu_baseline: the oracle's Boykov-Kolmogorov solver (oracle/, the CPU
        checker) on a bounded sample of the same images, one host thread.
reference_cuda: the reference's own CUDA path on the same GPU (its kernels
        compiled from its sources into a cubin, launched in GC_Optimize's
        order by oracle/refgpu/ref_gpu.cpp), one image at a time, on a bounded
        sample of the workload; its labels are compared with libgcfg's
        S_max.
--impl reference: the reference has no CPU implementation of this path, so
        this arm times the CPU port (oracle BK) on all host threads, one image
        per thread.
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path[:0] = [ROOT, os.path.join(ROOT, "gc-fg_gb300"), os.path.join(ROOT, "oracle")]

import numpy as np  # noqa: E402

METRIC = "exact-min-cut Mpixel/s"
# Stated service level of the serving workload (500 req/s Poisson, 256^2 / 1024^2 / 2048^2 mix): every
# request answered, exact, within this latency at the 99th percentile.
P99_TARGET_MS = 5.0
UNIT = "Mpixel/s"

# Algorithmic bytes per pixel per unit of work (int32 layout):
#   global relabel: read the residual and sign bits (6 bits), write the height
#     (4 B), once per pixel per global relabel; a tile that the BFS visits again
#     in the same relabel is overhead, not algorithmic bytes
#   push tile visit (a tile active in a push round; push and local relabel
#     fused): read 4 caps + excess + height (24 B), write the same (24 B; an
#     upper bound: rows that did not change are not written)
#   source reachability (cut): read the bits, write one, once per pixel at most
#   sink reachability (the termination check after push rounds, which also
#     gives S_max): the same, once per pixel per check
#   count pass: two words per tile
#   build: read RGB (3 B), write 4 caps + excess (20 B)
#   extract: read height (4 B) + reach bit, write two label bytes (2 B)
B_GR, B_PUSH, B_REACH, B_COUNT, B_BUILD, B_EXTRACT = 4.75, 48, 0.875, 12 / 1024, 23, 6

# Bytes a solver phase really moves per tile visit in the tile-arena layout
# (what DRAM counters see when nothing is served from L2):
#   global-relabel visit: read the tile's six residual mask planes (768 B),
#     the neighbours' facing border-height lines (4 x 128 B) and their
#     residual words (2 x 4 B + 2 x 128 B); write the heights (4096 B), the
#     border lines (512 B), the reached rows (128 B) and the active count (4 B)
#   per tile of the relabel launch besides its visits: fresh queue marks and
#     reach rows (8 + 128 B), the pull check (own and neighbours' border
#     lines and residual words, 512 + 512 + 264 B), the count pass (12 B)
#   push visit: read caps, excess and heights (24 KB) and the four halo
#     lines (512 B); write caps, excess and heights (24 KB), the mask planes
#     (768 B), the border lines (512 B) and the excess sum (8 B)
MOVED_GR_VISIT = 768 + 512 + 264 + 4096 + 512 + 128 + 4
MOVED_GR_TILE = 8 + 128 + 512 + 512 + 264 + 12
MOVED_PUSH_VISIT = 24576 + 512 + 24576 + 768 + 512 + 8


def headline(line):
    """The printed line: every key of the benchmark's own contract whole, and of
    the long legs their figures alone.  A line of many thousand characters gets
    cut on its way through logs, and a cut line holds no number at all."""
    def pick(d, *keys):
        return {k: (round(d[k], 4) if isinstance(d[k], float) else d[k]) for k in keys if d.get(k) is not None}

    out = {k: v for k, v in line.items() if not isinstance(v, dict)}
    out["config"] = {k: v for k, v in line["config"].items() if k not in ("tuning", "cuda_graph")}
    if line["config"].get("tuning"):
        out["config"]["tuning"] = pick(line["config"]["tuning"], "push_rounds_per_gr", "max_tile_sweeps",
                                       "sweeps_per_local_relabel", "blocks_per_sm", "threads_y")
    for k in ("clocks", "cpu_baseline", "parity"):
        if k in line:
            out[k] = line[k]
    for k in ("e2e", "e2e_sync", "plain_per_image"):
        if k in line:
            out[k] = pick(line[k], "value", "unit", "ms_per_step", "h2d_bytes_per_step", "d2h_bytes_per_step",
                          "flows_equal_batched", "cuts_equal_batched")
    if "roofline" in line:
        out["roofline"] = pick(line["roofline"], "bound", "kernel", "achieved", "peak", "unit", "frac", "peak_source",
                               "traffic", "alg_bytes_per_launch", "avg_launch_us", "share_of_step")
    if "reference_cuda" in line:
        out["reference_cuda"] = pick(line["reference_cuda"], "value", "unit", "images", "labels_equal_smax", "unavailable")
    if "serving" in line:
        out["serving"] = pick(line["serving"]["served"], "p50_ms", "p99_ms", "mpixel_s_over_busy")
        out["serving"].update(pick(line["serving"], "p99_target_ms", "p99_met", "results_equal"))
    if "single_image" in line:
        out["single_image"] = {k: dict(pick(v, "value", "ms_per_step"), e2e=round(v["e2e"]["value"], 4))
                               for k, v in line["single_image"].items() if "value" in v}
    return out


def emit(line):
    print("detail: " + json.dumps(line), file=sys.stderr, flush=True)
    print(json.dumps(headline(line)), flush=True)


def workload(name, rank=0):
    """Images of a workload.  Batches shard by image: under N ranks every
    rank solves its own 256 images (seeds 1000 + 256 * rank + i), so the
    per-GPU work is fixed and no image is shared (weak scaling)."""
    import shard
    import synth
    if name == "batch256":
        seed0 = shard.weak_seed0(1000, 256, rank)
        shapes = synth.batch_shapes(256, seed0)
        return dict(kind="batch", desc="256 uneven images (side log-U(64,1024), aspect U(0.5,2)), "
                                      f"scaled 256x256 ellipse generator, seeds {seed0}+i, lambda 50",
                    images=[(3, W, H, seed, 50.0) for (W, H, seed) in shapes])
    if name == "batch64":
        shapes = synth.batch_shapes(256, shard.weak_seed0(1000, 256, rank))[:64]
        return dict(kind="batch", desc="the first 64 images of batch256 (small profiling case)",
                    images=[(3, W, H, seed, 50.0) for (W, H, seed) in shapes])
    if name == "plain1080":
        return dict(kind="plain", desc="plain per-image, 1920x1080, lambda {10,50,200}, seeds 1-3",
                    images=[(1, 1920, 1080, 1, 10.0), (1, 1920, 1080, 2, 50.0), (1, 1920, 1080, 3, 200.0)])
    if name == "plain256":
        return dict(kind="plain", desc="plain per-image, 256x256, lambda 50, seed 0",
                    images=[(0, 256, 256, 0, 50.0)])
    if name == "plain4096":
        return dict(kind="plain", desc="plain per-image, 4096x4096, 2000 blobs, lambda 100, seed 2",
                    images=[(2, 4096, 4096, 2, 100.0)])
    raise SystemExit(f"unknown workload {name}")


def make_inputs(spec):
    import synth
    rgb, scrib, offs = synth.generate_packed([(c, W, H, s) for (c, W, H, s, _) in spec["images"]])
    Ws = np.array([W for (_, W, _, _, _) in spec["images"]], np.int32)
    Hs = np.array([H for (_, _, H, _, _) in spec["images"]], np.int32)
    lams = np.array([lam for (*_, lam) in spec["images"]], np.float64)
    return rgb, scrib, offs, Ws, Hs, lams


def image_views(rgb, scrib, offs, Ws, Hs):
    out = []
    for i in range(len(Ws)):
        n = int(Ws[i]) * int(Hs[i])
        o = int(offs[i])
        out.append((rgb[3 * o:3 * (o + n)].reshape(Hs[i], Ws[i], 3), scrib[o:o + n].reshape(Hs[i], Ws[i])))
    return out


def dist_info():
    return (int(os.environ.get("RANK", 0)), int(os.environ.get("WORLD_SIZE", 1)),
            int(os.environ.get("LOCAL_RANK", 0)))


class ClockSampler:
    """nvidia-smi clock/throttle samples during the timed region."""

    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu: int):
        self.gpu = gpu
        self.proc = None

    def start(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.gpu), f"--query-gpu={self.Q}", "--format=csv,noheader,nounits",
                 "-lms", "100"], stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
        except OSError:
            self.proc = None

    def stop(self):
        if not self.proc:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            out, _ = self.proc.communicate(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
            out, _ = self.proc.communicate()
        sm, smax, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in out.strip().splitlines():
            f = [x.strip() for x in line.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                smax.append(float(f[2]))
            except ValueError:
                continue
            for name, v in zip(names, f[5:9]):
                if v.lower() == "active":
                    reasons.add(name)
        return {"sm_mhz": statistics.median(sm) if sm else None,
                "sm_max_mhz": max(smax) if smax else None, "reasons": sorted(reasons),
                "samples": len(sm)}


def load_peaks():
    try:
        d = json.load(open(os.path.join(ROOT, "MEASURED_PEAKS.json")))
        return float(d["hbm_gbs"]), "measured"
    except Exception:
        return 6800.0, "fallback"


def ncu_traffic(kind: str, workload_name: str):
    """DRAM bytes per launch from a committed ncu summary, if one exists."""
    p = os.path.join(ROOT, "profiles", f"{kind}_{workload_name}.md")
    if not os.path.exists(p):
        return None
    for line in open(p):
        if line.startswith("traffic_bytes_per_launch:"):
            try:
                return float(line.split(":", 1)[1])
            except ValueError:
                return None
    return None


def cpu_baseline(views, lams, budget_s=10.0, flows_gpu=None, smin_gpu=None, smax_gpu=None, offs=None):
    """Oracle BK on a bounded sample of the workload, one host thread.  When
    the GPU's flows and packed cuts are given, every sampled image's flow,
    S_min and S_max are compared with the oracle's (the comparison is outside
    the timed span).  Returns (Mpixel/s, images solved, seconds, parity)."""
    import oracle as O
    t0 = time.perf_counter()
    px, k, secs = 0, 0, 0.0
    checked, eq_flow, eq_min, eq_max = set(), 0, 0, 0
    order = sorted(range(len(views)), key=lambda i: views[i][1].size)
    while k < len(order) or len(views) <= 8:
        i = order[k] if len(views) > 8 else k % len(views)
        rgb, scrib = views[i]
        t = time.perf_counter()
        r = O.segment(rgb, scrib, float(lams[i]), solver="bk")
        secs += time.perf_counter() - t
        px += scrib.size
        k += 1
        if flows_gpu is not None and i not in checked:
            checked.add(i)
            eq_flow += int(flows_gpu[i]) == r["flow"]
            if smin_gpu is not None:
                o, n = int(offs[i]), scrib.size
                eq_min += bool(np.array_equal(smin_gpu[o:o + n], r["smin"].reshape(-1)))
                eq_max += bool(np.array_equal(smax_gpu[o:o + n], r["smax"].reshape(-1)))
        if time.perf_counter() - t0 > budget_s or (len(views) <= 8 and k >= 64):
            break
    parity = None
    if flows_gpu is not None:
        n = len(checked)
        parity = {"images_checked": n, "flows_equal_oracle": eq_flow == n}
        if smin_gpu is not None:
            parity.update(smin_equal_oracle=eq_min == n, smax_equal_oracle=eq_max == n)
    return px / secs / 1e6, k, secs, parity


def reference_cuda_leg(views, lams, smax_all, offs, budget_s=15.0):
    """The reference's own CUDA path (its kernels compiled from its sources,
    oracle/ref_cuda.py) on the same GPU: GC_Init -> GC_SetGraph ->
    GC_Optimize -> GC_End per image, one image at a time as the reference's
    applications run it, on a bounded sample of the workload's images (in
    workload order until budget_s of reference solve time).  The t-links and
    n-links are computed on the host by the oracle (outside every timed span).
    value = pixels / the sum of the GC_SetGraph + GC_Optimize wall times; the
    reference's labels are compared with libgcfg's S_max."""
    import oracle as O
    import ref_cuda
    why = ref_cuda.unavailable()
    if why:
        return {"unavailable": why}
    px, ms_solve, ms_loop, ms_all, its, n_eq, n_conv, k = 0, 0.0, 0.0, 0.0, [], 0, 0, 0
    for i, (rgb, scrib) in enumerate(views):
        dp, dn = O.tlinks(rgb, scrib)
        up, down, left, right = O.nlinks(rgb, float(lams[i]))
        r = ref_cuda.solve(dp, dn, up=up, down=down, left=left, right=right, max_seconds=30.0)
        k += 1
        if r["rc"] != 0:
            return {"unavailable": f"image {i}: {r['status']}", "images": k}
        H, W = scrib.shape
        o = int(offs[i])
        n_eq += bool(np.array_equal(r["label"].astype(np.uint8).reshape(-1), smax_all[o:o + W * H]))
        n_conv += r["converged"]
        px += W * H
        ms_solve += r["ms_solve"]
        ms_loop += r["ms_loop"]
        ms_all += r["ms_init"] + r["ms_solve"] + r["ms_end"]
        its.append(r["iterations"])
        if ms_solve > budget_s * 1e3:
            break
    return {"value": px / (ms_solve / 1e3) / 1e6, "unit": UNIT, "images": k, "pixels": px,
            "ms_per_image": ms_solve / k, "loop_only_mpixel_s": px / (ms_loop / 1e3) / 1e6,
            "with_init_end_mpixel_s": px / (ms_all / 1e3) / 1e6,
            "iterations_median": float(np.median(its)), "converged": n_conv, "labels_equal_smax": n_eq,
            "how": "the reference's kernels (GraphCutKernels.cu, compiled from its sources for sm_103a) "
                   "launched in GC_Optimize's order with its blocking flag copies; one image at a time, "
                   "wall clock of GC_SetGraph + GC_Optimize (labels to the host included)"}


def _sleep_until(now, ta):
    while True:
        d = ta - now()
        if d <= 0:
            return
        if d > 1e-3:
            time.sleep(d - 5e-4)


def _busy_time(results):
    """Length of the union of the lanes' batch intervals (seconds)."""
    iv = sorted({(r["t_start"], r["t_done"]) for r in results})
    busy, end = 0.0, None
    for a, b in iv:
        if end is None or a > end:
            busy += b - a
            end = b
        elif b > end:
            busy += b - end
            end = b
    return busy


def _lane_overlap(results):
    """Fraction of the lanes' busy time during which two or more lanes ran."""
    ev = sorted({(r["lane"], r["t_start"], r["t_done"]) for r in results}, key=lambda b: b[1])
    pts = sorted([(b[1], 1) for b in ev] + [(b[2], -1) for b in ev])
    busy = multi = 0.0
    depth, last = 0, None
    for t, d in pts:
        if last is not None and depth > 0:
            busy += t - last
            if depth > 1:
                multi += t - last
        depth += d
        last = t
    return multi / busy if busy > 0 else 0.0


def serve_bench(torch, gcfg, n_req=1200, rate=500.0, lanes=2, cap=60 << 30, seed=4):
    """Serving workload: a Poisson request trace replayed through the server
    (continuous batching, resident images, warm edits) and through a plain
    cold-solve loop (one gcfg_seg_run_host per request, edits re-solved cold
    from the edited scribbles).  Both take host buffers (pinned) and return
    both label maps to the host.  Every request's flow and cuts must be equal
    across the served run, a saturated served run (all requests at once) and
    the plain loop."""
    import zlib
    import synth
    pool_specs, reqs = synth.serve_trace(n_req, rate, seed)
    rgb, scrib, offs = synth.generate_packed(pool_specs)
    p_rgb = torch.from_numpy(rgb).pin_memory().numpy()
    p_scrib = torch.from_numpy(scrib).pin_memory().numpy()
    sides = [W for (_, W, _, _) in pool_specs]

    def pool_view(i):
        o, s = int(offs[i]), sides[i]
        return p_rgb[3 * o:3 * (o + s * s)].reshape(s, s, 3), p_scrib[o:o + s * s].reshape(s, s)

    new_img = [q["img"] for q in reqs if q["kind"] == "new"]
    img_of = [q["img"] if q["kind"] == "new" else new_img[q["target"]] for q in reqs]
    npx = np.array([sides[i] ** 2 for i in img_of], np.int64)
    ooff = np.zeros(len(reqs), np.int64)
    ooff[1:] = np.cumsum(npx)[:-1]
    total_px = int(npx.sum())
    out_min = torch.empty(total_px, dtype=torch.uint8).pin_memory().numpy()
    out_max = torch.empty(total_px, dtype=torch.uint8).pin_memory().numpy()
    now = gcfg.Server.now

    def outs(k):
        o, n, s = int(ooff[k]), int(npx[k]), sides[img_of[k]]
        return out_min[o:o + n].reshape(s, s), out_max[o:o + n].reshape(s, s)

    def digest(k, flow):
        a, b = outs(k)
        return (int(flow), zlib.crc32(a), zlib.crc32(b))

    def served(open_loop, n=None):
        rq = reqs if n is None else reqs[:n]
        srv = gcfg.Server(mem_cap_bytes=cap, lanes=lanes, max_batch_images=256, max_batch_tiles=1 << 16,
                          max_sessions=len(new_img) + 16)
        sids, tick = [], []
        t0 = now() + 0.02
        for k, q in enumerate(rq):
            ta = t0 + (q["t"] if open_loop else 0.0)
            if open_loop:
                _sleep_until(now, ta)
            smin, smax = outs(k)
            if q["kind"] == "new":
                r, s = pool_view(q["img"])
                t, sid = srv.submit_new(r, s, q["lam"], smin, smax)
                sids.append(sid)
            else:
                t, _ = srv.submit_edit(sids[q["target"]], q["x"], q["y"], q["size"], q["cls"], smin, smax)
            tick.append((t, ta))
        res = [srv.wait(t, timeout_ms=600000) for t, _ in tick]
        st = srv.stats()
        srv.close()
        assert all(r["status"] == 0 for r in res), "served request failed"
        return res, np.array([ta for _, ta in tick]), st, [digest(k, r["flow"]) for k, r in enumerate(res)]

    served(True, n=60)  # warm-up
    res, tarr, st, dig_served = served(True)
    done = np.array([r["t_done"] for r in res])
    lat = done - tarr
    svc = np.array([r["t_done"] - r["t_start"] for r in res])
    is_edit = np.array([q["kind"] == "edit" for q in reqs])
    side_of = np.array([sides[i] for i in img_of])
    qwait = np.array([r["t_start"] for r in res]) - tarr
    slow = sorted(np.nonzero(is_edit)[0], key=lambda k: -lat[k])[:6]
    edit_tail = {"p50_queue_ms": round(float(np.percentile(qwait[is_edit], 50)) * 1e3, 3),
                 "p99_queue_ms": round(float(np.percentile(qwait[is_edit], 99)) * 1e3, 3),
                 "p50_service_ms": round(float(np.percentile(svc[is_edit], 50)) * 1e3, 3),
                 "p99_service_ms": round(float(np.percentile(svc[is_edit], 99)) * 1e3, 3),
                 "p99_by_side_ms": {int(sd): round(float(np.percentile(lat[is_edit & (side_of == sd)], 99)) * 1e3, 3)
                                    for sd in sorted(set(side_of[is_edit].tolist()))},
                 "slowest": [{"side": int(side_of[k]), "latency_ms": round(float(lat[k]) * 1e3, 3),
                              "queue_ms": round(float(qwait[k]) * 1e3, 3),
                              "service_ms": round(float(svc[k]) * 1e3, 3),
                              "batch_images": int(res[k]["batch_images"]), "lane": int(res[k]["lane"])}
                             for k in slow]}
    res_sat, tarr_sat, st_sat, dig_sat = served(False)
    make_sat = max(r["t_done"] for r in res_sat) - tarr_sat[0]

    # plain cold-solve loop on the same schedule
    seg = gcfg.Segmenter(max(sides), max(sides))
    edited = {q["target"] for q in reqs if q["kind"] == "edit"}
    sess_scrib = {}
    n_new = 0
    for q in reqs:
        if q["kind"] == "new":
            if n_new in edited:
                sess_scrib[n_new] = torch.from_numpy(pool_view(q["img"])[1].copy()).pin_memory().numpy()
            n_new += 1
    p_lat, p_svc, p_done, dig_plain = [], [], [], []
    for warm in (True, False):
        n_new = 0
        t0 = now() + 0.02
        for k, q in enumerate(reqs[:60] if warm else reqs):
            ta = t0 + q["t"]
            _sleep_until(now, ta)
            ts = now()
            if q["kind"] == "new":
                r, s = pool_view(q["img"])
                if not warm and n_new in sess_scrib:
                    s = sess_scrib[n_new]
                n_new += 1
            else:
                r = pool_view(new_img[q["target"]])[0]
                s = sess_scrib[q["target"]] if not warm else pool_view(new_img[q["target"]])[1].copy()
                s[q["y"]:q["y"] + q["size"], q["x"]:q["x"] + q["size"]] = q["cls"]
            smin, smax = outs(k)
            out = seg.run_host(r, s, s.shape[1], s.shape[0], 50.0, smin, smax)
            td = now()
            if not warm:
                p_lat.append(td - ta)
                p_svc.append(td - ts)
                p_done.append(td - t0)
                dig_plain.append(out["flow"])
    seg.close()
    dig_plain = [digest(k, f) for k, f in enumerate(dig_plain)]
    p_lat = np.array(p_lat)
    p_svc = np.array(p_svc)
    p_span = max(p_done) - reqs[0]["t"]

    def ms(a, p):
        return round(float(np.percentile(a, p)) * 1e3, 3)

    return {
        "workload": f"Poisson {rate:g} req/s, {len(reqs)} requests ({int((~is_edit).sum())} new images "
                    f"256^2/1024^2/2048^2 at 60/30/10%, {int(is_edit.sum())} scribble edits 15x15 of earlier "
                    f"images), 1920x1080-family generator, lambda 50, trace seed {seed}; host buffers (pinned) "
                    f"in and both label maps out",
        "pixels": total_px, "lanes": lanes, "mem_cap_gb": cap / 2 ** 30,
        "served": {"p50_ms": ms(lat, 50), "p99_ms": ms(lat, 99),
                   "p50_new_ms": ms(lat[~is_edit], 50), "p99_new_ms": ms(lat[~is_edit], 99),
                   "p50_edit_ms": ms(lat[is_edit], 50), "p99_edit_ms": ms(lat[is_edit], 99),
                   "mpixel_s_over_span": total_px / (done.max() - tarr[0]) / 1e6,
                   "mpixel_s_over_busy": total_px / _busy_time(res) / 1e6,
                   "mean_service_ms": float(np.mean(svc)) * 1e3,
                   "batches": st["batches"], "mean_batch_images": len(reqs) / max(st["batches"], 1),
                   "lane_overlap_frac": round(_lane_overlap(res), 4),
                   "resident_gb_at_end": st["bytes_in_use"] / 2 ** 30, "evicted": st["evicted"],
                   "edit_tail": edit_tail},
        "served_saturated": {"mpixel_s": total_px / make_sat / 1e6, "makespan_ms": make_sat * 1e3,
                             "batches": st_sat["batches"]},
        "plain_cold_loop": {"p50_ms": ms(p_lat, 50), "p99_ms": ms(p_lat, 99),
                            "p50_new_ms": ms(p_lat[~is_edit], 50), "p99_new_ms": ms(p_lat[~is_edit], 99),
                            "p50_edit_ms": ms(p_lat[is_edit], 50), "p99_edit_ms": ms(p_lat[is_edit], 99),
                            "mpixel_s_over_span": total_px / p_span / 1e6,
                            "mpixel_s_over_busy": total_px / float(np.sum(p_svc)) / 1e6,
                            "mean_service_ms": float(np.mean(p_svc)) * 1e3,
                            "p99_edit_service_ms": round(float(np.percentile(p_svc[is_edit], 99)) * 1e3, 3),
                            "p99_edit_by_side_ms": {int(sd): round(float(np.percentile(
                                p_lat[is_edit & (side_of == sd)], 99)) * 1e3, 3)
                                for sd in sorted(set(side_of[is_edit].tolist()))}},
        "throughput_note": "mpixel_s_over_span = all pixels / (last completion - first arrival): at 500 req/s the "
                           "arrival rate bounds it for both; mpixel_s_over_busy = all pixels / the time the GPU "
                           "side was busy (union of the lanes' batch intervals; the plain loop's summed service "
                           "times); served_saturated submits the whole trace at once",
        "p99_target_ms": P99_TARGET_MS, "p99_met": bool(ms(lat, 99) <= P99_TARGET_MS),
        "results_equal": bool(dig_served == dig_plain and dig_sat == dig_plain),
    }


def nvtx_range(name):
    """NVTX push/pop around a block (ncu --nvtx-include filters on it); a
    no-op where NVTX is unavailable."""
    import contextlib

    @contextlib.contextmanager
    def cm():
        import torch
        pushed = False
        try:
            torch.cuda.nvtx.range_push(name)
            pushed = True
        except Exception:
            pass
        try:
            yield
        finally:
            if pushed:
                torch.cuda.nvtx.range_pop()
    return cm()


def tiles_of(Ws, Hs):
    return int(sum(((int(w) + 31) // 32) * ((int(h) + 31) // 32) for w, h in zip(Ws, Hs)))


def peak_source(peak_kind):
    return ("of measured (MEASURED_PEAKS.json hbm_gbs)" if peak_kind == "measured" else "of fallback 6.8 TB/s")


def phase_record(ms, alg, moved, traffic, peak, **extra):
    """Device time of a phase with three byte counts over it: algorithmic
    (B_GR and so on above), moved (what the phase reads and writes in this
    layout) and, when an ncu capture exists, DRAM traffic."""
    r = {"ms": round(ms, 4), "alg_bytes": int(alg), "moved_bytes": int(moved)}
    if ms > 0:
        a, m = alg / (ms / 1e3) / 1e9, moved / (ms / 1e3) / 1e9
        r.update(achieved_alg_gbs=round(a, 1), frac_alg=round(a / peak, 4),
                 achieved_moved_gbs=round(m, 1), frac_moved=round(m / peak, 4))
    r["traffic"] = traffic
    if traffic and ms > 0:
        t = traffic / (ms / 1e3) / 1e9
        r.update(achieved_dram_gbs=round(t, 1), frac_dram=round(t / peak, 4))
    r.update(extra)
    return r


def ncu_phase_traffic(kind, workload_name):
    """DRAM bytes of one phase over one pass of the workload, from a committed
    ncu summary (profiles/solve_<kind>_<workload>.md, line traffic_bytes:)."""
    p = os.path.join(ROOT, "profiles", f"solve_{kind}_{workload_name}.md")
    if not os.path.exists(p):
        return None
    for line in open(p):
        if line.startswith("traffic_bytes:"):
            try:
                return float(line.split(":", 1)[1])
            except ValueError:
                return None
    return None


def solve_phases(gcfg, stream, Ws, Hs, lams, d_rgb, d_scrib, offs, peak, workload_name, batched, bs=None):
    """The solver's first global relabel (up to its height limit) and the push rounds after it,
    each as a launch of its own (gcfg_batch_phase_split), inside the NVTX
    range "phase_split".  A batch is split as one batch; the images of a
    per-image workload one at a time, as the plain solver runs them."""
    own = bs is None
    if own:
        bs = gcfg.BatchSolver(len(Ws) if batched else 1,
                              int(max(int(w) * int(h) for w, h in zip(Ws, Hs))) if not batched else
                              int(sum(int(w) * int(h) for w, h in zip(Ws, Hs))))
        bs.set_stream(stream)
    groups = [list(range(len(Ws)))] if batched else [[i] for i in range(len(Ws))]
    tot = {"ms_relabel": 0.0, "ms_push": 0.0, "relabel_tiles": 0, "push_tiles": 0, "push_sweeps": 0,
           "push_local_relabels": 0, "relabel_rounds": 0, "push_phases": 0, "active_pixels": 0, "tiles": 0}
    grid = []
    timeline = None
    for g in groups:
        w, h, lam = Ws[g], Hs[g], lams[g]
        if batched:
            rgb, scr = d_rgb, d_scrib
        else:
            i = g[0]
            o, n = int(offs[i]), int(Ws[i]) * int(Hs[i])
            rgb, scr = d_rgb[3 * o:3 * (o + n)], d_scrib[o:o + n]
        with nvtx_range("phase_split"):
            ps = bs.phase_split(w, h, lam, rgb, scr)
        if timeline is None:  # the first launch's relabel, round by round (device clock)
            timeline = {"round0_us": round(ps["relabel_round0_us"], 2), "pull_check_us": round(ps["relabel_pull_us"], 2),
                        "frontier_round_us": ps["relabel_front_us"], "frontier_round_tiles": ps["relabel_front_tiles"],
                        "frontier_round_work_us": ps["relabel_front_work_us"],
                        "frontier_round_longest_visit_kcyc": ps["relabel_front_maxvisit_kcyc"]}
        for k in tot:
            if k != "tiles":
                tot[k] += ps[k]
        tot["tiles"] += tiles_of(w, h)
        grid.append(ps["grid_blocks"])
    if own:
        bs.close()
    nt = tot["tiles"]
    gr = phase_record(tot["ms_relabel"],
                      1024 * (B_GR * min(tot["relabel_tiles"], nt) + B_COUNT * nt),
                      MOVED_GR_VISIT * tot["relabel_tiles"] + MOVED_GR_TILE * nt,
                      ncu_phase_traffic("gr", workload_name), peak,
                      launches=len(groups), tile_visits=tot["relabel_tiles"], frontier_rounds=tot["relabel_rounds"],
                      tiles=nt)
    gr["timeline_first_launch"] = timeline
    push = phase_record(tot["ms_push"], 1024 * B_PUSH * tot["push_tiles"], MOVED_PUSH_VISIT * tot["push_tiles"],
                        ncu_phase_traffic("push", workload_name), peak,
                        launches=len(groups), tile_visits=tot["push_tiles"], sweeps=tot["push_sweeps"],
                        local_relabels=tot["push_local_relabels"], colour_phases=tot["push_phases"])
    return {"global_relabel": gr, "push": push, "grid_blocks": max(grid),
            "how": "gcfg_batch_phase_split: launch 1 = initialisation + the first global relabel (up to its height "
                   "limit) + its count pass, launch 2 = the push rounds that follow (until the next global relabel), CUDA events "
                   "per launch; alg = bit planes read and heights written by the relabel (4.75 B/px once); "
                   "push 48 B/px per visited pixel; moved = what the phase reads and writes in this layout (relabel: mask "
                   "planes, halo lines, heights, border lines; push: the 24 KB tile in and out, halos, masks); "
                   "traffic = ncu dram__bytes_read.sum + dram__bytes_write.sum of the same launches"}


def profiled_roofline(gcfg, flush, run_once, Ws, Hs, batched, px, peak, peak_kind, workload_name):
    """One profiled pass (per-kernel CUDA events on the launching stream):
    the kernel with the largest device time and its algorithmic bytes."""
    gcfg.profile_enable(True)
    gcfg.profile_read()
    flush.fill_(7)
    recs = run_once()
    prof = gcfg.profile_read()
    gcfg.profile_enable(False)
    dom = max(prof, key=lambda k: prof[k]["ms"])
    tiles_total = tiles_of(Ws, Hs)
    solve_bytes = 0
    for j, r in enumerate(recs[:1] if batched else recs):
        nt = tiles_total if batched else tiles_of(Ws[j:j + 1], Hs[j:j + 1])
        solve_bytes += 1024 * (B_GR * min(r["gr_tiles"], nt * r["global_relabels"]) + B_PUSH * r["push_tiles"] +
                               B_REACH * min(r["reach_tiles"], nt) + B_COUNT * nt * r["global_relabels"] +
                               B_REACH * nt * r.get("closure_checks", 0))
    alg = {"solve": solve_bytes, "build": B_BUILD * 1024 * tiles_total, "extract": B_EXTRACT * px,
           "hist": 4 * px, "sigma": 3 * px}
    launches_dom = max(prof[dom]["launches"], 1)
    alg_bytes = alg.get(dom, 0)
    achieved = alg_bytes / (prof[dom]["ms"] / 1e3) / 1e9 if prof[dom]["ms"] > 0 else 0.0
    step_prof_ms = sum(v["ms"] for v in prof.values())
    return {"bound": "hbm", "kernel": dom, "achieved": achieved, "peak": peak, "unit": "GB/s",
            "frac": achieved / peak, "peak_source": peak_source(peak_kind),
            "traffic": ncu_traffic(dom, workload_name),
            "alg_bytes_per_launch": alg_bytes / launches_dom,
            "avg_launch_us": prof[dom]["ms"] / launches_dom * 1e3,
            "share_of_step": prof[dom]["ms"] / step_prof_ms if step_prof_ms else None,
            "kernels_ms": {k: round(v["ms"], 4) for k, v in prof.items() if v["launches"]}}, recs


def tuned_vs_default(gcfg, stream, Ws, Hs, lams, d_rgb, d_scrib, offs, flows, smin_all, smax_all, reps=5):
    """Each image of a single-image workload solved as a batch of one
    (gcfg_batch_run, device-resident) under the default solver settings and
    under the settings gcfg_batch_autotune picks for it (tile shape = the
    solver's thread block over each 32x32 tile, sweeps per global relabel,
    blocks per SM = blocks per image / SMs): best-of-`reps` device times
    (data term, build, solve, extraction) and the check that the tuned run's
    flow and cuts equal the plain solver's."""
    import torch
    out, eq, t_def, t_tun = [], True, 0.0, 0.0
    for i in range(len(Ws)):
        o, n = int(offs[i]), int(Ws[i]) * int(Hs[i])
        w, h, lam = Ws[i:i + 1], Hs[i:i + 1], lams[i:i + 1]
        rgb, scr = d_rgb[3 * o:3 * (o + n)], d_scrib[o:o + n]
        smin = torch.empty(n, dtype=torch.uint8, device="cuda")
        smax = torch.empty(n, dtype=torch.uint8, device="cuda")
        bs = gcfg.BatchSolver(1, n)
        bs.set_stream(stream)

        def best_ms():
            ms, fl = [], None
            for _ in range(reps):
                fl, res = bs.run(w, h, lam, rgb, scr, smin, smax, results=True)
                ms.append(res[0]["ms"])
            return min(ms), fl

        bs.set_solver()
        ms_def, fl_def = best_ms()
        tuning = bs.autotune(w, h, lam, rgb, scr, reps=2)
        ms_tun, fl_tun = best_ms()
        eq &= bool(fl_def[0] == flows[i] and fl_tun[0] == flows[i] and
                   np.array_equal(smin.cpu().numpy(), smin_all[o:o + n]) and
                   np.array_equal(smax.cpu().numpy(), smax_all[o:o + n]))
        bs.close()
        t_def += ms_def
        t_tun += ms_tun
        out.append({k: tuning[k] for k in ("threads_y", "push_rounds_per_gr", "max_tile_sweeps",
                                           "sweeps_per_local_relabel", "blocks_per_sm", "local_relabel_first",
                                           "push_only")} | {"default_ms": round(ms_def, 4), "tuned_ms": round(ms_tun, 4)})
    return {"default_ms": round(t_def, 4), "tuned_ms": round(t_tun, 4), "speedup": round(t_def / t_tun, 3),
            "per_image": out, "results_equal": eq,
            "how": "each image as a batch of one through gcfg_batch_run; best of 5 device times (data term to cuts) "
                   "under the default settings (solver block by size: 32 x 16 up to 2048 tiles, else 32 x 8; 2 push "
                   "rounds per global relabel, 16 sweeps, local relabel every 4) and under gcfg_batch_autotune's "
                   "choice for that image"}


def plain_leg(torch, gcfg, name, steps, warmup, flush, stream, peak, peak_kind, cpu_budget=10.0, ref_budget=5.0):
    """One single-image workload through the plain per-image solver
    (gcfg_seg_run): images resident in HBM (value), the same through
    gcfg_seg_run_host with pinned host buffers (e2e), the profiled roofline,
    the two solver phases as separate launches, the oracle on one host thread
    (cpu_baseline, with flow / S_min / S_max parity on every image) and the
    reference's CUDA path on the same images."""
    spec = workload(name)
    rgb, scrib, offs, Ws, Hs, lams = make_inputs(spec)
    views = image_views(rgb, scrib, offs, Ws, Hs)
    n_img, px = len(Ws), int(scrib.size)
    offs_l = [int(o) for o in offs]
    d_rgb, d_scrib = torch.from_numpy(rgb).cuda(), torch.from_numpy(scrib).cuda()
    d_smin = torch.empty(px, dtype=torch.uint8, device="cuda")
    d_smax = torch.empty(px, dtype=torch.uint8, device="cuda")
    h_rgb = torch.from_numpy(rgb).pin_memory().numpy()
    h_scrib = torch.from_numpy(scrib).pin_memory().numpy()
    h_smin = torch.empty(px, dtype=torch.uint8).pin_memory().numpy()
    h_smax = torch.empty(px, dtype=torch.uint8).pin_memory().numpy()
    seg = gcfg.Segmenter(int(Ws.max()), int(Hs.max()))
    seg.set_stream(stream)

    def step():
        out = []
        for i in range(n_img):
            o, n = offs_l[i], int(Ws[i]) * int(Hs[i])
            out.append(seg.run(d_rgb[3 * o:3 * (o + n)], d_scrib[o:o + n], int(Ws[i]), int(Hs[i]),
                               float(lams[i]), d_smin[o:o + n], d_smax[o:o + n]))
        return out

    def step_host():
        out = []
        for i in range(n_img):
            o, n = offs_l[i], int(Ws[i]) * int(Hs[i])
            out.append(seg.run_host(h_rgb[3 * o:3 * (o + n)], h_scrib[o:o + n], int(Ws[i]), int(Hs[i]),
                                    float(lams[i]), h_smin[o:o + n], h_smax[o:o + n]))
        return out

    for _ in range(warmup):
        step()
        step_host()
    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(steps)]
    res = None
    for i in range(steps):
        flush.fill_(i & 0xFF)
        ev[i][0].record(stream)
        res = step()
        ev[i][1].record(stream)
    torch.cuda.synchronize()
    ms = sum(a.elapsed_time(b) for a, b in ev) / steps
    flows = np.array([r["flow"] for r in res], np.int64)
    e2e_ms, res_h = [], None
    for i in range(steps):
        flush.fill_(i & 0xFF)
        torch.cuda.synchronize()
        t = time.perf_counter()
        res_h = step_host()
        e2e_ms.append((time.perf_counter() - t) * 1e3)
    e2e = float(np.mean(e2e_ms))
    host_equal = bool(np.array_equal(flows, [r["flow"] for r in res_h]) and np.array_equal(h_smin, d_smin.cpu().numpy())
                      and np.array_equal(h_smax, d_smax.cpu().numpy()))
    roof, _ = profiled_roofline(gcfg, flush, step, Ws, Hs, False, px, peak, peak_kind, name)
    roof["solve_phases"] = solve_phases(gcfg, stream, Ws, Hs, lams, d_rgb, d_scrib, offs, peak, name, False)
    smin_all, smax_all = d_smin.cpu().numpy(), d_smax.cpu().numpy()
    seg.close()
    tuned = tuned_vs_default(gcfg, stream, Ws, Hs, lams, d_rgb, d_scrib, offs, flows, smin_all, smax_all)
    cpu_v, n_chk, secs, parity = cpu_baseline(views, lams, budget_s=cpu_budget, flows_gpu=flows,
                                              smin_gpu=smin_all, smax_gpu=smax_all, offs=offs)
    leg = {"desc": spec["desc"], "images": n_img, "pixels": px, "value": px / (ms / 1e3) / 1e6, "unit": UNIT,
           "ms_per_step": ms, "steps": steps,
           "e2e": {"value": px / (e2e / 1e3) / 1e6, "unit": UNIT, "ms_per_step": e2e,
                   "h2d_bytes_per_step": 4 * px, "d2h_bytes_per_step": 2 * px,
                   "api": "gcfg_seg_run_host per image, pinned host buffers, wall clock per step",
                   "results_equal_device": host_equal},
           "roofline": roof, "tuned_vs_default": tuned,
           "solver": {k: res[0][k] for k in ("global_relabels", "closure_checks", "push_tiles", "gr_tiles",
                                             "push_sweeps", "push_local_relabels")},
           "cpu_baseline": {"value": cpu_v, "unit": UNIT, "cores": 1, "kind": "port",
                            "sample": f"{n_chk} solve(s) of the workload's images in {secs:.1f} s, oracle "
                                      "Boykov-Kolmogorov, 1 thread"},
           "parity": parity}
    if ref_budget > 0:
        leg["reference_cuda"] = reference_cuda_leg(views, lams, smax_all, offs, budget_s=ref_budget)
    return leg


def n8_leg(torch, gcfg, steps, warmup, peak, peak_kind, ref_budget=5.0):
    """8-neighbourhood graph (the reference's NEIGHBORHOOD == 8 build) at
    640x480: histogram t-links of a generated image, constant penalty 600 on
    all eight directions.  A step is GC_SetGraph8 + GC_Optimize8 (labels to
    the host) on device-resident t-links."""
    import oracle as O
    import synth
    W, H, pen = 640, 480, 600
    rgb, scrib = synth.generate(1, W, H, 7)
    d_rgb = torch.from_numpy(rgb.reshape(-1)).cuda()
    d_scrib = torch.from_numpy(scrib.reshape(-1)).cuda()
    dp = torch.empty(W * H, dtype=torch.int32, device="cuda")
    dn = torch.empty(W * H, dtype=torch.int32, device="cuda")
    gcfg.tlinks(d_rgb, d_scrib, dp, dn)
    gw = gcfg.GC_Init8(W, H, dp, dn, pen)
    label = torch.empty(W * H, dtype=torch.int32).pin_memory().numpy()
    d_smin = torch.empty(W * H, dtype=torch.uint8, device="cuda")
    for _ in range(warmup):
        gcfg.GC_SetGraph8(gw)
        gcfg.GC_Optimize8(gw, label)
    stream = torch.cuda.current_stream()
    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(steps)]
    torch.cuda.synchronize()
    solve_ms = []
    l0 = gcfg.launch_count()
    for i in range(steps):
        ev[i][0].record(stream)
        gcfg.GC_SetGraph8(gw)
        r = gcfg.GC_Optimize8(gw, label)
        ev[i][1].record(stream)
        solve_ms.append(r["ms"])
    torch.cuda.synchronize()
    launches = gcfg.launch_count() - l0
    ms = sum(a.elapsed_time(b) for a, b in ev) / steps
    gcfg.GC_GetCuts8(gw, d_smin, None)
    smin = d_smin.cpu().numpy().reshape(H, W)
    gcfg.GC_End8(gw)
    hdp, hdn = dp.cpu().numpy().reshape(H, W), dn.cpu().numpy().reshape(H, W)
    t = time.perf_counter()
    o = O.solve8(hdp, hdn, penalty=pen)
    cpu_s = time.perf_counter() - t
    value = W * H / (ms / 1e3) / 1e6
    # Algorithmic bytes of the solve kernel (eight int32 capacity planes): a
    # global relabel reads caps + excess for its masks and writes the height
    # (40 B/px; its count reads the masks); a visit of a 32x8 tile reads caps +
    # excess + height and writes them (80 B/px, an upper bound: only changes are
    # added back), a tile that is not due is one stamp (4 B); the cut pass reads
    # excess and writes the mark (8 B/px).
    n = W * H
    tiles8 = ((W + 31) // 32) * ((H + 7) // 8)
    visits, rounds = r["push_tiles"], r["push_rounds"]
    alg = r["global_relabels"] * n * 40 + visits * 256 * 80 + (rounds * tiles8 - visits) * 4 + n * 8
    avg_solve_ms = sum(solve_ms) / len(solve_ms)
    achieved = alg / (avg_solve_ms / 1e3) / 1e9
    roofline = {"bound": "hbm", "kernel": "k8_solve", "achieved": achieved, "peak": peak, "unit": "GB/s",
                "frac": achieved / peak, "peak_source": peak_source(peak_kind),
                "traffic": ncu_traffic("solve8", "n8_640x480"),
                "alg_bytes_per_launch": alg, "avg_launch_us": avg_solve_ms * 1e3,
                "note": "a 640x480 graph is about 15 MB in this layout and stays in L2; the solve is bound by "
                        "its grid barriers (one per tile or relabel round), not by HBM"}
    leg = {"desc": "8-neighbourhood graph, 640x480, histogram t-links of a generated image, penalty 600 on all "
                   "eight directions", "pixels": n, "value": value, "unit": UNIT, "ms_per_step": ms, "steps": steps,
           "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 4 * W * H,
                   "note": "labels to the host inside the timed step (GC_Optimize8); t-links resident"},
           "roofline": roofline, "gpu_launches": launches,
           "solver": {"global_relabels": r["global_relabels"], "gr_rounds": r["gr_sweeps"],
                      "tile_rounds": r["push_rounds"], "tile_visits": visits, "cut_rounds": r["cut_sweeps"]},
           "cpu_baseline": {"value": W * H / cpu_s / 1e6, "unit": UNIT, "cores": 1, "kind": "port",
                            "sample": f"one solve of the same graph, oracle 8-connected push-relabel, "
                                      f"{cpu_s:.2f} s"},
           "parity": {"flow_equal_oracle": bool(r["flow"] == o["flow"]),
                      "smax_equal_oracle": bool((label.reshape(H, W) == o["smax"]).all()),
                      "smin_equal_oracle": bool(np.array_equal(smin, o["smin"]))}}
    # the reference's own NEIGHBORHOOD 8 build of its kernels on the same GPU and graph
    import ref_cuda
    why = ref_cuda.unavailable(8) or ("not run (reference budget 0)" if ref_budget <= 0 else None)
    if why:
        leg["reference_cuda"] = {"unavailable": why}
    else:
        rr = [ref_cuda.solve8(hdp, hdn, penalty=pen, max_seconds=30.0) for _ in range(3)]
        best = min(x["ms_solve"] for x in rr)
        leg["reference_cuda"] = {
            "value": W * H / (best / 1e3) / 1e6, "unit": UNIT, "ms_per_image": best,
            "status": rr[-1]["status"], "iterations": rr[-1]["iterations"],
            "labels_equal": bool(np.array_equal(rr[-1]["label"], label.reshape(H, W))),
            "how": "the reference's kernels built with NEIGHBORHOOD 8 (GraphCutKernels.cu, sm_103a), launched in "
                   "GC_Optimize's order; best of 3 solves, wall clock of GC_SetGraph + GC_Optimize"}
    return leg


SINGLE_WORKLOADS = ("plain256", "plain1080", "plain4096")


def workload_config(name, spec, world):
    """The `config` object of a workload; both arms print the same one."""
    if name == "n8_640x480":
        return {"workload": name, "desc": "8-neighbourhood graph, 640x480, histogram t-links of a generated image, "
                "penalty 600 on all eight directions", "parallelism": f"replicas x{world}"}
    batched = spec["kind"] == "batch"
    px = int(sum(W * H for (_, W, H, _, _) in spec["images"]))
    return {"workload": name, "desc": spec["desc"], "images_per_step": len(spec["images"]),
            "pixels_per_step": px, "mode": "batched" if batched else "per-image",
            "l2": "GPU arm: flushed (256 MB write) before every step",
            "parallelism": (f"shard by image x{world}" if batched else f"replicas x{world}")}


def run_n8(args, rank, world):
    import torch
    import __graft_entry__ as ge
    ge.build()
    import gcfg
    peak, peak_kind = load_peaks()
    clocks = ClockSampler(torch.cuda.current_device())
    clocks.start()
    leg = n8_leg(torch, gcfg, args.steps, args.warmup, peak, peak_kind,
                 ref_budget=args.ref_cuda_budget)
    clk = clocks.stop()
    line = {"metric": METRIC, "value": leg["value"], "unit": UNIT, "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": leg["ms_per_step"], "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "int32", "data": "synthetic (seeded in-repo generator; no dataset)",
            "config": workload_config("n8_640x480", None, world), "clocks": clk}
    line.update({k: v for k, v in leg.items() if k not in ("desc", "value", "unit", "ms_per_step", "steps")})
    if rank == 0:
        emit(line)
    return 0


def run_reference_arm(args, spec, rank, world):
    """--impl reference: CPU port of the path on all host threads."""
    if rank != 0:
        return 0
    import oracle as O
    if args.workload == "n8_640x480":
        import synth
        W, H, pen = 640, 480, 600
        rgb, scrib = synth.generate(1, W, H, 7)
        dp, dn = O.tlinks(rgb, scrib)
        per_step = []
        for i in range(args.warmup + args.steps):
            t = time.perf_counter()
            O.solve8(dp, dn, penalty=pen)
            if i >= args.warmup:
                per_step.append(time.perf_counter() - t)
        value = W * H * len(per_step) / sum(per_step) / 1e6
        cores, sample, total_px = 1, "one 640x480 8-connected solve per step, oracle push-relabel, 1 thread", W * H
    else:
        rgb, scrib, offs, Ws, Hs, lams = make_inputs(spec)
        views = image_views(rgb, scrib, offs, Ws, Hs)
        cores = os.cpu_count() or 1
        reps = max(1, cores // len(views))
        per_step = []
        total_px = int(sum(s.size for _, s in views)) * reps
        for i in range(args.warmup + args.steps):
            t = time.perf_counter()
            O.segment_batch(views * reps, list(lams) * reps, cores)
            dt = time.perf_counter() - t
            if i >= args.warmup:
                per_step.append(dt)
        value = total_px * len(per_step) / sum(per_step) / 1e6
        sample = (f"{len(views)} image(s) x {reps} per step, oracle Boykov-Kolmogorov, one image per host thread; "
                  "the reference has no CPU solver (its CUDA path is timed in the reference_cuda leg of the "
                  "default arm)")
    line = {"impl": "reference", "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": sum(per_step) / len(per_step) * 1e3,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "int32",
            "data": "synthetic (seeded in-repo generator; no dataset)",
            "config": workload_config(args.workload, spec, world),
            "cpu_baseline": {"value": value, "unit": UNIT, "cores": cores, "kind": "port", "sample": sample},
            "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)
    return 0


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--workload", default="batch256")
    ap.add_argument("--cpu-budget", type=float, default=10.0)
    ap.add_argument("--no-plain", action="store_true", help="skip the per-image comparison leg")
    ap.add_argument("--no-serve", action="store_true", help="skip the serving leg")
    ap.add_argument("--no-single", action="store_true", help="skip the single-image legs")
    ap.add_argument("--no-tune", action="store_true", help="skip the autotuner (default solver settings)")
    ap.add_argument("--no-graph", action="store_true", help="run the batch without CUDA graph replay")
    ap.add_argument("--solver-params", default=None,
                    help="push_rounds,max_sweeps,sweeps_per_local_relabel[,blocks_per_sm[,relabel_first"
                         "[,push_only[,threads_y]]]] for the batch (skips the autotuner)")
    ap.add_argument("--serve-requests", type=int, default=1200)
    ap.add_argument("--ref-cuda-budget", type=float, default=15.0,
                    help="seconds of reference CUDA solve time for the reference_cuda leg (0 skips it)")
    args = ap.parse_args()
    args.warmup = max(args.warmup, 3)
    rank, world, local = dist_info()
    spec = None if args.workload == "n8_640x480" else workload(args.workload, rank)
    if args.impl == "reference":
        return run_reference_arm(args, spec, rank, world)
    if args.workload == "n8_640x480":
        import torch
        torch.cuda.set_device(local)
        return run_n8(args, rank, world)

    import torch
    import __graft_entry__ as ge
    ge.build()
    import gcfg

    torch.cuda.set_device(local)
    dist = None
    if world > 1:
        import torch.distributed as dist
        dist.init_process_group("nccl")

    def barrier():
        if dist is not None:
            dist.barrier()
        torch.cuda.synchronize()

    rgb, scrib, offs, Ws, Hs, lams = make_inputs(spec)
    views = image_views(rgb, scrib, offs, Ws, Hs)
    n_img = len(Ws)
    px_per_step = int(scrib.size)
    stream = torch.cuda.current_stream()
    d_rgb = torch.from_numpy(rgb).cuda()
    d_scrib = torch.from_numpy(scrib).cuda()
    d_smin = torch.empty(px_per_step, dtype=torch.uint8, device="cuda")
    d_smax = torch.empty(px_per_step, dtype=torch.uint8, device="cuda")
    h_rgb = torch.from_numpy(rgb).pin_memory().numpy()
    h_scrib = torch.from_numpy(scrib).pin_memory().numpy()
    h_smin = torch.empty(px_per_step, dtype=torch.uint8).pin_memory().numpy()
    h_smax = torch.empty(px_per_step, dtype=torch.uint8).pin_memory().numpy()
    flush = torch.empty(256 * 1024 * 1024, dtype=torch.uint8, device="cuda")
    peak, peak_kind = load_peaks()

    batched = spec["kind"] == "batch"
    bs = gcfg.BatchSolver(n_img, px_per_step)
    bs.set_stream(stream)
    seg = gcfg.Segmenter(int(Ws.max()), int(Hs.max()))
    seg.set_stream(stream)
    offs_l = [int(o) for o in offs]

    def step_batch():
        # flows only: the per-image diagnostic records are read in an untimed call
        flows, _ = bs.run(Ws, Hs, lams, d_rgb, d_scrib, d_smin, d_smax)
        return flows, None

    def step_plain():
        flows, res = [], []
        for i in range(n_img):
            o, n = offs_l[i], int(Ws[i]) * int(Hs[i])
            r = seg.run(d_rgb[3 * o:3 * (o + n)], d_scrib[o:o + n], int(Ws[i]), int(Hs[i]), float(lams[i]),
                        d_smin[o:o + n], d_smax[o:o + n])
            flows.append(r["flow"])
            res.append(r)
        return np.array(flows), res

    def step_host():
        if batched:
            return bs.run_host(Ws, Hs, lams, h_rgb, h_scrib, h_smin, h_smax)[0]
        flows = []
        for i in range(n_img):
            o, n = offs_l[i], int(Ws[i]) * int(Hs[i])
            r = seg.run_host(h_rgb[3 * o:3 * (o + n)], h_scrib[o:o + n], int(Ws[i]), int(Hs[i]),
                             float(lams[i]), h_smin[o:o + n], h_smax[o:o + n])
            flows.append(r["flow"])
        return np.array(flows)

    step = step_batch if batched else step_plain

    # solver settings for this batch (untimed), then CUDA graph replay
    tuning = None
    if batched and args.solver_params:
        keys = ("push_rounds_per_gr", "max_tile_sweeps", "sweeps_per_local_relabel", "blocks_per_sm",
                "local_relabel_first", "push_only", "threads_y")
        tuning = dict(zip(keys, (int(v) for v in args.solver_params.split(","))))
        bs.set_solver(**tuning)
        tuning["fixed"] = True
    elif batched and not args.no_tune:
        tuning = bs.autotune(Ws, Hs, lams, d_rgb, d_scrib, reps=2)
    if batched and not args.no_graph:
        bs.set_graph(True)

    def timed(fn, steps):
        ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(steps)]
        out = None
        for i in range(steps):
            flush.fill_(i & 0xFF)  # L2 flush (256 MB > 129 MB L2), outside the step's events
            ev[i][0].record(stream)
            out = fn()
            ev[i][1].record(stream)
        torch.cuda.synchronize()
        return sum(a.elapsed_time(b) for a, b in ev), out

    # host output buffers of the pipelined host leg (two batches in flight)
    h_out = [(h_smin, h_smax), (torch.empty(px_per_step, dtype=torch.uint8).pin_memory().numpy(),
                                torch.empty(px_per_step, dtype=torch.uint8).pin_memory().numpy())]

    def host_pipelined(steps):
        """`steps` batches through gcfg_batch_submit_host / gcfg_batch_wait,
        two in flight: each batch's inputs are copied in from pinned host
        memory and its labels copied out, overlapping the other's compute.
        No L2 flush: every batch uploads its inputs anew (187 MB on batch256,
        more than the 129 MB L2) and rebuilds its tile arena (about 1.5 GB)."""
        torch.cuda.synchronize()
        t = time.perf_counter()
        pending, fl = [], None
        for i in range(steps):
            o = h_out[i % 2]
            pending.append(bs.submit_host(Ws, Hs, lams, h_rgb, h_scrib, o[0], o[1]))
            if len(pending) == 2:
                fl, _ = bs.wait(pending.pop(0))
        for tk in pending:
            fl, _ = bs.wait(tk)
        return (time.perf_counter() - t) * 1e3, fl

    for _ in range(args.warmup):
        step()
        step_host()
    if batched:
        host_pipelined(max(2, args.warmup))
    if batched and not args.no_plain:
        step_plain()

    # ---- timed region: device-resident inputs ----
    clocks = ClockSampler(local)
    clocks.start()
    barrier()
    l0 = gcfg.launch_count()
    total_ms, (flows, results) = timed(step, args.steps)
    barrier()
    launches = gcfg.launch_count() - l0
    smin_dev, smax_dev = d_smin.cpu().numpy(), d_smax.cpu().numpy()

    # ---- e2e through the host entry point ----
    barrier()
    e2e_ms = []
    for i in range(args.steps):
        flush.fill_(i & 0xFF)
        torch.cuda.synchronize()
        t = time.perf_counter()
        flows_h = step_host()
        e2e_ms.append((time.perf_counter() - t) * 1e3)
    barrier()
    e2e_sync_total = sum(e2e_ms)
    e2e_total = e2e_sync_total
    flows_p = None
    if batched:
        barrier()
        e2e_total, flows_p = host_pipelined(args.steps)
        barrier()
    # the clock samples cover every timed region of the headline (device-resident and end to end)
    clk = clocks.stop()
    clk["window"] = "device-resident and end-to-end timed regions"
    cuts_host_equal = bool(np.array_equal(h_out[(args.steps - 1) % 2][0] if batched else h_smin, smin_dev) and
                           np.array_equal(h_out[(args.steps - 1) % 2][1] if batched else h_smax, smax_dev))

    # ---- the same images, plain per-image path (batched workload only) ----
    plain = None
    if batched and not args.no_plain:
        psteps = max(1, min(args.steps, 3))
        plain_ms, (pflows, _) = timed(step_plain, psteps)
        plain = {"value": px_per_step * psteps / (plain_ms / 1e3) / 1e6, "unit": UNIT,
                 "ms_per_step": plain_ms / psteps, "steps": psteps,
                 "flows_equal_batched": bool(np.array_equal(pflows, flows)),
                 "cuts_equal_batched": bool(np.array_equal(d_smin.cpu().numpy(), smin_dev) and
                                            np.array_equal(d_smax.cpu().numpy(), smax_dev))}

    import shard
    total_ms = shard.max_over_ranks(total_ms, device="cuda")
    e2e_total = shard.max_over_ranks(e2e_total, device="cuda")
    e2e_sync_total = shard.max_over_ranks(e2e_sync_total, device="cuda")
    value = world * px_per_step * args.steps / (total_ms / 1e3) / 1e6
    e2e_value = world * px_per_step * args.steps / (e2e_total / 1e3) / 1e6

    # ---- roofline: one profiled step, then the two solver phases as separate launches ----
    def run_once():
        if batched:
            return bs.run(Ws, Hs, lams, d_rgb, d_scrib, d_smin, d_smax, results=True)[1]
        return step_plain()[1]

    roofline, recs = profiled_roofline(gcfg, flush, run_once, Ws, Hs, batched, px_per_step, peak, peak_kind,
                                       args.workload)
    roofline["solve_phases"] = solve_phases(gcfg, stream, Ws, Hs, lams, d_rgb, d_scrib, offs, peak, args.workload,
                                            batched, bs=bs if batched else None)
    # in-solve phase timers of the profiled full solve (the same byte accounting)
    r_ph = recs[0]
    nt0 = tiles_of(Ws, Hs) if batched else tiles_of(Ws[:1], Hs[:1])
    inside = {}
    for name, nbytes, ms in (("global_relabel", 1024 * (B_GR * min(r_ph["gr_tiles"], nt0 * r_ph["global_relabels"]) +
                                                     B_REACH * nt0 * r_ph.get("closure_checks", 0)),
                              r_ph["t_global_relabel_ms"]),
                             ("push", 1024 * B_PUSH * r_ph["push_tiles"], r_ph["t_push_ms"])):
        if ms > 0:
            gbs = nbytes / (ms / 1e3) / 1e9
            inside[name] = {"achieved_alg_gbs": round(gbs, 1), "frac_alg": round(gbs / peak, 4), "ms": ms,
                            "alg_bytes": nbytes}
    inside["note"] = ("phase timers inside the whole solve (every global relabel and termination check, every push "
                      "round), algorithmic bytes")
    roofline["solve_phases"]["inside_full_solve"] = inside

    r0 = recs[0]
    config = workload_config(args.workload, spec, world)
    config.update(tuning=tuning, cuda_graph=bs.graph_info() if batched else None)
    line = {"metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": total_ms / args.steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "int32",
            "data": "synthetic (seeded in-repo generator; no dataset)",
            "config": config,
            "e2e": {"value": e2e_value, "unit": UNIT, "h2d_bytes_per_step": 4 * px_per_step,
                    "d2h_bytes_per_step": 2 * px_per_step, "ms_per_step": e2e_total / args.steps,
                    "api": ("gcfg_batch_submit_host/gcfg_batch_wait, 2 batches in flight, wall clock over "
                            "all steps; inputs uploaded anew every step (larger than L2), no flush" if batched else
                            "gcfg_seg_run_host per image, wall clock per step")},
            "e2e_sync": {"value": world * px_per_step * args.steps / (e2e_sync_total / 1e3) / 1e6,
                         "unit": UNIT, "ms_per_step": e2e_sync_total / args.steps,
                         "api": "one blocking host call per step (gcfg_batch_run_host / gcfg_seg_run_host)"},
            "roofline": roofline, "clocks": clk, "gpu_launches": launches,
            "solver": {k: (round(r0[k], 4) if isinstance(r0[k], float) else r0[k])
                       for k in ("global_relabels", "closure_checks", "closure_ends", "gr_sweeps", "push_rounds",
                                 "cut_sweeps", "push_tiles",
                                 "gr_tiles", "reach_tiles", "push_sweeps", "push_local_relabels",
                                 "t_global_relabel_ms", "t_count_ms", "t_push_ms", "t_push_tail_ms", "t_reach_ms",
                                 "cyc_load", "cyc_local_relabel", "cyc_sweeps", "cyc_writeback",
                                 "cyc_take", "bfs_iters_push", "bfs_iters_gr", "cyc_global_relabel")}}
    if plain is not None:
        line["plain_per_image"] = plain
    if batched and not args.no_serve and rank == 0:
        line["serving"] = serve_bench(torch, gcfg, n_req=args.serve_requests)
    line["flows_host_equal_device"] = bool(np.array_equal(np.asarray(flows_h), np.asarray(flows)) and
                                           (flows_p is None or np.array_equal(np.asarray(flows_p),
                                                                              np.asarray(flows))))
    line["cuts_host_equal_device"] = cuts_host_equal
    bs.close()
    seg.close()
    if rank == 0:
        cpu_v, n_chk, secs, parity = cpu_baseline(views, lams, budget_s=args.cpu_budget, flows_gpu=flows,
                                                  smin_gpu=smin_dev, smax_gpu=smax_dev, offs=offs)
        line["cpu_baseline"] = {"value": cpu_v, "unit": UNIT, "cores": 1, "kind": "port",
                                "sample": f"{n_chk} image(s) of the workload in {secs:.1f} s, oracle "
                                          "Boykov-Kolmogorov, 1 thread"}
        line["parity"] = parity
        if args.ref_cuda_budget > 0:
            line["reference_cuda"] = reference_cuda_leg(views, lams, smax_dev, offs,
                                                        budget_s=args.ref_cuda_budget)
        if batched and not args.no_single:
            legs = {}
            sclk = ClockSampler(local)
            sclk.start()
            for name in SINGLE_WORKLOADS:
                legs[name] = plain_leg(torch, gcfg, name, max(3, min(args.steps, 10)), args.warmup, flush, stream,
                                       peak, peak_kind, cpu_budget=min(args.cpu_budget, 5.0),
                                       ref_budget=min(args.ref_cuda_budget, 3.0))
            legs["n8_640x480"] = n8_leg(torch, gcfg, max(3, min(args.steps, 10)), args.warmup, peak, peak_kind,
                                        ref_budget=min(args.ref_cuda_budget, 3.0))
            legs["clocks"] = sclk.stop()
            line["single_image"] = legs
        emit(line)
    if dist is not None:
        dist.destroy_process_group()
    return 0


if __name__ == "__main__":
    sys.exit(main())
