"""Benchmark of the kazen GB300 hot path.

Headline workload (one step = one full frame): the plain wavefront path
tracer on the procedural terrain scene — 1024 x 1024-cell fBm heightfield
(2,097,152 triangles) + 64 icospheres (1,280 triangles each), Lambert / GGX
conductor / smooth dielectric materials, 4 quad lights, 1920 x 1080, 64 spp,
max depth 8, 16M-path wavefront, FP32. Metric: Mpaths*bounces/s (closest-hit
extension rays traced, camera rays included, per second).

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

`value` is device-resident throughput (scene built, film in HBM, CUDA events
around each frame on the scene stream, L2 flushed between frames); `e2e` is
the same metric through the C ABI with a host output buffer (the frame's
device->host copy inside the timed region). The traversal microbenchmark
(1,048,576-triangle soup, 16,777,216 incoherent rays) is reported alongside.
N > 1: independent replicas (the path tracer does not shard: no collective),
one per GPU, weak scaling, max-over-ranks time.
"""
from __future__ import annotations

import argparse
import json
import os
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

METRIC = "Mpaths*bounces/s (plain GPU wavefront PT)"
UNIT = "Mpaths*bounces/s"
NODE_BYTES = 80  # one 8-wide BVH node (kz_bvh.h)


def parse():
    p = argparse.ArgumentParser()
    p.add_argument("--gpus", type=int, default=1)
    p.add_argument("--steps", type=int, default=5)
    p.add_argument("--warmup", type=int, default=3)
    p.add_argument("--impl", default="ours", choices=["ours", "reference"])
    p.add_argument("--small", action="store_true", help="reduced workload (quick checks only)")
    p.add_argument("--profile", action="store_true",
                   help="full-size scene, 640x360 frame at 128 spp (29.5 M paths: full 2^24-path wavefronts), for ncu "
                        "captures of single launches")
    p.add_argument("--wavefront-log2", type=int, default=None,
                   help="paths in flight as a power of two (default 24 for the frame workloads)")
    p.add_argument("--no-cpu-baseline", action="store_true")
    p.add_argument("--no-traversal", action="store_true")
    p.add_argument("--no-guiding", action="store_true")
    p.add_argument("--no-box", action="store_true")
    p.add_argument("--no-batch", action="store_true")
    p.add_argument("--no-features", action="store_true")
    p.add_argument("--profile-wgrad", action="store_true",
                   help="guiding training steps at 2^18 rows (fused tcgen05, split tcgen05, mma.sync), for ncu "
                        "captures of the training kernels; prints the step times and exits")
    p.add_argument("--profile-guide", action="store_true",
                   help="one small guided render with training (slit room 128x128, 32 spp), for ncu captures "
                        "of the guiding network kernels; prints its stats and exits")
    return p.parse_args()


def workload(args):
    w = _workload(args)
    if getattr(args, "wavefront_log2", None):
        w["wavefront"] = 1 << args.wavefront_log2
    return w


def _workload(args):
    if args.small:
        return dict(width=320, height=180, spp=8, max_depth=8, cells=256, n_spheres=64, wavefront=1 << 18)
    if getattr(args, "profile", False):
        return dict(width=640, height=360, spp=128, max_depth=8, cells=1024, n_spheres=64, wavefront=1 << 24)
    return dict(width=1920, height=1080, spp=64, max_depth=8, cells=1024, n_spheres=64, wavefront=1 << 24)


def config_dict(w, extra=None):
    c = {"workload": "terrain_pt_%dx%d_%dspp_depth%d" % (w["width"], w["height"], w["spp"], w["max_depth"]),
         "triangles": None, "resolution": [w["width"], w["height"]], "spp": w["spp"], "max_depth": w["max_depth"],
         "wavefront": w["wavefront"], "scene": "fBm heightfield %dx%d cells + %d icospheres (subdiv 3) + 4 quad lights"
         % (w["cells"], w["cells"], w["n_spheres"]),
         "l2": "flushed between frames (256 MiB write); scene BVH+triangles and path state exceed L2"}
    if extra:
        c.update(extra)
    return c


def measured_peaks():
    path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(path):
        d = json.load(open(path))
        return d.get("hbm_gbs", 6800.0), "measured"
    return 6800.0, "fallback"


class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled during the timed region."""

    def __init__(self, index=0):
        self.index = index
        self.proc = None
        self.lines = []

    def start(self):
        q = ("clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,clocks_event_reasons.hw_slowdown,"
             "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
             "clocks_event_reasons.sw_power_cap")
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.index), "--query-gpu=" + q,
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except Exception:
            self.proc = None

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def stop(self):
        if not self.proc:
            return None
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        sm, mx, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            f = [x.strip() for x in ln.split(",")]
            if len(f) < 8:
                continue
            try:
                sm.append(float(f[0]))
                mx.append(float(f[1]))
            except ValueError:
                continue
            for k, nm in enumerate(names):
                if f[4 + k].lower().startswith("active"):
                    reasons.add(nm)
        if not sm:
            return None
        return {"sm_mhz": float(np.median(sm)), "sm_max_mhz": float(max(mx)), "reasons": sorted(reasons),
                "samples": len(sm)}


def dist_setup(n):
    if n <= 1 and "WORLD_SIZE" not in os.environ:
        return 0, 1, None
    import torch.distributed as dist
    rank = int(os.environ.get("RANK", 0))
    world = int(os.environ.get("WORLD_SIZE", n))
    backend = os.environ.get("KZ_BENCH_BACKEND", "nccl")
    if backend == "nccl":
        import torch
        torch.cuda.set_device(int(os.environ.get("LOCAL_RANK", 0)))
    dist.init_process_group(backend, rank=rank, world_size=world)
    return rank, world, dist


def aggregate(units_local: float, seconds_local: float, dist):
    """Whole-job throughput of replicas: total units / max-over-ranks time."""
    if dist is None:
        return units_local, seconds_local
    import torch
    dev = "cuda" if dist.get_backend() == "nccl" else "cpu"
    t = torch.tensor([seconds_local], dtype=torch.float64, device=dev)
    u = torch.tensor([units_local], dtype=torch.float64, device=dev)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    dist.all_reduce(u, op=dist.ReduceOp.SUM)
    return float(u.item()), float(t.item())


# ---------------------------------------------------------------- CPU baseline (restatement)
def strided_rows(H, count, offset=0):
    """`count` film rows spread evenly over the whole frame (shifted by
    `offset`), so a row sample sees the sky, the terrain and the spheres in
    the proportions the full frame has."""
    return sorted({(int((j + 0.5) * H / count) + offset) % H for j in range(count)})


def cpu_baseline(desc, w, budget_s=15.0):
    """The CPU restatement rendering whole rows of the same frame at the same
    spp on all host cores, rows strided over the whole frame, until about
    budget_s of work."""
    from oracle import oracle as O
    t0 = time.perf_counter()
    sc = O.Scene.from_desc(desc)
    build_s = time.perf_counter() - t0
    c = desc.camera
    cam = O.make_camera(c.eye, c.lookat, c.up, c.fov, c.flip)
    cores = os.cpu_count() or 1
    H = w["height"]
    bounces, secs, rows = 0, 0.0, 0
    for a in strided_rows(H, 64, offset=0) + strided_rows(H, 64, offset=3) + strided_rows(H, 128, offset=5):
        if secs >= budget_s:
            break
        ts = time.perf_counter()
        _, st = sc.render(cam, w["width"], H, w["spp"], w["max_depth"], seed=0, nthreads=cores, rows=(a, a + 1))
        secs += time.perf_counter() - ts
        bounces += st["path_bounces"]
        rows += 1
    return {"value": bounces / secs / 1e6, "unit": UNIT, "cores": cores, "kind": "port",
            "sample": "%d rows strided over the whole %d-row frame x %d px x %d spp (%d path*bounces, %.1f s; oracle "
                      "BVH build %.1f s untimed)" % (rows, H, w["width"], w["spp"], bounces, secs, build_s)}


# ---------------------------------------------------------------- traversal microbenchmark
def traversal_bench(steps, warmup):
    import torch

    from kazen_proto_gb300 import scenes
    tv = scenes.triangle_soup(1 << 20, seed=1)
    rays = scenes.soup_rays(1 << 24, seed=2)
    s = scenes.soup_desc(tv).build()
    stream = torch.cuda.Stream()  # a real stream: handle 0 would mean "the library's own stream"
    s.set_stream(stream)
    dr = torch.from_numpy(rays.view(np.float32).reshape(-1, 8)).cuda()
    n = dr.shape[0]
    out = {"t": torch.empty(n, dtype=torch.float32, device="cuda"),
           "prim_id": torch.empty(n, dtype=torch.int32, device="cuda")}
    occ = torch.empty(n, dtype=torch.uint8, device="cuda")
    flush = torch.empty(256 << 20, dtype=torch.uint8, device="cuda")
    nodes, tris = s.intersect_stats(dr)
    res = {}
    for name, fn in (("closest", lambda: s.intersect(dr, out=out)), ("any", lambda: s.occluded(dr, out=occ))):
        for _ in range(warmup):
            fn()
        s.synchronize()
        ms = 0.0
        for _ in range(steps):
            flush.fill_(1)
            torch.cuda.synchronize()
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream)
            fn()
            b.record(stream)
            torch.cuda.synchronize()
            ms += a.elapsed_time(b)
        s.synchronize()
        res[name + "_grays_per_s"] = n * steps / (ms / 1e3) / 1e9
        res[name + "_ms"] = ms / steps
    res["node_fetches_per_ray"] = nodes / n
    res["tri_fetches_per_ray"] = tris / n
    bytes_per_ray = 32 + 8 + NODE_BYTES * nodes / n + 48 * tris / n
    res["closest_alg_bytes_per_ray"] = bytes_per_ray
    res["closest_alg_gbs"] = bytes_per_ray * n / (res["closest_ms"] / 1e3) / 1e9
    res["workload"] = "1,048,576-triangle soup, 16,777,216 incoherent rays, device-resident"
    info = s.info()
    res["bvh_nodes"] = info["n_bvh_nodes"]
    res["bvh_depth"] = info["bvh_depth"]
    s.close()
    return res


# ---------------------------------------------------------------- the widened rows
def features_bench(W=960, H=540, spp=16, max_depth=8, frames=3):
    """Scene-file loading, the vertex-attribute shading variant and the closure
    kernels, each measured on its own (not part of the headline):
    * XML + OBJ + OSL lowering of the two scene fixtures (host seconds);
    * the terrain frame at 960x540, 16 spp with a checkerboard-textured
      terrain and smooth (vertex-normal) spheres, against the same frame
      plain: Mpaths*bounces/s of each, device-resident, L2 flushed;
    * kz_closure_eval_batch / kz_closure_sample_batch over 21 closure kinds
      (2^22 random lobes, device buffers): lobes per second."""
    import time

    import torch

    from kazen_proto_gb300 import _native as N
    from kazen_proto_gb300 import api, scene_xml, scenes
    here = os.path.dirname(os.path.abspath(__file__))
    res = {}
    for name in ("box_room", "textured_room"):
        t0 = time.perf_counter()
        L = scene_xml.load(os.path.join(here, "tests", "golden", "scenes", name, "scene.xml"))
        res[f"load_{name}_s"] = round(time.perf_counter() - t0, 4)
        res[f"load_{name}_triangles"] = int(L.desc.n_triangles())

    flush = torch.empty(256 << 20, dtype=torch.uint8, device="cuda")
    rgb = torch.empty((H, W, 3), dtype=torch.float32, device="cuda")

    def frame_rate(desc):
        s = desc.build()
        stream = torch.cuda.Stream()
        s.set_stream(stream)
        r = api.Renderer(spp=spp, max_depth=max_depth, seed=5)
        r.render(s, desc.camera, W, H, device_out=(rgb, None))
        s.synchronize()
        ms, bounces = 0.0, 0
        for _ in range(frames):
            flush.fill_(1)
            torch.cuda.synchronize()
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream)
            r.render(s, desc.camera, W, H, device_out=(rgb, None))
            b.record(stream)
            torch.cuda.synchronize()
            ms += a.elapsed_time(b)
            bounces += r.last_stats["path_bounces"]
        s.close()
        return bounces / (ms / 1e3) / 1e6

    plain = scenes.terrain_scene(W, H, spp, max_depth)
    res["terrain_plain_mpaths_bounces_per_s"] = round(frame_rate(plain), 1)
    feat = scenes.terrain_scene(W, H, spp, max_depth)
    feat.textures = [api.checker_texture(64, 64, (0.7, 0.7, 0.65), (0.3, 0.3, 0.35))]
    feat.materials[0] = api.material([api.textured(api.diffuse((0.8, 0.8, 0.8)), 0)])
    for g in range(1, len(feat.meshes)):
        v, i, m, light = feat.meshes[g]
        if not light:  # the icospheres: radial vertex normals about their centroid
            n = v - v.mean(axis=0)
            feat.normals[g] = (n / np.linalg.norm(n, axis=1, keepdims=True)).astype(np.float32)
    res["terrain_textured_smooth_mpaths_bounces_per_s"] = round(frame_rate(feat), 1)
    res["terrain_frame"] = f"{W}x{H}, {spp} spp, depth {max_depth}"

    rng = np.random.default_rng(3)
    n = 1 << 22
    a, e = 0.3, 1.4
    kinds = [api.diffuse(), api.mirror(), api.dielectric(1.5, 1.0), api.microfacet("ggx", a, 0.5 * a, e, 0),
             api.microfacet("beckmann", a, a, e, 0), api.microfacet("ggx", a, a, e, 1),
             api.microfacet("beckmann", a, a, e, 2), api.conductor_ggx((0.9, 0.6, 0.5), a),
             api.principle_specular((0.1, 0.1, 0.1), a, e, 0.3), api.phong(30.0), api.ward(a), api.ward(a, 0.5 * a),
             api.reflection(e), api.refraction(e), api.transparent(), api.translucent(),
             api.kp_microfacet(a, 1.5, 1.0, 0.4), api.principle_diffuse(), api.principle_retro(0.5),
             api.principle_fakess(0.5), api.principle_clearcoat(0.1)]
    rec = np.array([kinds[k % len(kinds)] for k in range(1 << 16)], dtype=N.LOBE_DTYPE)
    lobes = torch.from_numpy(rec.view(np.uint8).reshape(1 << 16, -1)).cuda().repeat(n >> 16, 1)

    def dirs(m):
        d = rng.standard_normal((m, 3)).astype(np.float32)
        return d / np.linalg.norm(d, axis=1, keepdims=True)
    wi = torch.from_numpy(np.tile(dirs(1 << 16), (n >> 16, 1))).cuda()
    wo = torch.from_numpy(np.tile(dirs(1 << 16), (n >> 16, 1))).cuda()
    u = torch.rand((n, 3), device="cuda")
    f = torch.empty((n, 3), device="cuda")
    pdf = torch.empty(n, device="cuda")
    w3 = torch.empty((n, 3), device="cuda")
    fl = torch.empty(n, dtype=torch.uint8, device="cuda")
    lib = N.lib()

    def timed(fn, reps=5):
        fn()
        torch.cuda.synchronize()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(reps):
            fn()
        b.record()
        torch.cuda.synchronize()
        return a.elapsed_time(b) / reps

    P = lambda t: t.data_ptr()  # noqa: E731
    ev = timed(lambda: N.check(lib.kz_closure_eval_batch(P(lobes), P(wi), P(wo), n, N.KZ_CONVENTION_INTEGRATOR,
                                                         P(f), P(pdf), N.KZ_MEM_DEVICE)))
    sm = timed(lambda: N.check(lib.kz_closure_sample_batch(P(lobes), P(wi), P(u), n, P(wo), P(w3), P(pdf), P(fl),
                                                           N.KZ_MEM_DEVICE)))
    res["closure_eval_globes_per_s"] = round(n / (ev / 1e3) / 1e9, 3)
    res["closure_sample_globes_per_s"] = round(n / (sm / 1e3) / 1e9, 3)
    res["closure_batch"] = f"{n} lobes of {len(kinds)} closure kinds, device buffers"
    return res


# ---------------------------------------------------------------- small box (the reference CPU-path config)
def box_bench(frames=20, W=256, H=256, spp=16, max_depth=5):
    """The small-box workload at its stated size (36 triangles, 256 x 256,
    16 spp, depth 5, NEE+MIS, FP32): device-resident frames (CUDA events on
    the scene stream), frames through the C ABI with a host film, relMSE of
    the GPU image against the restatement's FP64 render of the same PCG32
    streams and of its 1024-spp image against an independent 16,384-spp FP64
    GPU render, and the restatement rendering the whole frame on all host
    cores."""
    import torch

    from kazen_proto_gb300 import api, scenes
    from oracle import oracle as O

    def rel_mse(img, ref, eps=1e-2):
        return float(np.mean((np.asarray(img, np.float64) - ref) ** 2 / (ref ** 2 + eps)))

    d = scenes.box_scene(W, H, spp=spp, max_depth=max_depth)
    s = d.build()
    stream = torch.cuda.Stream()
    s.set_stream(stream)
    r = api.Renderer(spp=spp, max_depth=max_depth, seed=1)
    rgb = torch.empty((H, W, 3), dtype=torch.float32, device="cuda")
    for _ in range(3):
        r.render(s, d.camera, W, H, device_out=(rgb, None))
    s.synchronize()
    ms, bounces = 0.0, 0
    for _ in range(frames):
        torch.cuda.synchronize()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        r.render(s, d.camera, W, H, device_out=(rgb, None))
        b.record(stream)
        torch.cuda.synchronize()
        ms += a.elapsed_time(b)
        bounces += r.last_stats["path_bounces"]
    e2e_s = 0.0
    for _ in range(frames):
        t0 = time.perf_counter()
        r.render(s, d.camera, W, H)
        e2e_s += time.perf_counter() - t0
    img, img64 = r.render(s, d.camera, W, H, fp64=True)
    osc = O.Scene.from_desc(d)
    c = d.camera
    cam = O.make_camera(c.eye, c.lookat, c.up, c.fov, c.flip)
    cores = os.cpu_count() or 1
    t0 = time.perf_counter()
    ref, cst = osc.render(cam, W, H, spp, max_depth, seed=1, nthreads=cores)
    cpu_s = time.perf_counter() - t0
    img1k = api.Renderer(spp=1024, max_depth=max_depth, seed=3).render(s, d.camera, W, H)
    hi = api.Renderer(spp=16384, max_depth=max_depth, seed=77).render(s, d.camera, W, H, fp64=True)[1]
    s.close()
    per_frame = bounces / frames
    return {"workload": "box_256x256_16spp_depth5 (36 triangles, NEE+MIS, FP32)",
            "device_ms_per_frame": round(ms / frames, 3),
            "mpaths_bounces_per_s": round(bounces / (ms / 1e3) / 1e6, 1),
            "e2e_ms_per_frame": round(e2e_s / frames * 1e3, 3),
            "e2e_mpaths_bounces_per_s": round(per_frame * frames / e2e_s / 1e6, 1),
            "relmse_vs_restatement_fp64_same_streams": rel_mse(img64, ref),
            "relmse_1024spp_vs_independent_16384spp_fp64": rel_mse(img1k, hi),
            "cpu_baseline": {"value": round(cst["path_bounces"] / cpu_s / 1e6, 2), "unit": UNIT, "cores": cores,
                             "kind": "port", "seconds": round(cpu_s, 3),
                             "sample": "the whole 256x256 frame at 16 spp (%d path*bounces)" % cst["path_bounces"]}}


# ---------------------------------------------------------------- learned guiding, equal time
def guiding_bench(R=1024, budgets_spp=(1024, 2048), ref_spp=65536, max_depth=10, lr=1e-3, rows=1 << 18):
    """Learned guiding at its stated size: the narrow-aperture slit room at
    R x R, depth 10, Adam at lr 1e-3 on 2^18 radiance samples per training
    step. For each budget, plain path tracing at that spp sets the wall-clock
    time and guided path tracing (network trained online from scratch, inside
    the same wall-clock time) renders until the time is up; relMSE of each
    against a plain FP64 reference of ref_spp, rendered as two independent
    halves so the reference's own noise is stated (and subtracted in the
    `_net` ratios). Also the equal-spp error of the network trained in the
    first budget."""
    from kazen_proto_gb300 import api, scenes

    def rel_mse(img, ref, eps=1e-2):
        return float(np.mean((np.asarray(img, np.float64) - ref) ** 2 / (ref ** 2 + eps)))

    d = scenes.slit_room_scene(R, R, max_depth=max_depth)
    s = d.build()
    t0 = time.perf_counter()
    chunk = min(ref_spp // 2, (1 << 31) // (R * R))  # path ids of one render stay below 2^32
    halves = []
    for h in range(2):
        parts = [api.Renderer(spp=chunk, max_depth=max_depth, seed=99 + 1000 * h + k).render(
            s, d.camera, R, R, fp64=True)[1] for k in range(max(1, (ref_spp // 2) // chunk))]
        halves.append(np.mean(parts, axis=0))
    ref = 0.5 * (halves[0] + halves[1])
    ref_noise = float(np.mean(((halves[0] - halves[1]) * 0.5) ** 2 / (ref ** 2 + 1e-2)))
    ref_s = time.perf_counter() - t0
    g = api.Guide(seed=3)
    api.render_guided(s, g, d.camera, R, R, spp=4, max_depth=max_depth, seed=2,
                      gcfg=api.guide_config(train=False, spp_per_pass=4))  # warm-up (kernels, buffers)
    g.close()
    runs = []
    frozen = None
    for bi, spp in enumerate(budgets_spp):
        r = api.Renderer(spp=spp, max_depth=max_depth, seed=1 + bi)
        if bi == 0:
            r.render(s, d.camera, R, R)  # warm-up
        t0 = time.perf_counter()
        img_p = r.render(s, d.camera, R, R)
        T = time.perf_counter() - t0
        e_plain = rel_mse(img_p, ref)
        g = api.Guide(seed=3)
        gc = GUIDE_SETTINGS(lr, rows, T, spp)
        t0 = time.perf_counter()
        img_g, _, st, gst = api.render_guided(s, g, d.camera, R, R, spp=1 << 20, max_depth=max_depth, seed=7 + bi,
                                              gcfg=gc)
        Tg = time.perf_counter() - t0
        e_guided = rel_mse(img_g, ref)
        runs.append({"plain": {"spp": spp, "seconds": round(T, 4), "relmse": e_plain},
                     "guided": {"seconds": round(Tg, 4), "spp": gst["spp_done"], "train_steps": gst["train_steps"],
                                "train_ms": round(gst["train_ms"], 1), "train_samples": gst["train_samples"],
                                "relmse": e_guided},
                     "relmse_ratio_plain_over_guided": round(e_plain / e_guided, 3),
                     "relmse_ratio_plain_over_guided_net": round((e_plain - ref_noise) / max(1e-12, e_guided - ref_noise),
                                                                 3)})
        if bi == 0:
            t0 = time.perf_counter()
            img_f, _, _, _ = api.render_guided(s, g, d.camera, R, R, spp=spp, max_depth=max_depth, seed=11,
                                               gcfg=api.guide_config(alpha=gc.alpha, train=False, spp_per_pass=64))
            Tf = time.perf_counter() - t0
            e_f = rel_mse(img_f, ref)
            frozen = {"spp": spp, "seconds": round(Tf, 4), "relmse": e_f, "train_steps": gst["train_steps"],
                      "relmse_ratio_plain_over_guided": round(e_plain / e_f, 3),
                      "cost_per_sample_vs_plain": round(Tf / T, 3)}
        g.close()
    s.close()
    net = network_bench()
    return {"scene": "slit room %dx%d, max depth %d, 24 Lambert quads + 32 GGX spheres, 4x4 exterior light "
                     "(radiance 200) behind a 0.05x0.5 slit" % (R, R, max_depth),
            "training_step": net,
            "network": "51 -> 64 -> 64 -> 64 -> 40 (8 vMF lobes), BF16 weights, FP32 accumulation, Adam lr %g, "
                       "%d radiance samples per training step" % (lr, rows),
            "reference": "plain, %d spp, FP64 accumulation, two independent halves (%.1f s)" % (ref_spp, ref_s),
            "reference_noise_relmse": ref_noise,
            "equal_time": runs, "guided_trained_equal_spp": frozen}


def GUIDE_SETTINGS(lr, rows, seconds, budget_spp):
    """Guided-render settings of the equal-time runs (online training from
    scratch inside the wall-clock budget): one spp per training pass, eight
    Adam steps per pass, as many steps as the plain budget has spp (then the
    network is frozen and the remaining time renders with it). Measured at
    1024^2 on the slit room against 16-spp passes with 4 steps (0.40x /
    0.45x of plain at 1,024 / 2,048 spp budgets): 0.51x / 0.75x."""
    from kazen_proto_gb300 import api
    return api.guide_config(spp_per_pass=1, steps_per_pass=8, learning_rate=lr, max_train_steps=budget_spp,
                            max_train_samples=rows, time_budget_ms=seconds * 1e3)


# ---------------------------------------------------------------- batched uneven jobs
def batch_bench(n_jobs=256):
    """256 seeded soup jobs (50k-500k triangles; 64..512 squared; 4/16/64
    spp; depth 4 or 8): one kz_render_batch call (autotuned mode and shape,
    CUDA graphs) against the same jobs rendered one kz_render call each."""
    from kazen_proto_gb300 import api, autotune, scenes

    t0 = time.perf_counter()
    jobs = scenes.build_batch_scenes(scenes.batch_jobs(n_jobs=n_jobs, seed=5), workers=16)
    build_s = time.perf_counter() - t0
    # autotune on a sample of the jobs at reduced spp
    sample = [dict(j, spp=min(j["spp"], 4)) for j in jobs[::8]]
    best, table = autotune.tune(sample, reps=1)
    cfg = autotune.tuned_config(use_graph=True)
    api.render_batch(jobs[:4], cfg)  # warm-up
    t0 = time.perf_counter()
    imgs, st = api.render_batch(jobs, cfg)
    wall_b = time.perf_counter() - t0
    # one launch (one kz_render call) per job
    singles_ms, singles_wall, bounces_single = 0.0, 0.0, 0
    errs = []
    for j, img in zip(jobs, imgs):
        r = api.Renderer(spp=j["spp"], max_depth=j["max_depth"], seed=j["seed"], flags=0)
        t0 = time.perf_counter()
        ref = r.render(j["scene"], j["camera"], j["width"], j["height"])
        singles_wall += time.perf_counter() - t0
        bounces_single += r.last_stats["path_bounces"]
        errs.append(float(np.abs(img - ref).max() / max(1e-6, float(np.abs(ref).max()))))
        j["scene"].release_scratch()
    # the megakernel mode at its own best tuned shape, for comparison
    mega = [t for t in table if t[0].get("mode") == api.BATCH_MEGAKERNEL]
    best_mega = min(mega, key=lambda t: t[1])[0] if mega else {"mode": api.BATCH_MEGAKERNEL}
    mcfg = autotune.config_of(best_mega, use_graph=True)
    t0 = time.perf_counter()
    _, mst = api.render_batch(jobs, mcfg)
    wall_m = time.perf_counter() - t0
    # the whole wavefront loop in one cooperative launch, at its best tuned shape
    pers = [t for t in table if t[0].get("mode") == api.BATCH_PERSISTENT]
    best_pers = min(pers, key=lambda t: t[1])[0] if pers else {"mode": api.BATCH_PERSISTENT}
    t0 = time.perf_counter()
    pimgs, pst = api.render_batch(jobs, autotune.config_of(best_pers, use_graph=True))
    wall_p = time.perf_counter() - t0
    perr = max(float(np.abs(a - b).max() / max(1e-6, float(np.abs(b).max()))) for a, b in zip(pimgs, imgs))
    del pimgs
    for j in jobs:
        j["scene"].close()
    mb = st["path_bounces"] / (st["device_ms"] / 1e3) / 1e6
    return {"jobs": n_jobs, "paths": st["paths"], "path_bounces": st["path_bounces"],
            "triangles_total": int(sum(j["desc_args"][0] + 2 for j in jobs)), "scene_build_s": round(build_s, 1),
            "autotuned": best, "autotune_candidates": len(table), "persistent_lanes": st["threads"],
            "autotune_sample_ms_best_per_mode": {
                "wavefront": min((ms for c, ms in table if c.get("mode") == api.BATCH_WAVEFRONT), default=None),
                "megakernel": min((ms for c, ms in table if c.get("mode") == api.BATCH_MEGAKERNEL), default=None),
                "persistent": min((ms for c, ms in table if c.get("mode") == api.BATCH_PERSISTENT), default=None)},
            "autotune_wavefront_by_refill_period": {
                str(p): min((ms for c, ms in table if c.get("mode") == api.BATCH_WAVEFRONT
                             and c.get("refill_period") == p), default=None) for p in autotune.WAVE_PERIODS},
            "megakernel_tuned": best_mega,
            "batched_graph": {"device_ms": round(st["device_ms"], 2), "wall_s": round(wall_b, 3),
                              "mpaths_bounces_per_s": round(mb, 1)},
            "persistent_tuned": best_pers,
            "persistent_one_launch_graph": {
                "device_ms": round(pst["device_ms"], 2), "wall_s": round(wall_p, 3),
                "mpaths_bounces_per_s": round(pst["path_bounces"] / (pst["device_ms"] / 1e3) / 1e6, 1),
                "max_rel_difference_vs_batched": perr},
            "megakernel_graph": {"device_ms": round(mst["device_ms"], 2), "wall_s": round(wall_m, 3),
                                 "mpaths_bounces_per_s": round(mst["path_bounces"] / (mst["device_ms"] / 1e3) / 1e6,
                                                               1)},
            "one_launch_each": {"wall_s": round(singles_wall, 3),
                                "mpaths_bounces_per_s": round(bounces_single / singles_wall / 1e6, 1)},
            "speedup_wall": round(singles_wall / wall_b, 3),
            "max_rel_film_difference": max(errs)}


TRACE_KERNEL = "k_trace_paths_persistent"


def load_traffic():
    """Per-ray DRAM bytes and the issue/divergence counters of the closest-hit
    kernel from the committed ncu summary."""
    import re
    path = os.path.join(ROOT, "profiles", "k_trace_paths_persistent_terrain_profile.md")
    if not os.path.exists(path):
        return None
    txt = open(path).read()
    out = {"kernel": TRACE_KERNEL}
    for key in ("dram_bytes_per_ray", "simt_lanes_active", "issue_active"):
        m = re.search(r"^%s:\s*([0-9.]+)" % key, txt, re.M)
        if m:
            out[key] = float(m.group(1))
    return out if "dram_bytes_per_ray" in out else None


def network_bench(rows=1 << 18, steps=20):
    """The guiding network's training step at its stated batch (2^18 radiance
    samples, random positions, normals and directions, device-resident): mean
    wall time per step (forward + mixture loss + backward + weight gradients)
    of the three implementations: one tcgen05 kernel (the default), the
    warp-level forward/backward with tcgen05 weight gradients, and both
    warp-level (KZ_GUIDE_TRAIN = fused / tc / mma)."""
    import ctypes as C

    import torch

    from kazen_proto_gb300 import _native as N
    from kazen_proto_gb300 import api
    rng = np.random.default_rng(1)
    smp = np.zeros((rows, 12), np.float32)
    smp[:, 0:3] = rng.random((rows, 3))
    smp[:, 3] = rng.random(rows) + 0.1
    n = rng.standard_normal((rows, 3))
    smp[:, 4:7] = n / np.linalg.norm(n, axis=1, keepdims=True)
    dv = rng.standard_normal((rows, 3))
    smp[:, 8:11] = dv / np.linalg.norm(dv, axis=1, keepdims=True)
    dsmp = torch.from_numpy(smp).cuda()
    g = api.Guide(seed=2)
    lib = N.lib()
    loss = C.c_float()
    out = {}
    for name, val in (("fused_tcgen05", "fused"), ("split_tcgen05_wgrad", "tc"), ("mma_sync", "mma")):
        os.environ["KZ_GUIDE_TRAIN"] = val
        for _ in range(3):
            N.check(lib.kz_guide_train_step(g.handle, C.c_void_p(dsmp.data_ptr()), rows, 1e-3, 0, C.byref(loss),
                                            None, N.KZ_MEM_DEVICE))
        t0 = time.perf_counter()
        for _ in range(steps):
            N.check(lib.kz_guide_train_step(g.handle, C.c_void_p(dsmp.data_ptr()), rows, 1e-3, 0, C.byref(loss),
                                            None, N.KZ_MEM_DEVICE))
        out[name + "_ms_per_step"] = round((time.perf_counter() - t0) / steps * 1e3, 3)
    os.environ.pop("KZ_GUIDE_TRAIN", None)
    g.close()
    out["rows"] = rows
    out["note"] = "wall time per kz_guide_train_step call (device samples, gradient only, one host sync per step)"
    return out


def profile_wgrad():
    """Training steps at 2^18 rows in each implementation (three warm-up
    steps, then four timed ones, per implementation): the command the
    training-kernel ncu captures run."""
    from kazen_proto_gb300 import build as kbuild
    kbuild.build()
    print(json.dumps({"workload": "guide_train_step_262144_rows", **network_bench(steps=4)}))


def profile_guide():
    """Small guided render with online training: the command the guiding
    network's ncu captures run."""
    from kazen_proto_gb300 import api, build as kbuild, scenes
    kbuild.build()
    R, D = 128, 10
    d = scenes.slit_room_scene(R, R, max_depth=D)
    s = d.build()
    g = api.Guide(seed=3)
    _, _, st, gst = api.render_guided(s, g, d.camera, R, R, spp=32, max_depth=D, seed=7,
                                      gcfg=api.guide_config(spp_per_pass=16, steps_per_pass=4, learning_rate=1e-2))
    print(json.dumps({"workload": "slit_room_128x128_32spp_guided_training", "render": st, "guide": gst}))
    g.close()
    s.close()


# ---------------------------------------------------------------- our arm
def run_ours(args):
    import torch

    rank, world, dist = dist_setup(args.gpus)
    from kazen_proto_gb300 import _native as N
    from kazen_proto_gb300 import api, build as kbuild, scenes
    kbuild.build()
    dev_index = int(os.environ.get("LOCAL_RANK", 0))
    torch.cuda.set_device(dev_index)
    w = workload(args)
    desc = scenes.terrain_scene(w["width"], w["height"], w["spp"], w["max_depth"], w["cells"], w["n_spheres"])
    s = desc.build()
    stream = torch.cuda.Stream()  # a real stream: handle 0 would mean "the library's own stream"
    s.set_stream(stream)
    W, H = w["width"], w["height"]
    seed = 1000 * rank
    r = api.Renderer(spp=w["spp"], max_depth=w["max_depth"], seed=seed, wavefront_size=w["wavefront"],
                     flags=N.KZ_RENDER_FLAG_TIMING)
    rgb = torch.empty((H, W, 3), dtype=torch.float32, device="cuda")
    flush = torch.empty(256 << 20, dtype=torch.uint8, device="cuda")

    for _ in range(args.warmup):
        r.render(s, desc.camera, W, H, device_out=(rgb, None))
    torch.cuda.synchronize()
    clocks = ClockSampler(dev_index)
    clocks.start()
    if dist is not None:
        dist.barrier()
    total_ms, bounces, shadow, launches, iterations = 0.0, 0, 0, 0, 0
    stage = {"generate_ms": 0.0, "trace_ms": 0.0, "shade_ms": 0.0, "shadow_ms": 0.0}
    for _ in range(args.steps):
        flush.fill_(1)
        torch.cuda.synchronize()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        r.render(s, desc.camera, W, H, device_out=(rgb, None))
        b.record(stream)
        torch.cuda.synchronize()
        total_ms += a.elapsed_time(b)
        st = r.last_stats
        bounces += st["path_bounces"]
        shadow += st["shadow_rays"]
        launches += st["kernel_launches"] + 1  # + the film scale kernel
        iterations += st["iterations"]
        for k in stage:
            stage[k] += st[k]
    if dist is not None:
        dist.barrier()
    torch.cuda.synchronize()
    clk = clocks.stop()
    units, secs = aggregate(bounces, total_ms / 1e3, dist)

    # e2e through the C ABI with a host output buffer (pinned, reused across
    # frames as a renderer would)
    img = torch.empty((H, W, 3), dtype=torch.float32, pin_memory=True)
    e2e_bounces, e2e_s = 0, 0.0
    for k in range(args.steps):
        flush.fill_(1)
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        img = r.render(s, desc.camera, W, H, out=img)
        e2e_s += time.perf_counter() - t0
        e2e_bounces += r.last_stats["path_bounces"]
    e_units, e_secs = aggregate(e2e_bounces, e2e_s, dist)

    # The roofline's kernel traces the rays after the camera's: those are traced
    # in bundles, by a kernel that also generates them. Its time is the trace
    # stage's less that of frames of depth 1, its fetches those of a counted frame
    # at reduced spp less those of depth 1 (untimed, after the timed region so
    # profiler launch indices are unaffected).
    def stats_of(**kw):
        k = api.Renderer(seed=seed, wavefront_size=w["wavefront"], **kw)
        k.render(s, desc.camera, W, H, device_out=(rgb, None))
        return k.last_stats
    camera_ms = min(stats_of(spp=w["spp"], max_depth=1, flags=N.KZ_RENDER_FLAG_TIMING)["trace_ms"] for _ in range(3))
    cs, c1 = (stats_of(spp=max(1, w["spp"] // 16), max_depth=d, flags=N.KZ_RENDER_FLAG_COUNT)
              for d in (w["max_depth"], 1))
    counted_rays = max(1, cs["path_bounces"] - c1["path_bounces"])
    nodes_per_ray = (cs["closest_node_fetches"] - c1["closest_node_fetches"]) / counted_rays
    tris_per_ray = (cs["closest_tri_fetches"] - c1["closest_tri_fetches"]) / counted_rays

    sections = {}

    def timed_section(name, fn):
        t0 = time.perf_counter()
        out = fn()
        sections[name] = round(time.perf_counter() - t0, 1)
        return out

    trav = None
    if rank == 0 and not args.no_traversal and not args.small and not args.profile:
        trav = timed_section("traversal", lambda: traversal_bench(max(3, args.steps), max(3, args.warmup)))

    box = None
    if rank == 0 and not args.no_box and not args.small and not args.profile:
        box = timed_section("box", box_bench)

    guide = None
    if rank == 0 and not args.no_guiding and not args.small and not args.profile:
        guide = timed_section("guiding", guiding_bench)

    batch = None
    if rank == 0 and not args.no_batch and not args.small and not args.profile:
        batch = timed_section("batch", batch_bench)

    feats = None
    if rank == 0 and not args.no_features and not args.small and not args.profile:
        feats = timed_section("features", features_bench)

    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline and not args.profile:
        cpu = timed_section("cpu_baseline", lambda: cpu_baseline(desc, w, budget_s=4.0 if args.small else 15.0))

    if rank != 0:
        return
    peak, peak_kind = measured_peaks()
    trace_ms_frame = stage["trace_ms"] / args.steps - camera_ms
    rays_frame = bounces / args.steps - W * H * w["spp"]
    alg_bytes_ray = 32 + 16 + NODE_BYTES * nodes_per_ray + 48 * tris_per_ray
    alg_bytes_frame = alg_bytes_ray * rays_frame
    achieved = alg_bytes_frame / (trace_ms_frame / 1e3) / 1e9
    iters_frame = iterations / args.steps
    rays_launch = rays_frame / iters_frame
    tr = load_traffic()
    traffic = None
    limiter = None
    launch_ms = trace_ms_frame / iters_frame
    if tr and tr.get("kernel") == TRACE_KERNEL and tr.get("dram_bytes_per_ray"):
        traffic = round(tr["dram_bytes_per_ray"] * rays_launch)
        # what bounds the kernel: the DRAM fraction (ncu bytes over the live
        # launch time) is small; issue slots and SIMT lanes are the limit
        limiter = {"kind": "issue/divergence (node and triangle data served from L1/L2)",
                   "dram_gbs": round(traffic / (launch_ms / 1e3) / 1e9, 1),
                   "dram_frac": round(traffic / (launch_ms / 1e3) / 1e9 / peak, 4),
                   "simt_efficiency": round(tr["simt_lanes_active"] / 32.0, 4) if "simt_lanes_active" in tr else None,
                   "issue_active": tr.get("issue_active"),
                   "source": "dram_frac: ncu DRAM bytes per ray (profile-size capture) x rays per launch / live "
                             "launch time / measured HBM peak; simt_efficiency and issue_active: ncu counters of "
                             "the same capture"}
    value = units / secs / 1e6
    frame_ms = total_ms / args.steps
    line = {
        "metric": METRIC, "value": round(value, 3), "unit": UNIT, "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": round(frame_ms, 3), "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f32", "data": "synthetic (seeded procedural scene)",
        "config": config_dict(w, {"triangles": desc.n_triangles()}),
        "e2e": {"value": round(e_units / e_secs / 1e6, 3), "unit": UNIT,
                "h2d_bytes_per_step": 64 + 40, "d2h_bytes_per_step": W * H * 12,
                "note": "kz_render with a host film buffer: camera+config in, W*H*3 float out per frame"},
        "roofline": {"bound": "hbm", "kernel": TRACE_KERNEL, "achieved": round(achieved, 1), "peak": peak,
                     "unit": "GB/s", "frac": round(achieved / peak, 4), "traffic": traffic,
                     "alg_bytes_per_launch": round(alg_bytes_ray * rays_launch),
                     "launch_ms": round(launch_ms, 4), "limiter": limiter,
                     "peak_source": peak_kind + " (MEASURED_PEAKS.json hbm_gbs)" if peak_kind == "measured" else peak_kind,
                     "alg_bytes_per_ray": round(alg_bytes_ray, 1),
                     "node_fetches_per_ray": round(nodes_per_ray, 2), "tri_fetches_per_ray": round(tris_per_ray, 2),
                     "note": "rays after the camera's (camera rays are traced in bundles by a kernel of their own; "
                             "its time, from frames of depth 1, is taken off the trace stage); achieved/frac count "
                             "algorithmic bytes = 32 B ray + 16 B hit + 80 B per 8-wide node fetch + 48 B per "
                             "triangle fetch; node/triangle fetches are served mostly from L1/L2, so the kernel is "
                             "issue- and divergence-bound (see limiter), not HBM-bound"},
        "stages_ms_per_frame": {k: round(v / args.steps, 3) for k, v in stage.items()},
        "mrays_per_s": round((bounces + shadow) / (total_ms / 1e3) / 1e6, 2),
        "gpu_launches": launches,
        "clocks": clk,
        "cpu_baseline": cpu,
        "traversal": trav,
        "box": box,
        "guiding": guide,
        "batch": batch,
        "features": feats,
        "section_seconds": sections,
    }
    if img is not None:
        line["image_mean"] = float(np.asarray(img).mean())
    print(json.dumps(line))


# ---------------------------------------------------------------- reference arm
def run_reference(args):
    rank = int(os.environ.get("RANK", 0))
    if rank != 0:
        return
    from kazen_proto_gb300 import scenes
    from oracle import oracle as O
    w = workload(args)
    desc = scenes.terrain_scene(w["width"], w["height"], w["spp"], w["max_depth"], w["cells"], w["n_spheres"])
    sc = O.Scene.from_desc(desc)
    c = desc.camera
    cam = O.make_camera(c.eye, c.lookat, c.up, c.fov, c.flip)
    cores = os.cpu_count() or 1
    H = w["height"]
    per_step = 4  # rows per step, strided over the whole frame; the offset moves each step

    def step_rows(k):
        return strided_rows(H, per_step, offset=(37 * k) % H)
    for k in range(args.warmup):
        for a in step_rows(1000 + k):
            sc.render(cam, w["width"], H, w["spp"], w["max_depth"], seed=0, nthreads=cores, rows=(a, a + 1))
    secs, bounces = 0.0, 0
    for k in range(args.steps):
        t0 = time.perf_counter()
        for a in step_rows(k):
            _, st = sc.render(cam, w["width"], H, w["spp"], w["max_depth"], seed=0, nthreads=cores, rows=(a, a + 1))
            bounces += st["path_bounces"]
        secs += time.perf_counter() - t0
    v = bounces / secs / 1e6
    sample = ("%d rows per step strided over the whole %d-row frame (offset moving by 37 rows a step) x %d px x "
              "%d spp" % (per_step, H, w["width"], w["spp"]))
    line = {"impl": "reference", "metric": METRIC, "value": round(v, 4), "unit": UNIT, "n_gpus": 0,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(secs / args.steps * 1e3, 1),
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
            "data": "synthetic (seeded procedural scene)", "config": config_dict(w, {"triangles": desc.n_triangles()}),
            "cpu_baseline": {"value": round(v, 4), "unit": UNIT, "cores": cores, "kind": "port", "sample": sample,
                             "note": "the reference itself cannot be built here (Embree 4, OSL, OIIO, TBB, boost, "
                                     "pcg32 absent); this is the CPU restatement of its hot path"},
            "e2e": {"value": round(v, 4), "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line))


if __name__ == "__main__":
    a = parse()
    if a.profile_guide:
        profile_guide()
    elif a.profile_wgrad:
        profile_wgrad()
    elif a.impl == "reference":
        run_reference(a)
    else:
        run_ours(a)
