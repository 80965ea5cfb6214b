"""Benchmark of the B200 Gaussian-splat rasterizer (one JSON line on rank 0).

Workload: the "plain forward at working size" shape -- a 740,000-Gaussian SH-degree-3 scene
(seeded synthetic, 20x6x20 box) seen by 16 cameras on a radius-8 ring at 1280x720, f = 1100.
A step renders the 16 views once. Metric: Gaussians/s forward = 16 * N / step time.

    python bench.py [--steps K] [--warmup W] [--gpus N]          # this library
    python bench.py --impl reference [--steps K] [--warmup W]    # the reference CPU renderer

`value` is device-timed (CUDA events on the render stream, scene resident in HBM, images
written to device memory). `e2e` renders the same views through the public C ABI call
aniso_b200_render (the drop-in for GpuRenderer::render) into pinned host memory, so each view's
camera upload and the image's trip to the host (written across PCIe by the blend kernel itself,
since the buffer is page-locked) are inside the timed region. Under torchrun each rank renders its own
replica's 16 views (weak scaling, no collective); time is the max over ranks.

Three more workloads of the same metric family ride along at N = 1 (skip with --no-extra):
  "batched":  one 1M-Gaussian scene, 64 Fibonacci-sphere views of mixed resolution, rendered by one
              autotuned, graph-replayed batch versus 64 plain per-view launches (views/s);
  "fwd_bwd":  the 2.2M-Gaussian scene at 1280x720, forward + hand-written adjoint through the
              torch.autograd.Function against an L2 loss (ms/view);
  "train_batch": 8 scenes (11.3M Gaussians), 32 views, one batched forward + adjoint versus the
              views one by one (ms/view).
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

WORKLOAD = "740k-Gaussian SH3 synthetic scene, 16 ring views 1280x720 (forward)"
METRIC = "Gaussians/s fwd"
UNIT = "Gaussians/s"
N_GAUSS = 740_000
# The reference's published GPU forward on its 0.74M-Gaussian *train* scene at 1280 wide:
# 2.3 ms/frame on an RTX 5090 (README.md:28) = 741,883 / 2.3 ms.
PUBLISHED_GAUSSIANS_PER_S = 741_883 / 2.3e-3
# One blend launch on ring view 0, from an ncu capture (profiles/kernels_of_the_cases.md): DRAM bytes and
# warp instructions (smsp__inst_executed.sum).
BLEND_TRAFFIC_BYTES = 34_940_000
BLEND_WARP_INSTRUCTIONS = 79_557_323


def measured_peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            p = json.load(f)
        return float(p["hbm_gbs"]), "measured"
    except Exception:
        return 6650.0, "fallback"


class ClockSampler:
    """nvidia-smi clocks and throttle reasons, sampled every 100 ms while running."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index: int):
        self.rows = []
        self.gpu = gpu_index
        self.proc = None
        self.t0 = self.t1 = None

    def start(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "--query-gpu=" + self.FIELDS, "--format=csv,noheader,nounits",
                                          "-lms", "100", "-i", str(self.gpu)], stdout=subprocess.PIPE,
                                         stderr=subprocess.DEVNULL, text=True)
        except Exception:
            self.proc = None
            return
        self.thread = threading.Thread(target=self._read, daemon=True)
        self.thread.start()
        deadline = time.time() + 3
        while not self.rows and time.time() < deadline:
            time.sleep(0.01)

    def _read(self):
        for line in self.proc.stdout:
            self.rows.append((time.time(), [x.strip() for x in line.split(",")]))

    def mark_begin(self):
        self.t0 = time.time()

    def mark_end(self):
        self.t1 = time.time()

    def stop(self):
        if self.proc:
            time.sleep(0.25)
            self.proc.terminate()
            self.proc.wait(timeout=5)

    def summary(self):
        if not self.rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        t0, t1 = self.t0 or 0, self.t1 or time.time()
        inside = [r for t, r in self.rows if t0 - 0.2 <= t <= t1 + 0.2] or [self.rows[-1][1]]
        sm = [float(r[1]) for r in inside if r[1].replace(".", "").isdigit()]
        mx = [float(r[2]) for r in inside if r[2].replace(".", "").isdigit()]
        names = ["active", "hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = set()
        for r in inside:
            for k, nm in enumerate(names[1:], start=5):
                if len(r) > k and r[k].lower().startswith("active"):
                    reasons.add(nm)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": sorted(reasons), "samples": len(inside)}


def load_workload():
    from aniso_b200 import scenes

    scs, cams = scenes.config(2)
    gauss, sh = scenes.activate(scs[0])
    return gauss, sh, cams[0]


def reference_arm(args, rank):
    """The reference's own CPU renderer (render.cpp), all host threads, one view per step."""
    if rank != 0:
        return
    import oracle

    gauss, sh, cams = load_workload()
    if oracle.ReferenceCPU.available():
        # The scene is built once, as the reference CLI does; each timed step is aniso::render.
        scene, kind = oracle.ReferenceCPU().scene(gauss, sh, 3), "reference"
        render = scene.render
    else:
        port, kind = oracle.Restatement(), "port"
        render = lambda cam: port.render(gauss, sh, 3, cam)
    for k in range(args.warmup):
        render(cams[k % len(cams)])
    t = time.perf_counter()
    for k in range(args.steps):
        render(cams[k % len(cams)])
    dt = time.perf_counter() - t
    value = args.steps * N_GAUSS / dt
    cores = os.cpu_count() if kind == "reference" else 1
    line = {"metric": METRIC, "value": value, "unit": UNIT, "impl": "reference", "n_gpus": args.gpus,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1000 * dt / args.steps,
            "ms_per_frame": 1000 * dt / args.steps, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "fp32", "data": "synthetic (seeded generator, 740k SH3)",
            "config": {"workload": WORKLOAD + "; one ring view per step", "gaussians": N_GAUSS},
            "cpu_baseline": {"value": value, "unit": UNIT, "cores": cores, "kind": kind,
                             "sample": "%d views of the 16 (one per step), reference render.cpp with "
                                       "std::thread::hardware_concurrency() threads; the scene built once "
                                       "outside the timed loop" % args.steps},
            "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    try:
        line["reference_gpu"] = reference_gpu_leg(gauss, sh, cams)
    except Exception as e:  # no GPU in this arm's environment: the CPU figure stands alone
        line["reference_gpu"] = {"unavailable": str(e).splitlines()[0][:200]}
    # This repository's shared libraries mapped by this process: only the reference builds under
    # oracle/ belong here, never the library under test.
    line["repo_libraries_loaded"] = repo_libraries_loaded()
    print(json.dumps(line), flush=True)


def repo_libraries_loaded():
    """Shared objects under this repository that the current process has mapped (Linux)."""
    try:
        with open("/proc/self/maps") as f:
            paths = {l.split()[-1] for l in f if l.rstrip().endswith(".so") or ".so." in l}
    except OSError:
        return None
    return sorted(os.path.relpath(p, ROOT) for p in paths if p.startswith(ROOT + os.sep))


def cpu_baseline_leg(gauss, sh, cams, images):
    """Reference CPU renderer on a bounded sample (2 views) and the image agreement there."""
    import oracle

    if oracle.ReferenceCPU.available():
        scene, kind, cores = oracle.ReferenceCPU().scene(gauss, sh, 3), "reference", os.cpu_count()
        render = scene.render
    else:
        port, kind, cores = oracle.Restatement(), "port", 1
        render = lambda cam: port.render(gauss, sh, 3, cam)
    views = [0, 8]
    render(cams[views[0]])  # warm-up
    worst_abs, worst_psnr = 0, float("inf")
    t = time.perf_counter()
    refs = [render(cams[v])[0] for v in views]
    dt = time.perf_counter() - t
    for v, ref in zip(views, refs):
        d = np.abs(images[v].astype(np.int32) - ref.astype(np.int32))
        worst_abs = max(worst_abs, int(d.max()))
        worst_psnr = min(worst_psnr, oracle.psnr(images[v], ref))
    base = {"value": len(views) * N_GAUSS / dt, "unit": UNIT, "cores": cores, "kind": kind,
            "sample": "ring views 0 and 8 of the 16, 1 warm-up, %s" % ("reference render.cpp -O3 (scene built "
                                                                     "once), hardware_concurrency threads"
                                                                     if kind == "reference" else "C restatement, 1 thread")}
    return base, {"max_abs_255": worst_abs, "psnr_db": worst_psnr, "views": views, "vs": "CPU renderer"}


def stage_rooflines(prof, frames, counts, pairs, W, H, peak, peak_kind):
    """HBM fractions of the projection and sort stages on their algorithmic bytes per view:
    preprocess N*44 (position, scale, rotation, opacity) + V*192 (SH3 of visible entries) + V*40
    (record and depth) + N*4 (depth keys); sort P*12 (pairs written) + 2*P*12 (one read and one
    write of every (key, value) pair, the least any pair sort moves) + T*8 (ranges)."""
    Vis = sum(c["visible"] for c in counts) / len(counts)
    T = ((W + 15) // 16) * ((H + 15) // 16)
    out = {}
    for name, key, nbytes in (("preprocess", "project_ms", N_GAUSS * 48 + Vis * 232),
                              ("sort", "sort_ms", pairs * 36 + T * 8)):
        ms = prof[key] / frames
        gbs = nbytes / (ms / 1000.0) / 1e9
        out[name] = {"bytes": nbytes, "ms": ms, "achieved": gbs, "peak": peak, "unit": "GB/s", "frac": gbs / peak,
                     "peak_source": peak_kind}
    out["visible_per_view"] = Vis
    return out


def measured_compute_peaks():
    """ex2 and FP32 FMA rates of this GPU from the library's throughput probe (ops/s)."""
    import ctypes

    lib = ctypes.CDLL(os.path.join(ROOT, "aniso_b200", "libaniso_b200_peaks.so"))
    ex2, fma = ctypes.c_double(), ctypes.c_double()
    if lib.ab2_measure_peaks(ctypes.byref(ex2), ctypes.byref(fma)) != 0:
        return None, None
    return ex2.value, fma.value


def batched_leg(torch, steps: int):
    """Workload 4: 1M Gaussians, 64 sphere views of mixed resolution; batch vs per-view launches."""
    from aniso_b200 import BatchRenderer, GpuRenderer, scenes
    from aniso_b200._lib import AnisoError
    from aniso_b200.autotune import time_batch, tune

    raws, camsets = scenes.config(4)
    cams = camsets[0]
    r = GpuRenderer.from_raw(raws[0])
    outs = [torch.empty((c.height, c.width, 3), dtype=torch.uint8, device="cuda") for c in cams]
    ptrs = [o.data_ptr() for o in outs]
    stream = torch.cuda.Stream()

    def per_view():
        for c, p in zip(cams, ptrs):
            r.render_device(c, p, stream.cuda_stream)

    for _ in range(3):
        for _attempt in range(3):
            per_view()
            try:
                r.sync()
                break
            except AnisoError as e:
                if "pair capacity" not in str(e):
                    raise
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for _ in range(steps):
        per_view()
    e1.record(stream)
    r.sync()
    ms_pv = e0.elapsed_time(e1) / steps
    ref = [o.cpu().numpy() for o in outs]
    candidates = []
    best = tune([r], [0] * len(cams), cams, cache_path=None, report=candidates)
    b = BatchRenderer([r], [0] * len(cams), best)
    ms_b = time_batch(b, cams, ptrs, stream, warmup=3, iters=steps)
    same = all(np.array_equal(o.cpu().numpy(), x) for o, x in zip(outs, ref))
    st = b.sync()
    V = len(cams)
    return {"workload": "1M-Gaussian SH3 scene, 64 Fibonacci-sphere views (radius 10), resolutions drawn from "
                        "320x180/640x360/1280x720/1920x1080, f = 0.9 W",
            "views_per_s": V * 1000.0 / ms_b, "views_per_s_per_view_launches": V * 1000.0 / ms_pv,
            "speedup_vs_per_view": ms_pv / ms_b, "ms_per_batch": ms_b, "ms_per_64_plain_launches": ms_pv,
            "gaussians_per_s": V * raws[0].n / (ms_b / 1000.0),
            "tuned": {"tile": "%dx%d" % best.tile, "blend_batch": best.blend_batch, "radix_bits": best.radix_bits,
                      "cuda_graph": True},
            "candidates_ms": {"%dx%d/%d/%db" % (c["tile"][0], c["tile"][1], c["blend_batch"], c["radix_bits"]):
                              round(c["ms"], 3) for c in candidates},
            "pairs": st["tile_pairs"], "images_equal_per_view": same}


def fwd_bwd_leg(torch, steps: int):
    """Workload 3: 2.2M Gaussians, 1280x720, L2 loss against the perturbed-scene target."""
    from aniso_b200 import scenes
    from aniso_b200.autograd import rasterize

    raws, camsets = scenes.config(3)
    raw, cam = raws[0], camsets[0][0]

    def params(rw, grad):
        n = rw.n
        sh = np.concatenate([rw.f_dc.reshape(n, 1, 3), rw.f_rest.reshape(n, 3, 15).transpose(0, 2, 1)], 1)
        arrs = [rw.xyz, rw.scale, rw.rot, rw.opacity, np.ascontiguousarray(sh)]
        return [torch.tensor(a, dtype=torch.float32, device="cuda", requires_grad=grad) for a in arrs]

    with torch.no_grad():
        target = rasterize(*params(scenes.perturbed_target(raw), False), cam)
    ps = params(raw, True)
    stream = torch.cuda.current_stream()

    def step():
        for p in ps:
            p.grad = None
        img = rasterize(*ps, cam)
        ((img - target) ** 2).sum().backward()

    for _ in range(3):
        step()
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for _ in range(steps):
        step()
    e1.record(stream)
    torch.cuda.synchronize()
    ms = e0.elapsed_time(e1) / steps
    with torch.no_grad():
        for _ in range(3):
            rasterize(*ps, cam)
        e0.record(stream)
        for _ in range(steps):
            rasterize(*ps, cam)
        e1.record(stream)
        torch.cuda.synchronize()
    ms_f = e0.elapsed_time(e1) / steps
    finite = all(bool(torch.isfinite(p.grad).all()) for p in ps)
    # What the checker needs (outside any timed region): the last step's gradients and the image
    # and target they came from.
    with torch.no_grad():
        image = rasterize(*ps, cam)
    check = {"raw": raw, "cam": cam, "grads": [p.grad.cpu().numpy().astype(np.float64) for p in ps],
             "image": image.cpu().numpy().astype(np.float64), "target": target.cpu().numpy()}
    del ps, target, image
    torch.cuda.empty_cache()

    # The plain forward (RGB8, the GpuRenderer::render path) of the same 2.2M scene and view.
    from aniso_b200 import GpuRenderer

    r = GpuRenderer.from_raw(raw)
    first = r.render(cam)  # sizes the pair buffers
    out = torch.empty(cam.height, cam.width, 3, dtype=torch.uint8, device="cuda")
    plain_stream = torch.cuda.Stream()
    for _ in range(3):
        r.render_device(cam, out.data_ptr(), plain_stream.cuda_stream)
    r.sync()
    e0.record(plain_stream)
    for _ in range(steps):
        r.render_device(cam, out.data_ptr(), plain_stream.cuda_stream)
    e1.record(plain_stream)
    r.sync()
    ms_plain = e0.elapsed_time(e1) / steps
    pinned = torch.empty(cam.height, cam.width, 3, dtype=torch.uint8).pin_memory().numpy()
    for _ in range(3):
        r.render(cam, out=pinned)
    t = time.perf_counter()
    for _ in range(steps):
        r.render(cam, out=pinned)
    ms_plain_e2e = 1000 * (time.perf_counter() - t) / steps
    check["rgb8"] = first
    check["rgb8_same_as_device"] = bool(np.array_equal(out.cpu().numpy(), first))
    del r
    return {"workload": "2.2M-Gaussian SH3 scene (30x8x30 box), 1280x720, L2 loss vs the perturbed-scene target, "
                        "grads of all 59 raw parameters through torch.autograd.Function",
            "ms_per_view_fwd_bwd": ms, "ms_per_view_fwd_train": ms_f, "gaussians": raw.n,
            "grads_finite": finite, "target_ms": 3.0,
            "plain_forward": {"ms_per_frame": ms_plain, "ms_per_frame_e2e": ms_plain_e2e,
                              "gaussians_per_s": raw.n / (ms_plain / 1000.0), "target_ms": 1.0,
                              "path": "aniso_b200_render_device (device-timed); e2e: aniso_b200_render into "
                                      "pinned host memory"}}, check


def accuracy_checks(check):
    """The checker, on the CPU after the timed legs (the FP64 oracle and the reference CPU
    renderer): the 2.2M plain forward against render.cpp, and the 2.2M gradients against FP64
    central differences on 256 sampled parameters and against the FP64 adjoint of every gradient."""
    import oracle
    from oracle import gradcheck

    out = {}
    raw, cam = check["raw"], check["cam"]
    gauss, sh = oracle.Restatement().activate(raw)
    if oracle.ReferenceCPU.available():
        cpu = oracle.ReferenceCPU().scene(gauss, sh, 3).render(cam)[0]
        vs = "reference render.cpp"
    else:
        cpu = oracle.Restatement().render(gauss, sh, 3, cam)[0]
        vs = "C restatement of render.cpp"
    d = np.abs(check["rgb8"].astype(np.int32) - cpu.astype(np.int32))
    out["plain_forward_accuracy"] = {"max_abs_255": int(d.max()), "psnr_db": oracle.psnr(check["rgb8"], cpu),
                                     "vs": vs, "device_equals_host_render": check["rgb8_same_as_device"]}
    params = [p.astype(np.float64) for p in gradcheck.raw_param_arrays(raw)]
    big = oracle.Restatement().big_frame(params, cam)
    grads = check["grads"]
    live = np.nonzero(np.abs(grads[0]).sum(1) > 0)[0]
    fd = gradcheck.fd_check(big, check["target"], grads, live, samples=256, step=1e-4)
    adj = gradcheck.window_check(big, 0, 0, 2 * (check["image"] - check["target"]), grads)
    ref_img = big.image(0, 0, cam.width, cam.height)
    out["grad_rel_err"] = {
        "vs_fp64_fd": {k: fd[k] for k in gradcheck.GROUPS},
        "fd_totals": fd["_totals"],
        "vs_fp64_adjoint": adj,
        "forward_max_abs_vs_fp64": float(np.abs(check["image"] - ref_img).max()),
        "bar": 1e-3,
        "rel": "||g_gpu - g_ref||_2 / ||g_ref||_2 per group; FD draws whose +h and -h renders take "
               "different branches (alpha cut, clamp, termination, order, rectangle) are redrawn"}
    big.close()
    return out


def reference_gpu_leg(gauss, sh, cams, rounds: int = 2):
    """Reference arm only: the reference's own GpuRenderer (gpu_render.cu with CUB, built for
    sm_100a with --use_fast_math as its CMake ships it) on the same 16 views, the GPU bar. Its
    RenderStats events cover preprocess + scan + the host read of the pair count, sort, blend; the
    wall clock adds its device-to-host image copy."""
    import oracle

    if not oracle.ReferenceGPU.available(fast_math=True):
        return {"unavailable": "oracle/_ref/libaniso_ref_gpu_fast.so not built (no reference sources)"}
    ref = oracle.ReferenceGPU(fast_math=True)
    h = ref.renderer(gauss, sh, 3)
    try:
        ref.render(h, cams[0])  # warm-up: grows its buffers
        ev, frames = 0.0, 0
        t = time.perf_counter()
        for _ in range(rounds):
            for cam in cams:
                _, st = ref.render(h, cam)
                ev += st["project_ms"] + st["sort_ms"] + st["blend_ms"]
                frames += 1
        wall = (time.perf_counter() - t) / frames
    finally:
        ref.destroy(h)
    return {"impl": "reference aniso::GpuRenderer (src/gpu_render.cu, CUB scan + radix sort), sm_100a, fast-math",
            "ms_per_frame_events": ev / frames, "ms_per_frame_wall": 1000 * wall,
            "gaussians_per_s_events": N_GAUSS / (ev / frames / 1000.0), "frames": frames}


def train_batch_leg(torch, steps: int):
    """Workload 5: 8 scenes of uneven size (0.2M..3.0M), 4 views each (960x540 / 1280x720), random
    N(0, 1) upstream gradients: one batched forward + adjoint for all 32 views versus the same
    views one by one through the single-view autograd Function."""
    from aniso_b200 import scenes
    from aniso_b200.autograd import rasterize, rasterize_batch

    raws, camsets = scenes.config(5)

    def params(rw):
        n = rw.n
        sh = np.concatenate([rw.f_dc.reshape(n, 1, 3), rw.f_rest.reshape(n, 3, 15).transpose(0, 2, 1)], 1)
        arrs = [rw.xyz, rw.scale, rw.rot, rw.opacity, np.ascontiguousarray(sh)]
        return [torch.tensor(a, dtype=torch.float32, device="cuda", requires_grad=True) for a in arrs]

    ps = [params(rw) for rw in raws]
    cams = [c for cs in camsets for c in cs]
    view_scene = [s for s, cs in enumerate(camsets) for _ in cs]
    rng = np.random.default_rng(4)
    ups = [torch.tensor(rng.standard_normal((c.height, c.width, 3)), dtype=torch.float32, device="cuda")
           for c in cams]

    def zero():
        for group in ps:
            for p in group:
                p.grad = None

    from aniso_b200.autotune import tune_train

    candidates = []
    best = tune_train(ps, cams, view_scene, cache_path=None, report=candidates, iters=2)

    def batched():
        zero()
        imgs = rasterize_batch(ps, cams, view_scene, options=best)
        torch.autograd.backward(imgs, ups)

    def per_view():
        zero()
        for k, (c, s) in enumerate(zip(cams, view_scene)):
            torch.autograd.backward([rasterize(*ps[s], c)], [ups[k]])

    out = {}
    for name, fn in (("batched", batched), ("per_view", per_view)):
        for _ in range(2):
            fn()
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        if name == "batched":  # lets a profiler started with collection off take these steps alone
            torch.cuda.profiler.start()
        e0.record()
        for _ in range(steps):
            fn()
        e1.record()
        if name == "batched":
            torch.cuda.profiler.stop()
        torch.cuda.synchronize()
        out[name] = e0.elapsed_time(e1) / steps
    grads_b = [p.grad.clone() for group in ps for p in group]  # from the last per-view run
    batched()
    flat = [p for group in ps for p in group]
    same = all(torch.equal(a, p.grad) for a, p in zip(grads_b, flat))
    from aniso_b200.autotune import grad_rel_diff

    rel = max(grad_rel_diff(p.grad, a) for a, p in zip(grads_b, flat))
    V = len(cams)
    return {"workload": "8 scenes of 0.2/0.4/0.7/1.0/1.5/2.0/2.5/3.0M Gaussians (SH3), 4 ring views each "
                        "(960x540 and 1280x720 alternating), upstream dL/dimage ~ N(0,1), fp32",
            "ms_per_view_batched": out["batched"] / V, "ms_per_view_per_view": out["per_view"] / V,
            "speedup": out["per_view"] / out["batched"], "views": V,
            "gaussians": sum(rw.n for rw in raws),
            "tuned": {"tile": "%dx%d" % best.tile, "blend_batch": best.blend_batch, "radix_bits": best.radix_bits,
                      "cuda_graph": bool(best.use_graph)},
            "candidates_ms_per_step": {"%dx%d/%d/%db" % (c["tile"][0], c["tile"][1], c["blend_batch"],
                                                         c["radix_bits"]): round(c["ms"], 3) for c in candidates},
            "grads_equal_per_view_sum": same, "grads_rel_diff_per_view_sum": rel,
            "note": "at 16x16 tiles the batched gradients equal the per-view gradients summed in view order "
                    "bit for bit; another tile grid sums the same per-pixel terms in other groups "
                    "(grads_rel_diff_per_view_sum: the largest norm-wise relative difference of a tensor); "
                    "the per-view adjoint is checked against FP64 in tests/test_gradients.py and "
                    "tests/test_gradients_config3.py"}


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=50)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="b200", choices=["b200", "reference"])
    ap.add_argument("--no-extra", action="store_true", help="skip the batched and fwd+bwd workloads")
    ap.add_argument("--only", choices=["batched", "fwd_bwd", "train_batch"], default=None,
                    help="run one extra workload alone and print its JSON object (for profiling)")
    args = ap.parse_args()
    args.warmup = max(args.warmup, 3)
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))

    if args.impl == "reference":
        reference_arm(args, rank)
        return

    import torch

    torch.cuda.set_device(local)
    if args.only:
        if rank == 0:
            leg = {"batched": batched_leg, "fwd_bwd": lambda t, s: fwd_bwd_leg(t, s)[0],
                   "train_batch": train_batch_leg}[args.only]
            print(json.dumps({"leg": args.only, **leg(torch, args.steps)}), flush=True)
        return
    dist = None
    if world > 1:
        import datetime

        import torch.distributed as dist

        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120), device_id=torch.device("cuda", local))

    from aniso_b200 import GpuRenderer

    gauss, sh, cams = load_workload()
    r = GpuRenderer(gauss, sh, 3)
    V = len(cams)
    H, W = cams[0].height, cams[0].width

    # Warm-up through the host API: sizes the pair buffers for every view, gives per-view counts.
    images, counts = [], []
    for cam in cams:
        st = {}
        images.append(r.render(cam, st).copy())
        counts.append(st)
    pairs_per_step = sum(c["tile_pairs"] for c in counts)

    out = torch.empty(V, H, W, 3, dtype=torch.uint8, device="cuda")
    stream = torch.cuda.Stream()

    def step():
        for v, cam in enumerate(cams):
            r.render_device(cam, out[v].data_ptr(), stream.cuda_stream)

    for _ in range(args.warmup):
        step()
    r.sync()
    # Kernel launches of one step, as the library counts them (the same frames as the timed loop).
    launches_per_step = 0
    for v, cam in enumerate(cams):
        r.render_device(cam, out[v].data_ptr(), stream.cuda_stream)
        launches_per_step += r.frame_kernels()
    r.sync()

    sampler = ClockSampler(local)
    sampler.start()
    if dist:
        dist.barrier()
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    sampler.mark_begin()
    e0.record(stream)
    for _ in range(args.steps):
        step()
    e1.record(stream)
    torch.cuda.synchronize()
    sampler.mark_end()
    r.sync()  # raises if any frame overflowed or a device wait gave up
    # Stage split (project / sort / blend) from events around each stage, in a separate loop of the
    # same frames: the events cut the frame's kernel chain, so the timed loop above runs without them.
    r.profile(True)
    for _ in range(args.steps):
        step()
    torch.cuda.synchronize()
    r.profile(False)
    prof = r.profile_read()
    r.sync()
    if dist:
        dist.barrier()
    sampler.stop()
    ms = e0.elapsed_time(e1)
    if dist:
        t = torch.tensor([ms], device="cuda", dtype=torch.float64)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        ms = float(t.item())
    ms_step = ms / args.steps
    value = world * V * N_GAUSS / (ms_step / 1000.0)

    # Images written by the timed loop agree with the host-API renders.
    same = bool(np.array_equal(out.cpu().numpy(), np.stack(images)))

    # End to end through the public C ABI into pinned host memory.
    pinned = torch.empty(V, H, W, 3, dtype=torch.uint8).pin_memory()
    host = pinned.numpy()
    for _ in range(args.warmup):
        for v, cam in enumerate(cams):
            r.render(cam, out=host[v])
    if dist:
        dist.barrier()
    t = time.perf_counter()
    for _ in range(args.steps):
        for v, cam in enumerate(cams):
            r.render(cam, out=host[v])
    e2e_s = (time.perf_counter() - t) / args.steps
    if dist:
        tt = torch.tensor([e2e_s], device="cuda", dtype=torch.float64)
        dist.all_reduce(tt, op=dist.ReduceOp.MAX)
        e2e_s = float(tt.item())
    e2e_value = world * V * N_GAUSS / e2e_s

    line = None
    if rank == 0:
        frames = max(prof["frames"], 1)
        blend_ms = prof["blend_ms"] / frames
        peak, peak_kind = measured_peaks()
        # Algorithmic bytes of one blend launch (per view): P*4 index + P*36 splat record + W*H*3 out.
        blend_bytes = pairs_per_step / V * 40 + W * H * 3
        achieved = blend_bytes / (blend_ms / 1000.0) / 1e9
        # The CPU baseline and the extra workloads run at N = 1 only: under torchrun the other ranks
        # wait at the closing barrier, whose timeout minutes of rank-0-only work would exceed.
        base, acc = cpu_baseline_leg(gauss, sh, cams, images) if world == 1 else (None, None)
        ex2_peak, fma_peak = measured_compute_peaks()
        # The blend is bound by instruction issue: its warp instructions against four a cycle and SM at the
        # clock seen under load.
        clocks = sampler.summary()
        sms = torch.cuda.get_device_properties(torch.cuda.current_device()).multi_processor_count
        issue_peak = 4.0 * sms * 1e6 * (clocks.get("sm_mhz") or 0.0)
        issued_per_s = BLEND_WARP_INSTRUCTIONS / (blend_ms / 1000.0)
        extra = {}
        if not args.no_extra and world == 1:
            extra["batched"] = batched_leg(torch, max(3, min(args.steps, 10)))
            extra["fwd_bwd"], check = fwd_bwd_leg(torch, max(3, min(args.steps, 10)))
            extra["train_batch"] = train_batch_leg(torch, 2)
            extra["fwd_bwd"].update(accuracy_checks(check))
        line = {
            "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ms_step, "ms_per_frame": ms_step / V,
            "higher_is_better": True, "scaling": "weak",
            "vs_baseline": value / world / PUBLISHED_GAUSSIANS_PER_S,
            "dtype": "fp32", "data": "synthetic: seeded 3DGS generator (uniform box, log-scale N(-4,0.5), "
                                     "logit opacity N(0,1.5), SH3), no dataset",
            "config": {"workload": WORKLOAD, "gaussians": N_GAUSS, "sh_degree": 3, "views_per_step": V,
                       "resolution": "%dx%d" % (W, H), "tile": "16x16",
                       "l2": "inputs larger than L2: scene %.0f MB (> 126 MB) re-read from HBM every view"
                             % (N_GAUSS * 240 / 1e6),
                       "parallelism": "replicas (views independent; no collective)" if world > 1 else "1 GPU",
                       "vs_baseline_source": "reference README.md:28: 2.3 ms/frame, 0.74M train scene, RTX 5090"},
            "stages_ms_per_frame": {k: prof[k] / frames for k in ("project_ms", "sort_ms", "blend_ms")},
            "pairs_per_frame": pairs_per_step / V,
            # The dominant kernel's roofline follows its bound, which is instruction issue (no stage is a
            # dense contraction, the blend reads far less than HBM could deliver, and its exponentials take a
            # fifth of the measured ex2 rate); its HBM figure rides along.
            "roofline": {"kernel": "blend", "bound": "issue", "achieved": issued_per_s, "peak": issue_peak,
                         "unit": "warp instructions/s", "frac": (issued_per_s / issue_peak) if issue_peak else None,
                         "peak_source": "4 per cycle and SM at the SM clock sampled in the timed region",
                         "traffic": BLEND_TRAFFIC_BYTES,
                         "work": "warp instructions of the blend on ring view 0, counted by ncu",
                         "ex2_peak": ex2_peak, "fp32_fma_peak": fma_peak,
                         "hbm": {"achieved": achieved, "peak": peak, "unit": "GB/s", "frac": achieved / peak,
                                 "peak_source": peak_kind, "bytes": "P*40 + W*H*3 per launch"}},
            "stage_rooflines": stage_rooflines(prof, frames, counts, pairs_per_step / V, W, H, peak, peak_kind),
            "cpu_baseline": base,
            "accuracy": acc,
            "e2e": {"value": e2e_value, "unit": UNIT, "h2d_bytes_per_step": V * 136,
                    "d2h_bytes_per_step": V * (H * W * 3 + 64),
                    "path": "aniso_b200_render (GpuRenderer::render drop-in), pinned host output written by the blend kernel"},
            "gpu_launches": launches_per_step * args.steps,
            "kernels_per_frame": launches_per_step / V,
            "timed_images_match_host_api": same,
            "clocks": clocks,
        }
        line.update(extra)
        print(json.dumps(line), flush=True)
    if dist:
        dist.barrier()
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
