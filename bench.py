"""Benchmark of the rasterizer hot path on the 1080p / 1M-triangle scene.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl axr|reference]

One step = one frame of the plain single-view workload: both 2048^2 shadow
cascades (clear + ortho setup + depth raster) and the 1920x1080 main view
(clear + drawAll: setup, small/large raster, shading with trilinear mips,
alpha test and the double-cascade lookup) over 1,044,288 triangles in 5
materials.  Synthetic seeded scene (no dataset).

Prints one JSON line (rank 0).  `value` = frames/s with the scene resident in
HBM, timed with CUDA events on the library's stream (max over ranks); `e2e`
= frames/s through the public API with the camera pose uploaded and the
frame (3 x u16 colour planes + f32 depth) read back into pinned host memory
every step.  Multi-GPU runs are replicas (one scene per GPU, weak scaling,
no data-path collective).  `--impl reference` times the reference's own
OpenCL kernels compiled for the host CPU (oracle/_ref) on the same scene.
"""
from __future__ import annotations

import argparse
import json
import math
import os
import subprocess
import sys
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "frames/s & Mtri/s at 1080p/1M tris; p50/p99 latency, batched vs plain"
W, H = 1920, 1080
PEAKS_FILE = os.path.join(ROOT, "MEASURED_PEAKS.json")
FALLBACK_HBM_GBS = 6650.0

# From one ncu capture of this frame's kernels: DRAM traffic per launch
# (dram__bytes.sum; the two cascades averaged for the shadow kernels, as the
# per-kernel event times are), and issued warp instructions of a frame's
# launches (smsp__inst_issued.sum; the two cascades together).
# A kernel whose code changed since its capture has no entry.  NCU_CAPTURE
# names the committed summary of that capture, reported in the JSON line.
NCU_CAPTURE = "profiles/ncu_kernels_1080p_1m.md"
NCU_TRAFFIC = {
    "k_raster_small": 32813824,
    "k_raster_small_alpha": 13466624,
    "k_shadow_raster": (46949632 + 50689024) // 2,
    "k_shadow_raster_alpha": (10291200 + 4465152) // 2,
    "k_shade": 30319872,
    "k_raster_tiled": 10353408,
    "k_raster_tiled_alpha": 8158464,
    "k_shadow_setup": (37617920 + 37619712) // 2,
    "k_setup": 54958336,
}
NCU_ISSUED = {
    "k_raster_small": 83122508,
    "k_raster_small_alpha": 69508703,
    "k_shadow_raster": 144633043 + 83271446,
    "k_shadow_raster_alpha": 34890508 + 12303716,
    "k_shade": 77281168,
    "k_raster_tiled": 20897991,
    "k_raster_tiled_alpha": 29877438,
    "k_shadow_setup": 14444480 + 14714699,
    "k_setup": 14435226,
}
ISSUE_PER_SM_PER_CLK = 4     # warp instructions: one per scheduler (4 per SM) per cycle


def progress(msg):
    """Stage marker on stderr (the JSON line alone goes to stdout)."""
    print(f"[bench {time.strftime('%H:%M:%S')}] {msg}", file=sys.stderr, flush=True)


def peaks():
    try:
        with open(PEAKS_FILE) as f:
            p = json.load(f)
        return float(p["hbm_gbs"]), "measured"
    except Exception:
        return FALLBACK_HBM_GBS, "fallback"


class Clocks:
    """Samples SM clocks and throttle reasons with nvidia-smi while running."""
    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,clocks_event_reasons.hw_slowdown,"
         "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
         "clocks_event_reasons.sw_power_cap")

    def __init__(self, index):
        self.index = index
        self.proc = None
        self.path = os.path.join("/tmp", f"axr_clocks_{os.getpid()}.csv")

    def start(self):
        try:
            self.f = open(self.path, "w")
            self.proc = subprocess.Popen(["nvidia-smi", f"--id={self.index}", f"--query-gpu={self.Q}",
                                          "--format=csv,noheader,nounits", "-lms", "50"],
                                         stdout=self.f, stderr=subprocess.DEVNULL)
        except Exception:
            self.proc = None

    def stop(self):
        if self.proc is None:
            return None
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        self.f.close()
        mhz, mx, reasons = [], 0.0, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in open(self.path):
            p = [x.strip() for x in line.split(",")]
            if len(p) < 9:
                continue
            try:
                mhz.append(float(p[1]))
                mx = max(mx, float(p[2]))
            except ValueError:
                continue
            for n, v in zip(names, p[5:9]):
                if v.lower().startswith("active"):
                    reasons.add(n)
        if not mhz:
            return None
        return {"sm_mhz": float(np.median(mhz)), "sm_max_mhz": mx, "reasons": sorted(reasons), "samples": len(mhz)}


# ------------------------------------------------------------------ roofline bookkeeping

def algorithmic_bytes(scene, q, shadow_q, visible_tris):
    """Lower-bound bytes each kernel must move per launch: the geometry it has
    to read once and the framebuffer / map bytes it has to write once.  `q`
    is the last drawAll's queues by kind (CLDraw.lastQueues), `shadow_q`
    each map's last pass (CLDraw.shadowStats); per-map figures are averaged
    over the maps, as the per-kernel times are."""
    T = scene.ntris
    cull_T = sum(g.ntris for g in scene.groups if g.flags & 8)
    npx = W * H
    nm = max(1, len(scene.shadows))
    smap = sum(sc.dim * sc.dim for sc in scene.shadows) / nm
    cast = sum(s["casters"] for s in shadow_q) / nm
    cast_a = sum(s["casters_alpha"] for s in shadow_q) / nm
    units = sum(s["units"] for s in shadow_q) / nm
    return {
        # xyz of every triangle (+ normals of culled groups), 4 B per list entry
        "k_setup": 36 * T + 36 * cull_T + 4 * (q["small"] + q["small_alpha"] + q["large"]),
        # xyz (+ uv of alpha-tested ones) of every small triangle; the
        # visibility word of every pixel updated once by the opaque pass
        "k_raster_small": 36 * q["small"] + 8 * npx,
        "k_raster_small_alpha": 60 * q["small_alpha"],
        # xyz of every large triangle and its (triangle, tile) units
        "k_coarse": 36 * q["large"] + 8 * (q["units"] + q["units_alpha"]),
        "k_raster_tiled": 36 * q["large"] + 8 * q["units"],
        "k_raster_tiled_alpha": 8 * q["units_alpha"],
        # visibility word read, colour + depth written, attributes of the visible triangles read once
        "k_shade": 8 * npx + 10 * npx + 132 * visible_tris,
        "k_init_keys": 4 * npx + 8 * npx,
        "k_clear_depth": 4 * npx,
        # per cascade: xyz of every triangle read, the casters listed
        "k_shadow_setup": 36 * T + 4 * (cast + cast_a),
        # xyz (+ uv) of the casters read, the map written once
        "k_shadow_raster": 36 * cast + 4 * smap,
        "k_shadow_raster_alpha": 60 * cast_a,
        # tiled pass: caster records (32 B) and units (4 B), map tiles read and written once
        "k_shadow_bin": 16 * (cast + cast_a) + 4 * units,
        "k_shadow_sort": 8 * units,
        "k_shadow_tiles": 32 * cast + 4 * units + 8 * smap,
        "k_shadow_tiles_alpha": 56 * cast_a,
        "k_clear_shadow": 4 * smap,
    }


def issue_of(kernel, avg_s, sms, sm_mhz):
    """The instruction-issue roofline of a kernel: the issued warp
    instructions of a frame's launches of it (ncu) / `avg_s`, their CUDA-event
    time in a frame, against sms x 4 schedulers x the SM clock sampled during
    the run."""
    n = NCU_ISSUED.get(kernel)
    if n is None or not avg_s:
        return None
    peak = sms * ISSUE_PER_SM_PER_CLK * sm_mhz * 1e6
    return {"warp_inst_per_launch": n, "achieved_winst_per_s": n / avg_s, "peak_winst_per_s": peak,
            "frac": n / avg_s / peak, "sm_mhz": sm_mhz, "capture": NCU_CAPTURE}


def roofline_of(kernel, ktimes, alg, hbm, peak_kind, steps, sms=148, sm_mhz=1965.0):
    """achieved = the kernel's algorithmic bytes per launch / its average
    CUDA-event launch time; frac against the measured HBM peak.  `issue`
    is the same launch against the instruction-issue peak."""
    ms, n = ktimes[kernel]
    avg_s = ms / n / 1000.0
    a = alg.get(kernel, 0)
    achieved = a / avg_s / 1e9
    t = NCU_TRAFFIC.get(kernel)
    return {"bound": "hbm", "kernel": kernel, "achieved": achieved, "peak": hbm, "unit": "GB/s",
            "frac": achieved / hbm, "peak_source": peak_kind, "traffic": t,
            "traffic_capture": NCU_CAPTURE if t is not None else None, "algorithmic_bytes": a,
            "avg_us": 1e6 * avg_s, "launches_per_frame": n / steps, "issue": issue_of(kernel, avg_s * n / steps, sms, sm_mhz)}


def frame_bytes(scene):
    """Per-frame algorithmic bytes B = 132 T + sum_c (36 T_cast + 24 T_alpha) + 10 W H + 4 sum S^2."""
    T = scene.ntris
    casts = sum(g.ntris for g in scene.groups if g.cast)
    alpha = sum(g.ntris for g in scene.groups if g.cast and g.flags & 2)
    return 132 * T + len(scene.shadows) * (36 * casts + 24 * alpha) + 10 * W * H + 4 * sum(
        sc.dim * sc.dim for sc in scene.shadows)


# ------------------------------------------------------------------ CPU legs

def cpu_oracle_baseline(scene, view, budget_s=12.0):
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle as O
    O.build_oracle()
    nthreads = os.cpu_count() or 1
    n, t0 = 0, time.perf_counter()
    while True:
        O.render(scene, view, nthreads=nthreads)
        n += 1
        el = time.perf_counter() - t0
        if el >= budget_s or n >= 20:
            break
    out = {"value": n / el, "unit": "frames/s", "cores": nthreads, "kind": "port",
           "sample": f"{n} full frames (2 shadow cascades + 1920x1080 drawAll, 1,044,288 triangles) "
                     f"on the C oracle with OpenMP, {el:.1f} s"}
    t0 = time.perf_counter()
    O.render(scene, view, nthreads=1)
    el1 = time.perf_counter() - t0
    out["one_core"] = {"value": 1.0 / el1, "unit": "frames/s", "cores": 1,
                       "sample": f"1 full frame of the same workload on one thread, {el1:.1f} s"}
    out["stages"] = cpu_stage_baseline(O, scene, view)
    return out


def cpu_stage_baseline(O, scene, view):
    """The reference's own kernels for the vertex stage and the post effects
    (Pipe/vert.c, Post/ssao.c, dof.c, blur.c + blur2.c, compiled for the CPU
    in oracle/_ref and run work-item by work-item on one core; the bloom's
    256 work-items run as threads over all cores) on the same
    work the vertex and post sections time on the GPU: one rotation of the
    two sphere groups, one vertLight of both with the same light set, and
    ssao, dof(8) and the bloom of one 1080p frame.  Milliseconds per call."""
    if not O.ref_available():
        return {"unavailable": "oracle/_ref is not built"}
    from axi_visualizer_b200 import scenes as S
    spheres = S.Scene([scene.groups[2], scene.groups[3]], [], scene.lint, scene.ldir, scene.amb, scene.shadows,
                      scene.bias)
    rd = O.RefDraw(spheres, view)
    out = {"kind": "reference", "cores": 1, "bloom_cores": os.cpu_count() or 1}   # the bloom: a thread a work-item
    t0 = time.perf_counter()
    rd.rotate(_rot_y(0.0), _rot_y(0.01), (0.0, 0.0, 0.0), 0, spheres.groups[0].ntris * 3, 0)
    rd.rotate(_rot_y(0.0), _rot_y(0.01), (0.0, 0.0, 0.0), 0, spheres.groups[1].ntris * 3, 1)
    out["rotate_two_sphere_groups_ms"] = 1000 * (time.perf_counter() - t0)
    L = VERTEX_LIGHTS
    t0 = time.perf_counter()
    rd.vert_light([1, 1], L["dirI"], L["dirD"], scene.amb, L["pointI"], L["pointP"], L["spotI"], L["spotD"],
                  L["spotP"])
    out["vert_light_two_sphere_groups_ms"] = 1000 * (time.perf_counter() - t0)
    fr, _ = O.render(scene, view, nthreads=os.cpu_count() or 1)
    rd.set_frame(fr.ro, fr.go, fr.bo, fr.db)
    rnd = np.random.default_rng(44).random(48).astype(np.float32)
    for name, fn in (("ssao_ms", lambda: rd.ssao(rnd)), ("dof_ms", lambda: rd.dof(8.0)), ("bloom_ms", rd.bloom)):
        t0 = time.perf_counter()
        fn()
        out[name] = 1000 * (time.perf_counter() - t0)
    return out


REF_BUDGET_S = 120.0     # wall time the reference arm's warm-up + timed steps aim at


def split_scene(scene, parts):
    """The scene with every group cut into `parts` contiguous triangle slices,
    slice-major: groups [k * G, (k + 1) * G) hold slice k of groups 0..G-1."""
    from axi_visualizer_b200 import scenes as S
    out = []
    for k in range(parts):
        for g in scene.groups:
            t = len(g.xyz) // 3
            a, b = 3 * (t * k // parts), 3 * (t * (k + 1) // parts)
            out.append(S.Group(g.xyz[a:b], g.uv[a:b], g.vn[a:b], g.li[a:b], g.tex, g.tex_size, g.flags,
                               g.alpha_index, g.mip_bias, g.cast))
    return S.Scene(out, scene.alphas, scene.lint, scene.ldir, scene.amb, scene.shadows, scene.bias)


def reference_arm(args):
    """The reference's own draw kernels (compiled for the host CPU from their
    sources, oracle/_ref) on the 1080p / 1,044,288-triangle scene, with all
    host threads.  A step is a bounded sample: 1/B of a frame -- slice k of
    every group's triangles through both shadow cascades and drawAll -- and
    B consecutive steps make one whole frame (clears at slice 0, read-back of
    the frame at slice B-1).  B is sized from one untimed frame so that the
    warm-up and timed steps take about REF_BUDGET_S; frames/s = steps / B /
    time."""
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return 0
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle as O
    from axi_visualizer_b200 import scenes as S
    if not O.ref_available():
        print(json.dumps({"impl": "reference", "unavailable": "oracle/_ref was not built (reference checkout absent at build time)"}))
        return 0
    scene = S.reference_kernel_variant(S.scene_c2())
    view = S.default_view(W, H)
    nthreads = os.cpu_count() or 1
    ng = len(scene.groups)

    # one untimed whole frame sizes the sample
    rd = O.RefDraw(scene, view)
    t0 = time.perf_counter()
    for k in range(len(scene.shadows)):
        rd.shadow_map(k, nthreads=nthreads, read=False)
    rd.clear_zbuffer()
    if rd.draw_all(nthreads=nthreads) != 0:
        raise RuntimeError("reference drawAll failed")
    rd.get_frame()
    t_frame = time.perf_counter() - t0
    del rd
    parts = int(min(64, max(1, math.ceil(t_frame * (args.steps + args.warmup) / REF_BUDGET_S))))
    sp = split_scene(scene, parts)
    rs = O.RefDraw(sp, view)
    masks = [np.array([0 if j // ng == k else 1 for j in range(ng * parts)], np.uint8) for k in range(parts)]
    casts = [np.array([(j // ng == k) and bool(g.cast) for j, g in enumerate(sp.groups)], np.uint8)
             for k in range(parts)]
    state = {"i": 0}

    def step():
        k = state["i"] % parts
        state["i"] += 1
        for m in range(len(scene.shadows)):
            rs.shadow_map(m, cast=casts[k], nthreads=nthreads, clear=(k == 0), read=False)
        if k == 0:
            rs.clear_zbuffer()
        if rs.draw_all(mask=masks[k], nthreads=nthreads) != 0:
            raise RuntimeError("reference drawAll failed")
        if k == parts - 1:
            rs.get_frame()

    for _ in range(args.warmup):
        step()
    state["i"] = 0
    lat = []
    t0 = time.perf_counter()
    for _ in range(args.steps):
        t1 = time.perf_counter()
        step()
        lat.append(time.perf_counter() - t1)
    el = time.perf_counter() - t0
    fps = args.steps / parts / el
    sample = (f"each step 1/{parts} of a frame (slice k of every group's triangles: both shadow cascades and "
              f"drawAll), {parts} steps = one frame; {args.steps} steps timed; one whole frame took "
              f"{t_frame:.2f} s")
    line = {
        "metric": METRIC, "value": fps, "unit": "frames/s", "n_gpus": args.gpus, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": 1000 * el / args.steps, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic (seeded)",
        "impl": "reference",
        "config": {"workload": "c2_plain_1080p_1m_tris", "width": W, "height": H, "triangles": scene.ntris,
                   "shadow_cascades": [sc.dim for sc in scene.shadows], "steps_per_frame": parts,
                   "shader": "reference kernels drawtexcolsmp/drawtexcolsmpalpha (bilinear base level, no shadow "
                             "lookup: the reference ships no trilinear+double-cascade kernel), drawmin/drawminalpha"},
        "Mtri_per_s": scene.ntris * fps / 1e6, "Mpix_per_s": W * H * fps / 1e6,
        "frame_ms_whole": 1000 * t_frame,
        "p50_step_ms": 1000 * float(np.percentile(lat, 50)), "p99_step_ms": 1000 * float(np.percentile(lat, 99)),
        "cpu_baseline": {"value": fps, "unit": "frames/s", "cores": nthreads, "kind": "reference",
                         "sample": sample + "; the reference's OpenCL kernels compiled for the CPU, one work-group "
                                            "per thread"},
        "e2e": {"value": fps, "unit": "frames/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line))
    return 0


# ------------------------------------------------------------------ batched multi-view

def batched_section(steps, device, log=progress):
    """Batched multi-view frame of the 24,192-triangle scene: 6 cube faces at
    512^2, cascades at 2048^2 and 1024^2 and the 1920x1080 main view, as one
    graph-replayed persistent launch, against the same nine views issued as
    plain per-view calls (two handles: 1920x1080 and 512x512, each with its
    own cascades because the plain API keeps shadow maps per handle)."""
    import torch
    from axi_visualizer_b200 import autotune
    from axi_visualizer_b200 import scenes as S
    from axi_visualizer_b200.batch import Batch, scene_batch_views
    from axi_visualizer_b200.ops import SceneRenderer

    sc = S.scene_c3()
    main = S.default_view(W, H)
    eye = (0.0, 5.0, -25.0)
    R = SceneRenderer(sc, W, H, device=device)
    descs = scene_batch_views(sc, main, faces_at=eye, face_side=512)
    B = Batch(R.draw, descs)
    flags = [g.flags for g in sc.groups]
    aidx = [g.alpha_index for g in sc.groups]
    tuned = autotune.tune(B, flags, aidx, ntris=sc.ntris, gpu=torch.cuda.get_device_name(device), log=log)
    stream = torch.cuda.ExternalStream(R.draw.stream_ptr(), device=f"cuda:{device}")
    for _ in range(3):
        B.render(flags, aidx)
    R.draw.sync()
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(steps + 1)]
    ev[0].record(stream)
    for i in range(steps):
        B.render(flags, aidx)
        ev[i + 1].record(stream)
    R.draw.sync()
    per = np.array([ev[i].elapsed_time(ev[i + 1]) for i in range(steps)])
    batch_ms = ev[0].elapsed_time(ev[-1]) / steps

    # plain per-view calls
    from axi_visualizer_b200.batch import cube_faces
    F = SceneRenderer(sc, 512, 512, device=device)
    faces = cube_faces(eye, 512)
    casc = [0, 1]

    def plain_frame():
        R.frame(main)
        F.shadow_pass()
        for fv in faces:
            F.set_view(fv)
            F.draw.clearZBuffer()
            F.draw.drawAll(F.shaders, shadowIds=casc)

    for _ in range(3):
        plain_frame()
    R.draw.sync()
    F.draw.sync()
    t0 = time.perf_counter()
    for _ in range(steps):
        plain_frame()
    R.draw.sync()
    F.draw.sync()
    plain_ms = 1000 * (time.perf_counter() - t0) / steps
    pix = sum(d.w * (d.h if d.kind == 0 else d.w) for d in descs)
    st = B.stats()
    return {"workload": "c3_batched_9_views", "triangles": sc.ntris,
            "views": [f"{'shaded' if d.kind == 0 else 'depth'} {d.w}x{d.h if d.kind == 0 else d.w}" for d in descs],
            "frames_per_s": 1000.0 / batch_ms, "ms_per_frame": batch_ms,
            "p50_ms": float(np.percentile(per, 50)), "p99_ms": float(np.percentile(per, 99)),
            "Mpix_per_s": pix * 1000.0 / batch_ms / 1e6,
            "plain_frames_per_s": 1000.0 / plain_ms, "plain_ms_per_frame": plain_ms,
            "speedup_vs_plain": plain_ms / batch_ms, "graph": st["graph"], "grid_blocks": st["grid"],
            "tuning": {k: tuned[k] for k in ("mode", "blocks_per_sm", "min_chunk", "ms", "cached")}}


# ------------------------------------------------------------------ 640x480

def small_section(device, frames=300):
    """The 640x480 scene (64x64 terrain + 200 icospheres = 24,192 triangles,
    one 512^2 trilinear texture, one 1024^2 shadow map): frames/s of shadow
    pass + drawAll, device-timed with CUDA events; a launch-bound frame."""
    import torch
    from axi_visualizer_b200 import scenes as S
    from axi_visualizer_b200.ops import SceneRenderer
    sc = S.scene_c1()
    view = S.default_view(640, 480)
    R = SceneRenderer(sc, 640, 480, device=device)
    stream = torch.cuda.ExternalStream(R.draw.stream_ptr(), device=f"cuda:{device}")
    for _ in range(10):
        R.frame(view)
    R.draw.sync()
    launches0 = R.draw.launchCount()
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(frames + 1)]
    ev[0].record(stream)
    for i in range(frames):
        R.frame(view)
        ev[i + 1].record(stream)
    R.draw.sync()
    launches = (R.draw.launchCount() - launches0) / frames
    per = np.array([ev[i].elapsed_time(ev[i + 1]) for i in range(frames)])
    ms = ev[0].elapsed_time(ev[-1]) / frames
    return {"workload": "c1_plain_640x480_24k_tris", "triangles": sc.ntris, "frames_per_s": 1000.0 / ms,
            "ms_per_frame": ms, "p50_ms": float(np.percentile(per, 50)), "p99_ms": float(np.percentile(per, 99)),
            "Mtri_per_s": sc.ntris / ms / 1e3, "Mpix_per_s": 640 * 480 / ms / 1e3,
            "launches_per_frame": launches}


# ------------------------------------------------------------------ vertex stage

def _rot_y(a):
    c, s = np.cos(a), np.sin(a)
    return np.array([[c, 0, s], [0, 1, 0], [-s, 0, c]])


def _vertex_lights():
    rng = np.random.default_rng(11)
    return {"dirI": np.array([(1.6, 1.4, 1.2), (0.5, 0.5, 0.5), (0.1, 0.2, 0.6)]),
            "dirD": np.array([(0.3, -0.8, 0.5), (-0.3, 0.8, -0.5), (0.0, 1.0, 0.0)]),
            "pointI": rng.uniform(0, 3, (4, 3)), "pointP": rng.uniform(-20, 20, (4, 3)) + (0, 8, 0),
            "spotI": rng.uniform(0, 3, (2, 3)), "spotD": np.array([(0, -1, 0), (0.6, -0.8, 0)]),
            "spotP": np.array([(0, 15, 0), (-10, 12, -5)])}


VERTEX_LIGHTS = _vertex_lights()


def vertex_section(R, view, hbm, frames=100, warmup=5):
    """An animated 1080p frame: both sphere groups (2 x 240,000 triangles)
    turn about the scene centre (CLDraw.rotate, undoing the previous turn and
    applying the next), the per-vertex light of every group is recomputed
    from 2 extra directional, 4 point and 2 spot lights (CLDraw.vertLight),
    then both cascades and drawAll render.  Frames/s device-timed with CUDA
    events; the vertex kernels' HBM throughput from their event times, at
    48 B a rotated vertex (position + normal read and written) and 36 B a
    lit vertex (position + normal read, light written)."""
    import torch
    D = R.draw
    scene = R.scene
    spheres = [2, 3]
    stream = torch.cuda.ExternalStream(D.stream_ptr(), device=torch.cuda.current_device())
    L = VERTEX_LIGHTS
    dirI, dirD, pointI, pointP = L["dirI"], L["dirD"], L["pointI"], L["pointP"]
    spotI, spotD, spotP = L["spotI"], L["spotD"], L["spotP"]
    mask = [1] * len(scene.groups)
    state = {"k": 0}

    def step():
        k = state["k"]
        prev, new = _rot_y(0.01 * k), _rot_y(0.01 * (k + 1))
        for g in spheres:
            D.rotate(prev, new, (0.0, 0.0, 0.0), 0, None, g)
        D.vertLight(mask, dirI, dirD, pointI, pointP, spotI, spotD, spotP)
        R.frame(view)
        state["k"] = k + 1

    for _ in range(warmup):
        step()
    D.sync()
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    ev[0].record(stream)
    for _ in range(frames):
        step()
    ev[1].record(stream)
    D.sync()
    ms = ev[0].elapsed_time(ev[1]) / frames
    D.setKernelTiming(True)
    for _ in range(frames):
        step()
    kt = D.kernelTimes()
    D.setKernelTiming(False)
    # the scene's own geometry and light back on the device
    for g in spheres:
        D.copyTo(g, scene.groups[g].xyz, scene.groups[g].vn)
    D.vertLight(mask, dirI, dirD, 1, None, 1)
    for g, G in enumerate(scene.groups):
        D.setVertLight(g, G.li)
    D.sync()
    nv_rot = sum(scene.groups[g].ntris * 3 for g in spheres)
    nv_all = scene.ntris * 3
    out = {"workload": "c2_animated_1080p_1m_tris", "rotated_vertices": nv_rot, "lit_vertices": nv_all,
           "lights": {"directional": len(dirI) - 1, "point": len(pointI), "spot": len(spotI)},
           "frames_per_s": 1000.0 / ms, "ms_per_frame": ms}
    for name, per_v, nv, calls in (("k_vert_xform", 48, nv_rot // len(spheres), len(spheres)),
                                   ("k_vert_light", 36, None, None)):
        if name not in kt:
            continue
        tot_ms, n = kt[name]
        avg_s = tot_ms / n / 1000.0
        if nv is None:   # all lit vertices over a frame's launches
            nv = nv_all / (n / frames)
        gbs = per_v * nv / avg_s / 1e9
        out[name] = {"avg_us": avg_s * 1e6, "launches_per_frame": n / frames, "bytes_per_vertex": per_v,
                     "achieved_gbs": gbs, "frac_of_hbm": gbs / hbm}
    return out


def post_section(R, view, hbm, frames=50):
    """Post effects on the 1080p frame (CLDraw.ssao, CLDraw.dof(8),
    CLDraw.blur) after every rendered frame: their kernels' CUDA-event times
    and HBM throughput.  ssao and dof: 16 algorithmic bytes a pixel each
    (depth and colour read, colour written; the gathered neighbours are
    re-reads that stay in cache).  The bloom's two launches: 6 + 6 bytes a
    half-resolution pixel (the horizontal blur written and read) and 18 a
    full-resolution one (colour read by both, written by the second)."""
    D = R.draw
    rnd = np.random.default_rng(44).random(48).astype(np.float32)

    def step():
        R.frame(view); D.ssao(rnd); D.dof(8.0); D.blur()

    for _ in range(3):
        step()
    D.sync()
    D.setKernelTiming(True)
    for _ in range(frames):
        step()
    kt = D.kernelTimes()
    D.setKernelTiming(False)
    D.sync()
    px = view.w * (view.h // 16 * 16)
    out = {"workload": "c2_post_1080p", "pixels": px}
    for name in ("k_ssao", "k_dof"):
        tot_ms, n = kt[name]
        avg_s = tot_ms / n / 1000.0
        gbs = 16 * px / avg_s / 1e9
        out[name] = {"avg_us": avg_s * 1e6, "bytes_per_pixel": 16, "achieved_gbs": gbs, "frac_of_hbm": gbs / hbm}
    names = ("k_bloom_h", "k_bloom_v")
    if all(k in kt for k in names):
        half = (view.w // 2) * (view.h // 2)
        us = sum(1000 * kt[k][0] / kt[k][1] for k in names)
        b = 12 * half + 18 * view.w * view.h
        out["bloom"] = {"avg_us": us, "passes_us": {k: 1000 * kt[k][0] / kt[k][1] for k in names},
                        "algorithmic_bytes": b, "achieved_gbs": b / us / 1e3, "frac_of_hbm": b / us / 1e3 / hbm}
    return out


# ------------------------------------------------------------------ stress

def stress_section(device, frames=10, log=progress):
    """Stress workload: 3840x2160, 9,988,608 triangles (2048^2 terrain in 12
    bands + 20,000 icospheres in 4 groups), 16 trilinear 4096^2 textures, 29%
    of the triangles alpha-tested, two 4096^2 cascades.  Plain frame (both
    cascades + drawAll) and the batched launch of the cascades, the main view
    and six 1024^2 cube faces, each device-timed with CUDA events."""
    import torch
    from axi_visualizer_b200 import scenes as S
    from axi_visualizer_b200.batch import Batch, scene_batch_views
    from axi_visualizer_b200.ops import SceneRenderer

    log("stress: building scene")
    t0 = time.perf_counter()
    sc = S.scene_c5()
    gen_s = time.perf_counter() - t0
    w, h = 3840, 2160
    main = S.default_view(w, h, pos=(0.0, 8.0, -40.0))
    R = SceneRenderer(sc, w, h, device=device)
    D = R.draw
    stream = torch.cuda.ExternalStream(D.stream_ptr(), device=f"cuda:{device}")

    def timed(step, n):
        for _ in range(2):
            step()
        D.sync()
        ev = [torch.cuda.Event(enable_timing=True) for _ in range(n + 1)]
        ev[0].record(stream)
        for i in range(n):
            step()
            ev[i + 1].record(stream)
        D.sync()
        return np.array([ev[i].elapsed_time(ev[i + 1]) for i in range(n)])

    log("stress: plain frames")
    plain = timed(lambda: R.frame(main), frames)
    st = D.lastStats()
    log("stress: batched launch")
    descs = scene_batch_views(sc, main, faces_at=(0.0, 8.0, -30.0), face_side=1024)
    B = Batch(D, descs)
    flags = [g.flags for g in sc.groups]
    aidx = [g.alpha_index for g in sc.groups]
    from axi_visualizer_b200 import autotune
    tuned = autotune.tune(B, flags, aidx, ntris=sc.ntris, reps=3, gpu=torch.cuda.get_device_name(device), log=log)
    batched = timed(lambda: B.render(flags, aidx), frames)
    graph = B.stats()["graph"]
    del B
    log("stress: the same views as plain per-view calls")
    from axi_visualizer_b200.batch import cube_faces
    F = SceneRenderer(sc, 1024, 1024, device=device)
    faces = cube_faces((0.0, 8.0, -30.0), 1024)

    def plain_views():
        R.frame(main)
        F.shadow_pass()                 # the plain API keeps shadow maps per handle
        for fv in faces:
            F.set_view(fv)
            F.draw.clearZBuffer()
            F.draw.drawAll(F.shaders, shadowIds=[0, 1])

    for _ in range(2):
        plain_views()
    D.sync()
    F.draw.sync()
    t1 = time.perf_counter()
    for _ in range(frames):
        plain_views()
    D.sync()
    F.draw.sync()
    plain_views_ms = 1000 * (time.perf_counter() - t1) / frames
    del F
    pix = sum(d.w * (d.h if d.kind == 0 else d.w) for d in descs)
    ntri = sc.ntris
    alpha = sum(g.ntris for g in sc.groups if g.flags & S.ALPHA) / ntri
    pm, bm = float(np.median(plain)), float(np.median(batched))
    return {"workload": "c5_stress_4k_10m_tris", "width": w, "height": h, "triangles": ntri,
            "materials": len(sc.groups), "texture_side": 4096, "alpha_fraction": round(alpha, 4),
            "shadow_cascades": [c.dim for c in sc.shadows], "scene_build_s": round(gen_s, 1),
            "queues": st,
            "plain": {"frames_per_s": 1000.0 / pm, "ms_per_frame": pm, "p99_ms": float(np.percentile(plain, 99)),
                      "Mtri_per_s": ntri / pm / 1e3, "Mpix_per_s": w * h / pm / 1e3},
            "batched": {"views": [f"{'shaded' if d.kind == 0 else 'depth'} {d.w}x{d.h if d.kind == 0 else d.w}"
                                  for d in descs],
                        "frames_per_s": 1000.0 / bm, "ms_per_frame": bm, "p99_ms": float(np.percentile(batched, 99)),
                        "Mpix_per_s": pix / bm / 1e3, "graph": graph,
                        "tuning": {k: tuned[k] for k in ("mode", "blocks_per_sm", "min_chunk", "ms", "cached")},
                        "plain_views_ms": plain_views_ms,
                        "plain_views_frames_per_s": 1000.0 / plain_views_ms,
                        "speedup_vs_plain": plain_views_ms / bm}}


# ------------------------------------------------------------------ serving

def served_section(device, n_poisson=1000, n_burst=400, rates=(200.0, 1000.0), tuning=None, log=progress):
    """Serving workload: 8 resident scenes (seeds 10-17, 50k-1M triangles
    each), Poisson arrivals, resolutions 640x360 / 1280x720 / 1920x1080 /
    2560x1440 with p = 0.4/0.3/0.2/0.1, random camera poses, a 150 GB HBM
    budget; each request's colour planes and depth are copied back to pinned
    host memory.  Runs the named rate (200 requests/s), a rate near the plain
    path's capacity, and a burst of requests all arriving at t=0 (the
    saturated rate); the same traces run through the plain per-view path
    (first come first served, one drawAll + getFrame each)."""
    from axi_visualizer_b200 import scenes as S
    from axi_visualizer_b200 import serve as SV

    log("served: building scenes")
    scenes = [S.scene_served(s) for s in S.SERVING_SEEDS]
    res = SV.ResidentScenes(scenes, device=device)
    srv = SV.Server(SV.GpuBackend(res, tuning=tuning), budget_bytes=SV.HBM_BUDGET, resident_bytes=res.nbytes,
                    max_slabs=8, depth=2)
    plain = SV.PlainServer(scenes, SV.RESOLUTIONS, device=device)
    warm = SV.poisson_trace(40, 1e6, len(scenes), seed=99, burst=True)
    log("served: warm-up")
    srv.prepare(srv.max_slabs)
    srv.prepare_solo()
    srv.run(warm)
    srv.run(SV.poisson_trace(8, 50.0, len(scenes), seed=98))    # warms the single-slot slabs too
    plain.run(SV.poisson_trace(40, 1e6, len(scenes), seed=99, burst=True))
    keep = ("frames_per_s", "Mpix_per_s", "p50_ms", "p99_ms", "max_ms", "done")
    sched = ("views_per_launch", "launches", "max_inflight", "slabs")
    runs, peak = [], 0
    cases = [(f"poisson_{r:g}", SV.poisson_trace(n_poisson if r <= 200 else 2 * n_poisson, r, len(scenes), seed=1 + i),
              r) for i, r in enumerate(rates)]
    cases.append(("burst", SV.poisson_trace(n_burst, 1.0, len(scenes), seed=7, burst=True), None))
    for name, trace, rate in cases:
        log(f"served: {name}")
        srv.reset_stats()
        st = srv.run(trace)
        peak = max(peak, st["hbm_used_peak_bytes"])
        twin = [SV.Request(r.rid, r.scene, r.w, r.h, r.pos, r.target, r.arrival) for r in trace]
        pst = plain.run(twin)
        runs.append({"trace": name, "rate_req_per_s": rate, "requests": len(trace),
                     "served": {k: st[k] for k in keep + sched}, "plain": {k: pst[k] for k in keep},
                     "speedup_vs_plain": st["frames_per_s"] / pst["frames_per_s"]})
    srv.close()
    return {
        "workload": "c4_served", "scenes": len(scenes), "scene_triangles": [d["tris"] for d in res.info],
        "resolutions": [f"{w}x{h}" for w, h in SV.RESOLUTIONS], "probs": list(SV.RES_PROBS),
        "slab_layout": {f"{w}x{h}": n for (w, h), n in SV.DEFAULT_LAYOUT.items()}, "pipeline_depth": srv.depth,
        "hbm_budget_gb": SV.HBM_BUDGET / 1e9, "resident_gb": res.nbytes / 1e9, "hbm_used_peak_gb": peak / 1e9,
        "slab_gb": srv.slab_bytes / 1e9, "d2h": "colour planes + depth per request", "runs": runs,
    }


# ------------------------------------------------------------------ GPU arm

class Ranks:
    """Rank plumbing of a replicas run: one process per GPU (RANK, LOCAL_RANK,
    WORLD_SIZE, MASTER_* from the launcher), each rendering its own frames of
    its own resident copy of the scene; no collective touches the data path.
    The only collectives are the barriers around the timed region and the
    max over ranks of its device time."""

    def __init__(self, backend="nccl", timeout_s=300):
        import torch
        import torch.distributed as dist
        self.dist = dist
        self.world = int(os.environ.get("WORLD_SIZE", "1"))
        self.rank = int(os.environ.get("RANK", "0"))
        self.local = int(os.environ.get("LOCAL_RANK", "0"))
        self.device = "cpu"
        if self.world > 1:
            import datetime
            if backend == "nccl":
                torch.cuda.set_device(self.local)
                self.device = f"cuda:{self.local}"
            dist.init_process_group(backend, timeout=datetime.timedelta(seconds=timeout_s))

    def barrier(self):
        if self.world > 1:
            self.dist.barrier()

    def max(self, x):
        """max over ranks of a float (every rank gets it)."""
        if self.world == 1:
            return x
        import torch
        t = torch.tensor([x], dtype=torch.float64, device=self.device)
        self.dist.all_reduce(t, op=self.dist.ReduceOp.MAX)
        return float(t.item())

    def close(self):
        if self.world > 1 and self.dist.is_initialized():
            self.dist.destroy_process_group()


def whole_job_rate(units_per_rank, world, slowest_s):
    """Whole-job throughput of a weak-scaling replicas run: every rank did
    the same units, the job took as long as its slowest rank."""
    return units_per_rank * world / slowest_s


def _smi_index(torch, local):
    """nvidia-smi id of the CUDA device `local` (PCI bus id when available)."""
    try:
        p = torch.cuda.get_device_properties(local)
        return f"{p.pci_domain_id:08X}:{p.pci_bus_id:02X}:{p.pci_device_id:02X}.0"
    except Exception:
        vis = os.environ.get("CUDA_VISIBLE_DEVICES", "")
        ids = [x for x in vis.split(",") if x.strip()]
        return ids[local] if local < len(ids) else str(local)


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=300)
    ap.add_argument("--warmup", type=int, default=10)
    ap.add_argument("--impl", default="axr", choices=["axr", "reference"])
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-batched", action="store_true")
    ap.add_argument("--no-served", action="store_true")
    ap.add_argument("--no-stress", action="store_true")
    ap.add_argument("--no-small", action="store_true")
    ap.add_argument("--no-vertex", action="store_true")
    args = ap.parse_args()
    args.warmup = max(args.warmup, 3)
    if args.impl == "reference":
        return reference_arm(args)

    import torch
    from axi_visualizer_b200 import scenes as S
    from axi_visualizer_b200.ops import SceneRenderer

    ranks = Ranks("nccl")
    world, rank, local = ranks.world, ranks.rank, ranks.local
    barrier, max_over_ranks = ranks.barrier, ranks.max

    progress("scene")
    scene = S.scene_c2()
    view = S.default_view(W, H)
    R = SceneRenderer(scene, W, H, device=local, pinned=True)
    D = R.draw
    stream = torch.cuda.ExternalStream(D.stream_ptr(), device=f"cuda:{local}")

    progress("warmup")
    for _ in range(args.warmup):
        R.frame(view)
    D.sync()
    stats = D.lastStats()

    progress("timed loop")
    # ---- device-timed loop (value): scene resident in HBM
    clocks = Clocks(_smi_index(torch, local))
    barrier()
    torch.cuda.synchronize()
    D.sync()
    launches0 = D.launchCount()
    evs = [torch.cuda.Event(enable_timing=True) for _ in range(args.steps + 1)]
    clocks.start()
    evs[0].record(stream)
    for i in range(args.steps):
        R.frame(view)
        evs[i + 1].record(stream)
    D.sync()
    torch.cuda.synchronize()
    clk = clocks.stop()
    gpu_launches = D.launchCount() - launches0
    frame_ms = np.array([evs[i].elapsed_time(evs[i + 1]) for i in range(args.steps)])
    t_ms = max_over_ranks(float(evs[0].elapsed_time(evs[-1])))
    barrier()
    fps = whole_job_rate(args.steps, world, t_ms / 1000.0)

    progress("render loop")
    # the reference's render loop (Compute.py ThreeDBackend.render: setPos,
    # setVM, clearZBuffer, drawAll) with the shadow maps resident, as its
    # apps render them once: reported beside the headline frame, which
    # renders both cascades every frame
    R.shadow_pass()
    D.sync()

    def render_loop_step():
        R.set_view(view)
        D.clearZBuffer()
        D.drawAll(R.shaders, shadowIds=[0, 1])

    for _ in range(args.warmup):
        render_loop_step()
    D.sync()
    rl = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    rl[0].record(stream)
    for _ in range(args.steps):
        render_loop_step()
    rl[1].record(stream)
    D.sync()
    rl_ms = max_over_ranks(float(rl[0].elapsed_time(rl[1]))) / args.steps

    progress("kernel timing")
    # ---- per-kernel device times (roofline) on a second pass
    D.setKernelTiming(True)
    for _ in range(args.steps):
        R.frame(view)
    ktimes = D.kernelTimes()
    D.setKernelTiming(False)
    tid, cov = D.getIDs()
    visible = int(np.unique(tid[tid >= 0]).size)
    queues = D.lastQueues()
    shadow_q = [D.shadowStats(k) for k in range(len(scene.shadows))]
    alg = algorithmic_bytes(scene, queues, shadow_q, visible)
    hbm, peak_kind = peaks()
    per_kernel = {k: {"avg_us": 1000 * ms / n, "launches_per_frame": n / args.steps,
                      "share": 0.0} for k, (ms, n) in ktimes.items()}
    tot = sum(ms for ms, n in ktimes.values())
    for k, (ms, n) in ktimes.items():
        per_kernel[k]["share"] = ms / tot if tot else 0.0
        per_kernel[k]["algorithmic_bytes"] = alg.get(k)
        if k in alg:
            per_kernel[k]["frac_of_hbm"] = alg[k] / (ms / n / 1000.0) / 1e9 / hbm
    # the dominant kernel by its share of the frame, and by its time per launch
    sms = torch.cuda.get_device_properties(local).multi_processor_count
    sm_mhz = clk["sm_mhz"] if clk else 1965.0
    for k, (ms, n) in ktimes.items():
        iss = issue_of(k, ms / args.steps / 1000.0, sms, sm_mhz)
        if iss:
            per_kernel[k]["issue_frac"] = iss["frac"]
    dom = max(ktimes.items(), key=lambda kv: kv[1][0])[0]
    dom_launch = max(ktimes.items(), key=lambda kv: kv[1][0] / kv[1][1])[0]
    roofline = roofline_of(dom, ktimes, alg, hbm, peak_kind, args.steps, sms, sm_mhz)
    roofline["by_launch"] = roofline_of(dom_launch, ktimes, alg, hbm, peak_kind, args.steps, sms, sm_mhz)
    fb = frame_bytes(scene)
    frame_roof = {"bytes": fb, "achieved_gbs": fb / (t_ms / args.steps / 1000.0) / 1e9}
    frame_roof["frac"] = frame_roof["achieved_gbs"] / hbm

    progress("e2e")
    # ---- end-to-end through the public API, host buffers, pinned memory
    barrier()
    pose = torch.empty(12, dtype=torch.float32, pin_memory=True).numpy()
    pose[:3] = view.pos
    pose[3:] = view.vv.reshape(-1)
    D.sync()
    e2e_lat = []

    def render_step():
        R.shadow_pass()
        D.setScaleCull(view.sscale, view.cax, view.cay)
        D.setPos(pose[:3])
        D.setVM(pose[3:].reshape(3, 3))
        D.clearZBuffer()
        D.drawAll(R.shaders, shadowIds=[0, 1])

    # frame loop with the asynchronous read-back: frame i's colour planes and
    # depth travel to pinned host memory while frame i + 1 renders (the
    # untimed warm-up makes the pinned host ring and the staging slots)
    for i in range(args.warmup):
        render_step()
        D.waitFrame(D.readFrameAsync())
    D.sync()
    barrier()
    t0 = time.perf_counter()
    prev = None
    for i in range(args.steps):
        t1 = time.perf_counter()
        render_step()
        tk = D.readFrameAsync()
        if prev is not None:
            D.waitFrame(prev[0])
            e2e_lat.append(time.perf_counter() - prev[1])
        prev = (tk, t1)
    D.waitFrame(prev[0])
    e2e_lat.append(time.perf_counter() - prev[1])
    e2e_s = max_over_ranks(time.perf_counter() - t0)
    e2e_fps = whole_job_rate(args.steps, world, e2e_s)
    # a display client: the frame read back as gamma-mapped 8-bit RGB packed
    # on the device (6.2 MB per frame instead of 20.7 MB), pipelined the same way
    for i in range(args.warmup):
        render_step()
        D.waitFrame(D.readFrameRGB8Async(1.0))
    D.sync()
    barrier()
    t0 = time.perf_counter()
    prev = None
    for i in range(args.steps):
        render_step()
        tk = D.readFrameRGB8Async(1.0)
        if prev is not None:
            D.waitFrame(prev)
        prev = tk
    D.waitFrame(prev)
    disp_s = max_over_ranks(time.perf_counter() - t0)
    disp_fps = whole_job_rate(args.steps, world, disp_s)
    # the same with the blocking getFrame of the reference's API
    barrier()
    D.sync()
    t0 = time.perf_counter()
    blk_lat = []
    for i in range(args.steps):
        t1 = time.perf_counter()
        render_step()
        D.getFrame()                      # D2H of colour planes + depth into pinned buffers (synchronises)
        blk_lat.append(time.perf_counter() - t1)
    blk_s = max_over_ranks(time.perf_counter() - t0)
    blk_fps = whole_job_rate(args.steps, world, blk_s)
    d2h = W * H * (3 * 2 + 4)
    h2d = 12 * 4 + 3 * 4 + 3 * len(scene.groups) * 96   # pose + scale/cull + 3 group tables per frame

    # the added sections are per-GPU measurements: rank 0 runs them (the
    # other replicas are done once the whole-job numbers above are taken)
    extra = rank == 0
    vertex = None
    if extra and not args.no_vertex:
        progress("vertex stage")
        vertex = vertex_section(R, view, hbm, frames=min(args.steps, 100))
    post = None
    if extra and not args.no_vertex:
        progress("post effects")
        post = post_section(R, view, hbm, frames=min(args.steps, 50))

    small = None
    if extra and not args.no_small:
        progress("640x480 scene")
        small = small_section(local)

    batched = None
    if extra and not args.no_batched:
        progress("batched multi-view")
        batched = batched_section(min(args.steps, 100), local)

    stress = None
    if extra and not args.no_stress:
        progress("stress")
        stress = stress_section(local)

    served = None
    if extra and not args.no_served:
        progress("served")
        tun = (batched["tuning"]["blocks_per_sm"], batched["tuning"]["min_chunk"]) if batched else None   # grid, rows
        served = served_section(local, tuning=tun)

    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        cpu = cpu_oracle_baseline(scene, view)

    if rank == 0:
        line = {
            "metric": METRIC, "value": fps, "unit": "frames/s", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": t_ms / args.steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic (seeded scene)",
            "config": {"workload": "c2_plain_1080p_1m_tris", "width": W, "height": H, "triangles": scene.ntris,
                       "materials": len(scene.groups), "shadow_cascades": [sc.dim for sc in scene.shadows],
                       "parallelism": f"replicas{world}", "l2": "inputs larger than L2 (geometry+textures "
                       f"{(sum(g.xyz.nbytes * 4 // 3 + g.tex[0].nbytes * 3 for g in scene.groups)) / 1e6:.0f} MB)"},
            "Mtri_per_s": scene.ntris * fps / 1e6, "Mpix_per_s": W * H * fps / 1e6,
            "p50_ms": float(np.percentile(frame_ms, 50)), "p99_ms": float(np.percentile(frame_ms, 99)),
            "e2e": {"value": e2e_fps, "unit": "frames/s", "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h,
                    "p50_ms": 1000 * float(np.percentile(e2e_lat, 50)), "p99_ms": 1000 * float(np.percentile(e2e_lat, 99)),
                    "read_back": "readFrameAsync / waitFrame (next frame renders during the copy)",
                    "blocking_getFrame": {"value": blk_fps, "p50_ms": 1000 * float(np.percentile(blk_lat, 50)),
                                          "p99_ms": 1000 * float(np.percentile(blk_lat, 99))},
                    "display_rgb8": {"value": disp_fps, "d2h_bytes_per_step": W * H * 3,
                                     "read_back": "readFrameRGB8Async (gamma + RGB8 packing on the device)"}},
            "gpu_launches": int(gpu_launches),
            "roofline": roofline,
            "frame_roofline": frame_roof,
            "render_loop": {"frames_per_s": whole_job_rate(1, world, rl_ms / 1000.0), "ms_per_frame": rl_ms,
                            "what": "setPos/setVM/clearZBuffer/drawAll with the cascades resident (the "
                                    "reference's render loop); the headline frame also renders both cascades"},
            "kernels": per_kernel,
            "queues": dict(stats, **queues, shadow=shadow_q),
            "clocks": clk,
            "cpu_baseline": cpu,
            "batched": batched,
            "served": served,
            "stress": stress,
            "small": small,
            "vertex": vertex,
            "post": post,
        }
        print(json.dumps(line))
    ranks.close()
    return 0


if __name__ == "__main__":
    sys.exit(main())
