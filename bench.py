#!/usr/bin/env python3
"""Benchmark: render throughput of the GB300 backend on the full-size plain
workload, beside the CPU renderer timed on this machine's host cores.

One step is one frame of the config-2 scene (4096 primitives in 512 CSG
groups with floor-based repetition, 40% matte / 40% GGX metal / 20%
dispersive glass, two quad lights and a constant 6500 K sky), 1920x1080 at
64 samples a pixel, paths of at most 16 surfaces: 132.7 M samples a step,
shown through the reference's reconstruction chain temporal + a-trous
(the record and the pixel-centre G-buffer as FP16 features; a still
camera, so each frame's history is the frame before's).
The scene is the reference renderer's own compilation of the seeded scene
text (tests/golden/scenes/c2.npz); the cut octree is built once before the
timed region and reported apart (build_s), as the reference reports its
tree build apart from its render time.

  value : Msamples/s over the K timed frames, device time (CUDA events on
          the backend's stream), scene resident in HBM, the L2 written over
          (a 512 MiB buffer) before every timed frame.
  e2e   : the same through the C ABI as a host caller drives it: each step
          uploads the frame's transport blocks (camera, lights, sky,
          materials, finishes) from host memory and reads the frame back to
          host memory; wall clock around the whole step.
  cpu_baseline : the oracle's C renderer (oracle/port) on the host cores
          over a bounded band of the same frame.

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl gb300|reference]
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
sys.path.insert(0, ROOT)

METRIC = "Msamples/s @1080p vs CPU; equal-time relMSE guided vs plain; p50/p99 latency"
SCENE = os.path.join(ROOT, "tests", "golden", "scenes", "c2.npz")
WIDTH, HEIGHT, SPP, SURFACES = 1920, 1080, 64, 16
DENOISE = True  # the temporal member and the a-trous denoiser on the frame's FP16 features
# The trace kernel's roof is FP32 issue (divergent SIMT work: neither HBM
# nor the tensor pipe bounds it).  From one ncu pass over every trace launch
# of a 960x540x8 config-2 frame (smsp__thread_inst_executed.sum and
# smsp__inst_executed.sum, with the frame's own program-step counters): the
# lane instructions the kernel issues a march-form program step, and the
# warp execution efficiency (active lanes an instruction / 32).
TRACE_LANE_INST_PER_PROGRAM_STEP = 78.2
TRACE_WARP_EFFICIENCY = 0.397
SM_COUNT, LANES_PER_SM = 152, 128
BUILD = dict(min_depth=7, max_depth=11, split_steps=32)


def env_int(name: str, default: int) -> int:
    try:
        return int(os.environ.get(name, default))
    except ValueError:
        return default


class Clocks:
    """nvidia-smi samples of the SM clock and throttle reasons while the
    timed region runs."""

    QUERY = "clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap"

    def __init__(self, index: int = 0):
        self.index = index
        self.samples: list[list[str]] = []
        self.proc = None

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.index), f"--query-gpu={self.QUERY}", "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.reader = threading.Thread(target=self._read, daemon=True)
            self.reader.start()
        except (FileNotFoundError, OSError):
            self.proc = None
        return self

    def _read(self):
        for line in self.proc.stdout:
            parts = [p.strip() for p in line.split(",")]
            if len(parts) >= 7:
                self.samples.append(parts)

    def __exit__(self, *exc):
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def summary(self) -> dict:
        if not self.samples:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["not sampled"]}
        sm = [float(s[0]) for s in self.samples if s[0].replace(".", "").isdigit()]
        mx = [float(s[1]) for s in self.samples if s[1].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[k] for s in self.samples for k in range(4) if s[3 + k].lower().startswith("active")})
        return {"sm_mhz": float(np.median(sm)) if sm else None, "sm_max_mhz": max(mx) if mx else None, "reasons": reasons, "samples": len(self.samples)}


WORKLOAD = "config-2: 4096 primitives, 1920x1080, 64 spp, 16 surfaces, FP32, temporal + a-trous denoiser on FP16 features"


def spread_rows(count: int) -> list[int]:
    """`count` rows spread evenly down the frame, so a CPU sample sees the
    frame's mix of sky, near and far geometry."""
    count = max(1, min(HEIGHT, count))
    return sorted({int((k + 0.5) * HEIGHT / count) for k in range(count)})


def cpu_rows(scene, rows: list[int], seed: int, threads: int) -> float:
    """The oracle's C renderer over the given rows; seconds."""
    import oracle.port as op
    t0 = time.perf_counter()
    for r in rows:
        op.render_band(scene, WIDTH, HEIGHT, SPP, SURFACES, seed, r, 1, threads, BUILD)
    return time.perf_counter() - t0


def cpu_baseline(scene, seconds: float = 15.0) -> dict:
    """The oracle's C renderer (double precision, the reference's algorithm)
    on every host core, over rows spread down the same frame: Msamples/s.
    The octree is built before the timed sample."""
    threads = os.cpu_count() or 1
    seed = int(scene.render["seed"])
    probe = spread_rows(4)
    cpu_rows(scene, probe[:1], seed, threads)  # builds the oracle's octree
    dt = cpu_rows(scene, probe, seed, threads)
    rows = spread_rows(max(1, int(len(probe) * seconds / max(dt, 1e-3))))
    dt = cpu_rows(scene, rows, seed, threads)
    samples = WIDTH * len(rows) * SPP
    return {"value": samples / dt / 1e6, "unit": "Msamples/s", "cores": threads, "kind": "port",
            "sample": f"{len(rows)} rows spread down the 1920x1080 frame at {SPP} spp ({samples} samples, {dt:.1f} s), no denoiser"}


def run_reference(args) -> None:
    """The reference arm runs the unmodified reference or nothing: neither its
    sources nor a build of it are on an Arm GPU machine, and a restatement of
    its algorithm is no reference (`cpu_baseline` times ours beside the GPU)."""
    if env_int("RANK", 0) == 0:
        print(json.dumps({"impl": "reference", "unavailable": "the reference renderer is not installed here: its sources are not on this machine and "
                          "its x86 build does not run on an Arm one"}), flush=True)


def run_gpu(args) -> None:
    import kodanuki_gb300 as K
    from kodanuki_gb300.scene import Scene

    rank, world = env_int("RANK", 0), env_int("WORLD_SIZE", 1)
    local = env_int("LOCAL_RANK", 0)
    dist = None
    if world > 1:
        import torch.distributed as dist
        dist.init_process_group("gloo")
    scene = Scene.load(SCENE)
    b = K.Backend(local)
    b.load(scene)
    t0 = time.perf_counter()
    b.build(**BUILD)
    build_s = time.perf_counter() - t0
    stats_world = b.world_stats()
    seed = int(scene.render["seed"])
    for k in range(args.warmup):
        b.render(WIDTH, HEIGHT, SPP, surfaces=SURFACES, seed=seed + 1000 + k, denoise=DENOISE)
    if dist:
        dist.barrier()
    device_ms, trace_ms, launches, march, program, segments, longest, capped, trace_launches = 0.0, 0.0, 0, 0, 0, 0, 0, 0, 0
    with Clocks(local) as clocks:
        wall0 = time.perf_counter()
        for k in range(args.steps):
            b.flush_l2()
            b.render(WIDTH, HEIGHT, SPP, surfaces=SURFACES, seed=seed + k, denoise=DENOISE)
            st = b.frame_stats()
            device_ms += st.total_ms
            trace_ms += st.trace_ms
            launches += st.launches
            march += st.march_steps
            program += st.program_steps
            segments += st.segments
            longest = max(longest, st.longest_march)
            capped += st.capped_rays
            trace_launches += st.trace_launches
        wall = time.perf_counter() - wall0
    if dist:
        t = np.array([device_ms])
        import torch
        tt = torch.tensor(t)
        dist.all_reduce(tt, op=dist.ReduceOp.MAX)
        device_ms = float(tt[0])
    samples = WIDTH * HEIGHT * SPP * args.steps
    value = samples * world / (device_ms / 1e3) / 1e6

    # e2e: as a host caller drives a frame through the C ABI
    blocks = K.scene_blocks(scene)
    per_frame = ["shot.camera", "lighting.lights", "lighting.sky", "looks.materials", "transport.finishes"]
    h2d = sum(blocks[n].nbytes for n in per_frame if n in blocks)
    d2h = WIDTH * HEIGHT * 3 * 4
    if dist:
        dist.barrier()
    e0 = time.perf_counter()
    for k in range(args.steps):
        for n in per_frame:
            if n in blocks:
                b.upload(n, blocks[n])
        img = b.render(WIDTH, HEIGHT, SPP, surfaces=SURFACES, seed=seed + k, denoise=DENOISE)
    e_dt = time.perf_counter() - e0
    e2e = samples * world / e_dt / 1e6

    # roofline of the dominant kernel, the sphere-trace kernel (72% of the
    # frame's launch time): FP32 issue.  Its lane instructions a second are
    # the march-form program steps it ran in the timed frames, counted live,
    # times the lane instructions a step, over the frames' device time (its
    # launches on the four render lanes overlap and cover the frame); the
    # peak is every SM's 128 FP32 lanes at the SM clock sampled meanwhile.
    rays_per_launch = segments / trace_launches if trace_launches else None
    clock_summary = clocks.summary()
    sm_hz = (clock_summary.get("sm_mhz") or 2070.0) * 1e6
    lane_inst_per_s = program * TRACE_LANE_INST_PER_PROGRAM_STEP / (device_ms / 1e3) if device_ms else None
    issue_peak = SM_COUNT * LANES_PER_SM * sm_hz
    line = {
        "metric": METRIC, "value": value, "unit": "Msamples/s", "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": device_ms / args.steps, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
        "data": "synthetic (seeded config-2 scene compiled by the reference renderer)",
        "config": {"workload": WORKLOAD + ("" if DENOISE else " (off)"),
                   "world": stats_world, "build_s": build_s, "l2": "512 MiB written before every timed frame",
                   "octree": "this backend's cut octree at min depth 7, max depth 11, cells split while their programs pass 32 steps; "
                             "config 2's 'octree depth 9' names the reference's packed 64-tree, another structure whose depths do not map one to one",
                   "parallelism": f"replicas x{world}"},
        "e2e": {"value": e2e, "unit": "Msamples/s", "h2d_bytes_per_step": int(h2d), "d2h_bytes_per_step": int(d2h)},
        "gpu_launches": int(launches),
        "clocks": clock_summary,
        "wall_s": wall,
        "march_steps_per_sample": march / samples,
        "segments_per_sample": segments / samples,
        "longest_march": int(longest),
        "capped_rays": int(capped),
        "program_steps_per_sample": program / samples,
        # trace launch time summed over both lanes' streams / frame time:
        # above 1 where the lanes' trace launches overlap
        "trace_share": trace_ms / device_ms if device_ms else None,
    }
    if rank == 0:
        line["roofline"] = {
            "bound": "fp32-issue", "achieved": lane_inst_per_s / 1e12 if lane_inst_per_s else None, "peak": issue_peak / 1e12,
            "unit": "Tlane-inst/s", "frac": lane_inst_per_s / issue_peak if lane_inst_per_s else None,
            "traffic": None,
            "kernel": "traceKernel", "peak_source": f"computed: {SM_COUNT} SMs x {LANES_PER_SM} FP32 lanes x the sampled SM clock",
            "warp_efficiency": TRACE_WARP_EFFICIENCY,
            "algorithmic": f"{program / max(1, segments):.0f} march-form program steps a ray x {TRACE_LANE_INST_PER_PROGRAM_STEP} lane instructions a step (ncu); "
                           f"{rays_per_launch:.0f} rays a launch" if rays_per_launch else None,
            "note": "traffic: none against this roof (the kernel's DRAM bytes, from an ncu capture of one launch, are in the trace kernel's "
                    "profile); the kernel issues at ~13 of 32 lanes (warp_efficiency), so its issue slots bind long before its FP32 lanes",
        }
        # over the frame's device time: the two render lanes' trace
        # launches overlap, so their summed launch time exceeds it
        line["trace_rates"] = {
            "rays_per_s": segments / (device_ms / 1e3) if device_ms else None,
            "program_steps_per_s": program / (device_ms / 1e3) if device_ms else None,
            "march_steps_per_s": march / (device_ms / 1e3) if device_ms else None,
        }
        if args.no_cpu:
            line["cpu_baseline"] = None
        else:
            try:
                line["cpu_baseline"] = cpu_baseline(scene)
            except Exception as e:  # the oracle is test infrastructure; report why it could not run
                line["cpu_baseline"] = {"value": None, "unit": "Msamples/s", "cores": os.cpu_count(), "kind": "port", "sample": f"failed: {e}"}
        if not (args.no_cpu or args.no_guide):
            try:
                line["guided"] = guided(local)
            except Exception as e:  # report why the guided run could not finish
                line["guided"] = {"failed": str(e)}
        if not (args.no_cpu or args.no_serve):
            try:
                line["serving"] = serving(b)
            except Exception as e:  # report why the serving run could not finish
                line["serving"] = {"failed": str(e)}
        print(json.dumps(line), flush=True)
    b.close()
    if dist:
        dist.destroy_process_group()


# The learned-guide run (config 4's scene: the config-1 primitives in a
# closed room lit through a 5% aperture) at 1920x1080: plain BSDF sampling
# against the learned guide at equal wall time, training included, in
# relative MSE against a plain frame of 512 spp (8x the plain frame's: its
# own noise adds about an eighth of the plain frame's relMSE to both
# figures).  The guide is config 4's (2^19 entries a level, Adam lr 1e-2,
# trained on the first 8 spp: one training frame of 8 spp).
GUIDE_SCENE = os.path.join(ROOT, "tests", "golden", "scenes", "room.npz")
GUIDE_W, GUIDE_H, GUIDE_SURFACES, GUIDE_REF_SPP, GUIDE_PLAIN_SPP, GUIDE_TRAIN_SPP = 1920, 1080, 8, 512, 64, 8
PROFILE_W, PROFILE_H = 480, 270


def guided(device: int) -> dict:
    import kodanuki_gb300 as K
    from kodanuki_gb300.scene import Scene

    sc = Scene.load(GUIDE_SCENE)

    def rel(img, ref):
        return float(np.mean((img - ref) ** 2 / (ref ** 2 + 0.01)))

    def timed(fn):
        t0 = time.perf_counter()
        out = fn()
        return out, time.perf_counter() - t0

    with K.Backend(device) as b:
        b.load(sc)
        b.build(5, 10, 64)
        b.render(GUIDE_W, GUIDE_H, 4, surfaces=GUIDE_SURFACES, seed=9)  # warm-up
        ref, ref_s = timed(lambda: b.render(GUIDE_W, GUIDE_H, GUIDE_REF_SPP, surfaces=GUIDE_SURFACES, seed=101))
        plain, plain_s = timed(lambda: b.render(GUIDE_W, GUIDE_H, GUIDE_PLAIN_SPP, surfaces=GUIDE_SURFACES, seed=7))
        lo = np.asarray(sc.region_lower, np.float64)
        hi = lo + np.asarray(sc.region_size, np.float64)
        with K.Guide(device, table_log2=19, seed=2, region=(lo, hi), learning_rate=1e-2, batch=16384, max_steps=256) as g:
            b.set_guide(g, 0.5, K.GUIDE_TRAIN)
            t0 = time.perf_counter()
            b.render(GUIDE_W, GUIDE_H, GUIDE_TRAIN_SPP, surfaces=GUIDE_SURFACES, seed=2000)
            train_s = time.perf_counter() - t0
            b.set_guide(g, 0.5, K.GUIDE_SAMPLE)
            b.render(GUIDE_W, GUIDE_H, 1, surfaces=GUIDE_SURFACES, seed=4)  # the guided path's buffers, allocated once
            _, pilot_s = timed(lambda: b.render(GUIDE_W, GUIDE_H, 8, surfaces=GUIDE_SURFACES, seed=3))
            spp = max(1, int((plain_s - train_s) / (pilot_s / 8)))
            img, guided_s = timed(lambda: b.render(GUIDE_W, GUIDE_H, spp, surfaces=GUIDE_SURFACES, seed=7))
            # equal samples too, to separate the sampling gain from the cost
            same, _ = timed(lambda: b.render(GUIDE_W, GUIDE_H, GUIDE_PLAIN_SPP, surfaces=GUIDE_SURFACES, seed=7))
            # the fallback: pilot frames (the frame's own size, 4 spp) keep the
            # guide's sampling only where it costs less at equal time; a pilot
            # of another size misjudges it, since a frame's time per sample
            # depends on its size
            (keep, plain_cost, guided_cost), select_s = timed(lambda: b.guide_select(GUIDE_W, GUIDE_H, 4, surfaces=GUIDE_SURFACES, seed=41))
            b.set_guide(None)
            # the network's kernels alone: a training step and a query launch
            rng = np.random.default_rng(5)
            n = 1 << 16
            p = rng.uniform(lo, hi, size=(n, 3))
            nv = rng.normal(size=(n, 3))
            nv /= np.linalg.norm(nv, axis=1, keepdims=True)
            d = rng.normal(size=(n, 3))
            d /= np.linalg.norm(d, axis=1, keepdims=True)
            samples = np.concatenate([p, nv, d, np.ones((n, 1))], axis=1).astype(np.float32)
            g.train(samples, batch=16384, steps=4)
            _, t_train = timed(lambda: g.train(samples, batch=16384, steps=64))
            rows = samples[:, :6].copy()
            g.query(rows)
            _, t_query = timed(lambda: g.query(rows))
    rp, rg, rs = rel(plain, ref), rel(img, ref), rel(same, ref)
    flops = 2 * (48 * 64 + 64 * 64 * 2 + 64 * 48)  # a sample's forward pass
    return {
        "workload": f"config-4 room scene (64 primitives in a closed room, 5% aperture), {GUIDE_W}x{GUIDE_H}, {GUIDE_SURFACES} surfaces; "
                    f"reference {GUIDE_REF_SPP} spp plain",
        "reference_s": ref_s,
        "plain": {"spp": GUIDE_PLAIN_SPP, "seconds": plain_s, "relmse": rp},
        "guided": {"train_spp": GUIDE_TRAIN_SPP, "train_s": train_s, "spp": spp, "seconds": train_s + guided_s, "relmse": rg,
                   "seconds_per_spp": pilot_s / 8, "plain_seconds_per_spp": plain_s / GUIDE_PLAIN_SPP},
        "select": {"kept_guide": keep, "plain_cost": plain_cost, "guided_cost": guided_cost, "seconds": select_s,
                   "pilot": f"pairs of plain and guided frames of {GUIDE_W}x{GUIDE_H} at 4 spp, 3 to 16 pairs (until the cost ratio is 2 standard errors from a 5% margin), after one untimed frame of each"},
        "equal_time_gain": rp / rg if rg > 0 else None,
        "equal_spp_gain": rp / rs if rs > 0 else None,
        "train_samples_per_s": 64 * 16384 / t_train,
        "train_tflops": 3 * flops * 64 * 16384 / t_train / 1e12,
        "query_rows_per_s": n / t_query,
        "note": "train and query rates are host-timed around whole calls (with copies); the network is 3 x 64 wide, so its tensor work is small beside the encoding's gathers",
    }


STRESS_SCENE = os.path.join(ROOT, "tests", "golden", "scenes", "c5.npz")
STRESS_W, STRESS_H, STRESS_SPP, STRESS_SURFACES = 3840, 2160, 256, 32


def stress(device: int) -> dict:
    """Config 5, the stress configuration: the 65536-box city with its
    dispersive sphere cluster at 3840x2160, 256 spp, 32 surfaces, on the
    octree the benchmark builds at depth 11; then learned guiding on it;
    then 4 progressive 1-spp sessions of it served alongside config-2
    batch frames.  Device times from the frames' CUDA events."""
    import kodanuki_gb300 as K
    from kodanuki_gb300.scene import Scene
    sc = Scene.load(STRESS_SCENE)
    out = {"workload": f"config 5: {sc.program_count} objects (a 256 x 256 city of rounded boxes, heights 0.4 LogNormal(0, 0.5), "
                       f"24 dispersive glass spheres), {STRESS_W}x{STRESS_H}, {STRESS_SPP} spp, {STRESS_SURFACES} surfaces, FP32"}
    with K.Backend(device) as b:
        b.load(sc)
        t0 = time.perf_counter()
        b.build(7, 11, 32)
        out["build_s"] = time.perf_counter() - t0
        out["world"] = b.world_stats()
        b.render(STRESS_W, STRESS_H, 1, surfaces=STRESS_SURFACES, seed=9)  # warm-up
        b.render(STRESS_W, STRESS_H, STRESS_SPP, surfaces=STRESS_SURFACES, seed=1)
        st = b.frame_stats()
        out["plain"] = {"ms": st.total_ms, "msamples_per_s": STRESS_W * STRESS_H * STRESS_SPP / st.total_ms / 1e3,
                        "capped_rays": int(st.capped_rays), "longest_march": int(st.longest_march)}
        lo = np.asarray(sc.region_lower, np.float64)
        hi = lo + np.asarray(sc.region_size, np.float64)
        with K.Guide(device, table_log2=19, seed=2, region=(lo, hi), learning_rate=1e-2, batch=16384, max_steps=256) as g:
            b.set_guide(g, 0.5, K.GUIDE_TRAIN)
            b.render(STRESS_W, STRESS_H, 8, surfaces=STRESS_SURFACES, seed=2000)
            train_ms = b.frame_stats().total_ms
            b.set_guide(g, 0.5, K.GUIDE_SAMPLE)
            b.render(STRESS_W, STRESS_H, 1, surfaces=STRESS_SURFACES, seed=4)
            b.render(STRESS_W, STRESS_H, 64, surfaces=STRESS_SURFACES, seed=3)
            guided_ms = b.frame_stats().total_ms
            b.set_guide(None)
        out["guided"] = {"train_spp": 8, "train_ms": train_ms, "spp": 64, "ms": guided_ms,
                         "msamples_per_s": STRESS_W * STRESS_H * 64 / guided_ms / 1e3}
        # served: 4 progressive 1-spp sessions of the city, 8 frames each,
        # beside config-2 batch frames (1080p, 64 spp)
        with K.Backend(device) as c2:
            c2.load(Scene.load(SCENE))
            c2.build(7, 11, 32)
            srv = K.Server(device, slots=8)
            city, batch = srv.add_scene(b), srv.add_scene(c2)
            warm = [srv.submit(city, STRESS_W, STRESS_H, 1, surfaces=STRESS_SURFACES, seed=5 + k, denoise=True, interactive=True, session=k + 1)
                    for k in range(4)]
            warm.append(srv.submit(batch, 640, 480, 1, surfaces=16, seed=1))
            for t in warm:
                srv.wait(t)
            srv.reset_latency()
            t0 = time.perf_counter()
            jobs = [srv.submit(batch, 1920, 1080, 64, surfaces=16, seed=100 + k) for k in range(3)]
            frames = 0
            for _ in range(8):
                tickets = [srv.submit(city, STRESS_W, STRESS_H, 1, surfaces=STRESS_SURFACES, seed=5 + k, denoise=True, interactive=True, session=k + 1)
                           for k in range(4)]
                for t in tickets:
                    frames += int(srv.wait(t)[0] == K.KDN_OK)
            done = sum(int(srv.wait(t)[0] == K.KDN_OK) for t in jobs)
            wall = time.perf_counter() - t0
            inter = srv.latency(True)
            for k in range(4):
                srv.end_session(k + 1)
            srv.close()
        out["served"] = {"sessions": 4, "session_frames": frames, "batch_frames": done, "wall_s": wall,
                         "interactive_4k_1spp_ms": {"p50": inter["p50_ms"], "p99": inter["p99_ms"], "count": inter["count"]},
                         "note": "each round submits the four sessions' next frames and waits for them; three config-2 batch frames run beside"}
    return out


def guide_profile(device: int) -> None:
    """Two training frames (each ends in Adam steps of 16384 samples) and one
    guided frame of the room scene at PROFILE_W x PROFILE_H: a short run for profilers."""
    import kodanuki_gb300 as K
    from kodanuki_gb300.scene import Scene

    sc = Scene.load(GUIDE_SCENE)
    with K.Backend(device) as b:
        b.load(sc)
        b.build(5, 10, 64)
        lo = np.asarray(sc.region_lower, np.float64)
        hi = lo + np.asarray(sc.region_size, np.float64)
        with K.Guide(device, table_log2=19, seed=2, region=(lo, hi), batch=16384, max_steps=16) as g:
            b.set_guide(g, 0.5, K.GUIDE_TRAIN)
            t0 = time.perf_counter()
            for k in range(2):
                b.render(PROFILE_W, PROFILE_H, 1, surfaces=GUIDE_SURFACES, seed=2000 + k)
            train_s = time.perf_counter() - t0
            b.set_guide(g, 0.5, K.GUIDE_SAMPLE)
            t0 = time.perf_counter()
            img = b.render(PROFILE_W, PROFILE_H, 4, surfaces=GUIDE_SURFACES, seed=7)
            guided_s = time.perf_counter() - t0
            b.set_guide(None)
    print(json.dumps({"guide_profile": True, "train_s": train_s, "guided_s": guided_s, "finite": bool(np.isfinite(img).all())}), flush=True)


# The serving run (config 3, bounded): Poisson arrivals at 200 requests a
# second over eight resident seeded scenes of 256 to 16384 config-1-style
# primitives for a fixed window; 70% single frames of a uniform resolution in
# {320x240, 640x480, 1280x720, 1920x1080} and spp in {1, 4, 16, 64}, 30%
# frames of four progressive 1280x720 sessions at 1 spp with the denoiser's
# history (interactive).  What is still queued when the window closes is
# cancelled; latency is over the completed requests.
SERVE_SCENES = [f"serve_{n}" for n in (256, 512, 1024, 2048, 4096, 6144, 10240, 16384)]
SERVE_RATE, SERVE_WINDOW_S, SERVE_SLOTS, SERVE_SESSIONS = 200.0, 5.0, 8, 4
SERVE_SIZES = [(320, 240), (640, 480), (1280, 720), (1920, 1080)]
SERVE_SPP = [1, 4, 16, 64]


def serving(main_backend, **options) -> dict:
    import kodanuki_gb300 as K
    from kodanuki_gb300.scene import Scene
    rng = np.random.default_rng(2024)
    backends = []
    for name in SERVE_SCENES:
        b = K.Backend(0)
        b.load(Scene.load(os.path.join(ROOT, "tests", "golden", "scenes", name + ".npz")))
        b.build(min_depth=6, max_depth=10, split_steps=64)
        backends.append(b)
    srv = K.Server(0, slots=options.pop("slots", SERVE_SLOTS), **options)
    ids = [srv.add_scene(b) for b in backends]
    session_scene = [ids[k % len(ids)] for k in range(SERVE_SESSIONS)]
    # warm-up (not counted): each session's first frame and a frame of each
    # scene, which open the contexts and their buffers
    warm = [srv.submit(session_scene[k], 1280, 720, 1, surfaces=8, seed=7 + k, denoise=True, interactive=True, session=k + 1) for k in range(SERVE_SESSIONS)]
    warm += [srv.submit(i, 640, 480, 1, surfaces=8, seed=1) for i in ids]
    for t in warm:
        srv.wait(t)
    srv.reset_latency()
    tickets, kinds = [], []
    t0 = time.perf_counter()
    next_at = 0.0
    samples_of = {}
    while True:
        next_at += rng.exponential(1.0 / SERVE_RATE)
        if next_at > SERVE_WINDOW_S:
            break
        delay = t0 + next_at - time.perf_counter()
        if delay > 0:
            time.sleep(delay)
        if rng.random() < 0.3:
            k = int(rng.integers(SERVE_SESSIONS))
            t = srv.submit(session_scene[k], 1280, 720, 1, surfaces=8, seed=7 + k, denoise=True, interactive=True, session=k + 1)
            kinds.append("interactive")
            samples_of[t] = 1280 * 720
        else:
            w, h = SERVE_SIZES[int(rng.integers(4))]
            spp = SERVE_SPP[int(rng.integers(4))]
            t = srv.submit(ids[int(rng.integers(len(ids)))], w, h, spp, surfaces=8, seed=int(rng.integers(1 << 30)))
            kinds.append("batch")
            samples_of[t] = w * h * spp
        tickets.append(t)
    cancelled = srv.cancel_queued()
    done_samples, completed, statuses = 0, {"interactive": 0, "batch": 0}, []
    for t, kind in zip(tickets, kinds):
        st, served, _ = srv.wait(t)
        statuses.append(st)
        if st == K.KDN_OK:
            completed[kind] += 1
            done_samples += samples_of[t]
    wall = time.perf_counter() - t0
    inter, every = srv.latency(True), srv.latency(False)
    for k in range(SERVE_SESSIONS):
        try:
            srv.end_session(k + 1)
        except K.KdnError:
            pass
    srv.close()
    for b in backends:
        b.close()
    return {
        "workload": f"config 3: Poisson {SERVE_RATE:.0f}/s for {SERVE_WINDOW_S:.0f} s over {len(ids)} resident scenes of 256 to 16384 primitives ({', '.join(SERVE_SCENES)}); "
                    f"70% frames of {{320x240,640x480,1280x720,1920x1080}} x {{1,4,16,64}} spp, 30% frames of {SERVE_SESSIONS} progressive "
                    f"1280x720 1-spp denoised interactive sessions; {SERVE_SLOTS} slots, 120 GB budget; queued requests cancelled at the window's end",
        "submitted": len(tickets), "completed": completed, "cancelled": int(cancelled),
        "failed": int(sum(1 for st in statuses if st not in (K.KDN_OK, K.KDN_NOT_READY))),
        "msamples_per_s": done_samples / wall / 1e6, "wall_s": wall,
        "interactive_720p_1spp_ms": {"p50": inter["p50_ms"], "p99": inter["p99_ms"], "count": inter["count"]},
        "all_ms": {"p50": every["p50_ms"], "p99": every["p99_ms"], "count": every["count"]},
    }


def main() -> None:
    global WIDTH, HEIGHT, SPP
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="gb300", choices=["gb300", "reference"])
    ap.add_argument("--width", type=int, default=WIDTH, help="a smaller frame for profiling captures only")
    ap.add_argument("--height", type=int, default=HEIGHT)
    ap.add_argument("--spp", type=int, default=SPP)
    ap.add_argument("--no-cpu", action="store_true", help="leave out the CPU baseline and the serving run (profiling captures)")
    ap.add_argument("--no-serve", action="store_true", help="leave out the serving run")
    ap.add_argument("--no-guide", action="store_true", help="leave out the learned-guide run")
    ap.add_argument("--guide-profile", action="store_true", help="a short learned-guide run alone (profiling captures): two training frames and one guided frame of the room scene")
    ap.add_argument("--stress", action="store_true", help="config 5 alone (the 65536-box city at 3840x2160, 256 spp, guided, served): one JSON line, a few minutes")
    args = ap.parse_args()
    WIDTH, HEIGHT, SPP = args.width, args.height, args.spp
    if args.impl == "reference":
        run_reference(args)
    elif args.guide_profile:
        guide_profile(env_int("LOCAL_RANK", 0))
    elif args.stress:
        print(json.dumps(stress(env_int("LOCAL_RANK", 0))), flush=True)
    else:
        run_gpu(args)


if __name__ == "__main__":
    main()
