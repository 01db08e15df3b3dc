"""Benchmark: ms/frame of the XPBD substep at 535k tets (synthetic humanV2 scene).

Workload: rlmusclev2_b200/configs/humanv2_synth.json -- 40 ellipsoidal
muscles + fascia shell (~129k verts / ~535k tets), 20 moving capsule bones,
ARAP-SVD + belly attach + tendon pins + aniso_arap on one muscle, 256^3 bone
SDF push-out, 10 substeps x 20 Jacobi iterations per frame, FP32.  A step is
one frame.  Inputs of every frame (bone poses, activation) are seeded
synthetic data.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

Prints one JSON line (rank 0).  ``value`` is device time per frame with the
frame inputs already on the GPU (CUDA events on the engine stream, max over
ranks); ``e2e`` is the same frame through the public API (host activation and
bone poses uploaded, positions read back every frame).  Multi-GPU runs are
independent replicas (the single-mesh path does not shard).
"""
from __future__ import annotations

import argparse
import json
import os
import subprocess
import sys
import threading
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))
CONFIGS = {
    "humanv2": (ROOT / "rlmusclev2_b200" / "configs" / "humanv2_synth.json",
                "humanv2_synth_535k_tets (10 substeps x 20 Jacobi iterations, SDF push-out)"),
    "humanv2_mg_dcd": (ROOT / "rlmusclev2_b200" / "configs" / "humanv2_synth_mg_dcd.json",
                       "humanv2_synth_535k_tets + 2-level multigrid (2 coarse + 1 fine iterations) + tri-tri DCD "
                       "with per-substep LBVH + SNH fascia"),
}
CONFIGS["batched"] = (ROOT / "rlmusclev2_b200" / "configs" / "batched_256.json",
                      "batched_256_box_muscles_3.5M_tets (256 independent instances, per-instance 64^3 SDF and "
                      "activation schedule, 10 substeps x 1 Jacobi iteration)")
CONFIGS["learned"] = (ROOT / "rlmusclev2_b200" / "configs" / "humanv2_synth_mg_dcd.json",
                      "humanv2_synth_535k_tets, config-3 mesh and cage, learned coarse warm start + 10 Jacobi "
                      "iterations per substep vs the plain solver at 20 (no DCD)")
CONFIGS["box"] = (None, "box_muscle_8x8x32_12288_tets (ARAP-SVD + volume, 10 substeps x 1 Jacobi iteration, "
                         "gravity, 5 % end pins)")
CONFIG = CONFIGS["humanv2"][0]
PEAKS = ROOT / "MEASURED_PEAKS.json"
TRAFFIC = ROOT / "profiles" / "ncu_traffic.json"
FALLBACK_HBM_GBS = 6650.0
WORKLOAD = CONFIGS["humanv2"][1]


def _peak_hbm():
    try:
        return float(json.loads(PEAKS.read_text())["hbm_gbs"]), "measured"
    except Exception:
        return FALLBACK_HBM_GBS, "fallback"


class ClockSampler:
    """SM clocks and throttle reasons sampled during the timed region, through
    NVML every 10 ms (nvidia-smi every 200 ms when NVML is unavailable).
    Reading only: no clock, power or mode setting is touched."""

    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.hw_slowdown,"
         "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
         "clocks_event_reasons.sw_power_cap")
    # NVML clocks-event reason bits
    BITS = {"sw_power_cap": 0x4, "hw_slowdown": 0x8, "sw_thermal_slowdown": 0x20, "hw_thermal_slowdown": 0x40}

    def __init__(self, gpu_index: int):
        vis = os.environ.get("CUDA_VISIBLE_DEVICES", "")
        ids = [x.strip() for x in vis.split(",") if x.strip()]
        self.idx = int(ids[gpu_index]) if gpu_index < len(ids) and ids[gpu_index].isdigit() else gpu_index
        self.rows = []
        self._stop = threading.Event()
        self._t = None
        self._nvml = None
        try:
            import pynvml
            pynvml.nvmlInit()
            self._h = pynvml.nvmlDeviceGetHandleByIndex(self.idx)
            self._nvml = pynvml
        except Exception:
            self._nvml = None

    def _sample_nvml(self):
        nv = self._nvml
        sm = nv.nvmlDeviceGetClockInfo(self._h, nv.NVML_CLOCK_SM)
        mx = nv.nvmlDeviceGetMaxClockInfo(self._h, nv.NVML_CLOCK_SM)
        try:
            r = nv.nvmlDeviceGetCurrentClocksEventReasons(self._h)
        except Exception:
            r = nv.nvmlDeviceGetCurrentClocksThrottleReasons(self._h)
        act = ["Active" if r & self.BITS[k] else "Not Active"
               for k in ("hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap")]
        self.rows.append([str(self.idx), str(sm), str(mx), ""] + act)

    def _run(self):
        while not self._stop.is_set():
            try:
                if self._nvml is not None:
                    self._sample_nvml()
                else:
                    out = subprocess.run(["nvidia-smi", f"--id={self.idx}", f"--query-gpu={self.Q}",
                                          "--format=csv,noheader,nounits"], capture_output=True, text=True, timeout=5)
                    for line in out.stdout.strip().splitlines():
                        self.rows.append([x.strip() for x in line.split(",")])
            except Exception:
                pass
            self._stop.wait(0.01 if self._nvml is not None else 0.2)

    def __enter__(self):
        self._t = threading.Thread(target=self._run, daemon=True)
        self._t.start()
        return self

    def __exit__(self, *a):
        self._stop.set()
        self._t.join(timeout=10)

    def summary(self):
        if not self.rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
        sm = [float(r[1]) for r in self.rows if r[1].replace(".", "").isdigit()]
        mx = [float(r[2]) for r in self.rows if r[2].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[k] for r in self.rows for k in range(4) if len(r) > 4 + k and r[4 + k] == "Active"})
        return {"sm_mhz": float(np.median(sm)) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": reasons, "samples": len(self.rows),
                "source": "nvml" if self._nvml is not None else "nvidia-smi"}


class CpuBaseline:
    """The CPU oracle stepping whole frames of the benchmark's program
    (OracleMultiGridSim.step_frame, the reference's MultiGridSim frame
    mg.py:1322-1418 restated in C with OpenMP over all host threads): bone
    targets and belly-attach targets, the 256^3 SDF bake, the hard pin, then
    per substep the prediction, the Jacobi iterations (every constraint, the
    averaged apply and the re-pin after each), the SDF push-out and the
    velocity update.  The same frames and inputs as the GPU arm."""

    def __init__(self, cfg, scene, batched: bool = False):
        from oracle import oracle as O
        self.orc = (O.OracleBatchSim if batched else O.OracleMultiGridSim)(cfg, scene, prec="f32")
        self.frame = int(cfg.get("start_frame", 1))
        self.n_iter = int(cfg["nsubsteps"]) * int(cfg["fine_iterations"])
        self.nsub = int(cfg["nsubsteps"])
        self.n_tets = int(scene.tets.shape[0])

    def frame_ms(self) -> float:
        """One whole frame (the next frame of the sequence), wall time in ms."""
        t0 = time.perf_counter()
        self.orc.step_frame(self.frame)
        self.frame += 1
        return (time.perf_counter() - t0) * 1e3

    def run(self, warmup: int, steps: int) -> float:
        for _ in range(warmup):
            self.frame_ms()
        self.times = [self.frame_ms() for _ in range(steps)]
        return float(np.mean(self.times))

    def describe(self, value: float, warmup: int, steps: int) -> dict:
        return {"value": round(value, 3), "unit": "ms/frame", "cores": _omp_threads(), "kind": "port",
                "sample": f"{steps} whole frame(s) after {warmup} untimed, mean wall time: the {self.n_tets}-tet "
                          f"mesh through the FP32 oracle's frame program (targets, SDF bake, pins, "
                          f"{self.nsub} substeps x {self.n_iter // self.nsub} Jacobi iterations, push-out, "
                          f"velocities)"}


def _omp_threads() -> int:
    v = os.environ.get("OMP_NUM_THREADS")
    return int(v) if v else (os.cpu_count() or 1)


def _dist_setup():
    import torch
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if world > 1:
        import datetime
        import torch.distributed as dist
        torch.cuda.set_device(local)
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120))
    return world, rank, local


def run_reference(args):
    """The reference arm: the oracle's restatement of the reference's CPU
    path (the reference itself runs on NVIDIA Warp, which cannot be installed
    here), whole frames of the benchmark workload, rank 0 only."""
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return 0
    from rlmusclev2_b200.mg import load_config, scene_from_cfg
    steps = max(1, args.steps)
    if args.config == "learned":
        print(json.dumps({"impl": "reference", "unavailable": "the learned warm start has no counterpart in the "
                          "reference (it replaces the V-cycle warm start); time --config humanv2_mg_dcd instead"}))
        return 0
    if args.config == "box":
        return _run_reference_box(args, world, steps)
    cfg = load_config(str(CONFIG))
    scene = scene_from_cfg(cfg)
    cb = CpuBaseline(cfg, scene, batched=args.config == "batched")
    v = cb.run(args.warmup, steps)
    line = {"impl": "reference", "metric": "ms/frame", "value": round(v, 3), "unit": "ms/frame", "n_gpus": world,
            "steps": steps, "warmup": args.warmup, "ms_per_step": round(v, 3), "higher_is_better": False,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
            "config": {"workload": WORKLOAD, "n_verts": int(scene.verts.shape[0]), "n_tets": int(scene.tets.shape[0])},
            "cpu_baseline": cb.describe(v, args.warmup, steps),
            "e2e": {"value": round(v, 3), "unit": "ms/frame", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
            "note": "the reference runs on NVIDIA Warp (warp-lang 1.13.0), which is not installable offline here; "
                    "its CPU path is restated by the C oracle (OpenMP) and timed on whole frames"}
    print(json.dumps(line), flush=True)
    return 0


def _run_reference_box(args, world, steps):
    """Reference arm of the box muscle: the FP32 oracle's MuscleSim program
    (musclesim.py:107-142), whole frames."""
    from oracle import oracle as O
    from rlmusclev2_b200.meshgen import box_muscle
    m = box_muscle()
    cons = [{"type": "tetarapsvd", "name": "arap", "compliance": 1e-7},
            {"type": "volume", "name": "volume", "compliance": 0.0}]
    orc = O.OracleMuscleSim(m.verts, m.tets, m.fiber_per_tet, constraint_configs=cons, stopped=m.stopped,
                            dts=1.0 / 24.0, num_substeps=10, density=1060.0, veldamping=0.02, gravity=-9.8, prec="f32")
    for _ in range(args.warmup):
        orc.step()
    ts = []
    for _ in range(steps):
        t0 = time.perf_counter()
        orc.step()
        ts.append((time.perf_counter() - t0) * 1e3)
    v = float(np.mean(ts))
    cb = {"value": round(v, 3), "unit": "ms/frame", "cores": _omp_threads(), "kind": "port",
          "sample": f"{steps} whole frame(s) after {args.warmup} untimed: the 12,288-tet box through the FP32 oracle's "
                    "MuscleSim program (10 substeps x 1 Jacobi iteration)"}
    line = {"impl": "reference", "metric": "ms/frame", "value": round(v, 3), "unit": "ms/frame", "n_gpus": world,
            "steps": steps, "warmup": args.warmup, "ms_per_step": round(v, 3), "higher_is_better": False,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
            "config": {"workload": WORKLOAD, "n_verts": int(m.verts.shape[0]), "n_tets": int(m.tets.shape[0])},
            "cpu_baseline": cb,
            "e2e": {"value": round(v, 3), "unit": "ms/frame", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)
    return 0


def run_ours(args):
    import ctypes as C
    import torch

    from rlmusclev2_b200 import _capi as capi
    from rlmusclev2_b200.mg import MultiGridSim, load_config

    world, rank, local = _dist_setup()
    torch.cuda.set_device(local)
    cfg = load_config(str(CONFIG))
    batched = args.config == "batched"
    tuned = None
    if batched:
        # instances sharded over the ranks by tet count (no collective on the data path)
        from rlmusclev2_b200.batch import BatchSim
        sim = BatchSim(cfg, device=f"cuda:{local}", shard=(rank, world) if world > 1 else None)
        sim.step_frame_inputs(sim.start_frame)
        tuned = sim.autotune()
        n_inst_total = int(sim.n_inst)
        if world > 1:
            t = torch.tensor([n_inst_total], device=sim.device)
            torch.distributed.all_reduce(t)
            n_inst_total = int(t.item())
    else:
        sim = MultiGridSim(cfg, device=f"cuda:{local}")
    sc = sim.scene
    nf = args.warmup + args.steps
    frames = [sim.start_frame + f for f in range(nf)]
    stream = sim._stream
    ev = lambda: torch.cuda.Event(enable_timing=True)  # noqa: E731

    # ---- device-resident inputs: all frames' bone poses and activations on the GPU
    trs = torch.from_numpy(np.stack([sc.bone_transforms(f).reshape(sc.n_bones, 12) for f in frames]).astype(
        np.float32)).to(sim.device)
    if batched:
        acts_src = torch.from_numpy(np.stack([sc.instance_activation(f) for f in frames])).to(sim.device)
        act_idx, act_n = sim._tet_inst_lib, sim.NT
    else:
        acts_src = torch.from_numpy(np.stack([sc.activation(f) for f in frames])).to(sim.device)
        act_idx, act_n = sim._tet_perm_d, sim.NT

    def frame_resident(i):
        with torch.cuda.stream(stream):
            sim._bone_tr.copy_(trs[i])
        capi.check(sim._lib.xpbd_gather(act_n, 1, C.c_void_p(act_idx.data_ptr()),
                                        C.c_void_p(acts_src[i].data_ptr()), 1, C.c_void_p(sim._t_act.data_ptr()), 1,
                                        sim._sp))
        sim._frame_loaded = frames[i]
        sim.step_frame(frames[i])

    flush = torch.empty(64 * 1024 * 1024, dtype=torch.float32, device=sim.device)  # 256 MB > L2 (126 MB)

    def flush_l2():
        with torch.cuda.stream(stream):
            flush.zero_()

    for i in range(args.warmup):
        frame_resident(i)
    stream.synchronize()
    if world > 1:
        torch.distributed.barrier()
    evs = [(ev(), ev()) for _ in range(args.steps)]
    with ClockSampler(torch.cuda.current_device()) as clk:
        for k, i in enumerate(range(args.warmup, nf)):
            flush_l2()
            evs[k][0].record(stream)
            frame_resident(i)
            evs[k][1].record(stream)
        stream.synchronize()
    ms_frame = sum(a.elapsed_time(b) for a, b in evs) / args.steps
    if world > 1:
        t = torch.tensor([ms_frame], device=sim.device)
        torch.distributed.all_reduce(t, op=torch.distributed.ReduceOp.MAX)
        ms_frame = float(t.item())

    # ---- e2e through the public API: host inputs in, positions out, every frame.
    # The per-frame activations are generated before timing: they are the
    # caller's host buffers, not work of the simulator.
    acts = {f: (sc.instance_activation(f) if batched else sc.activation(f)) for f in frames}

    def set_act(f):
        if batched:
            sim.set_instance_activation(acts[f])
        else:
            sim.set_fiber_activation(acts[f])

    for i in range(min(args.warmup, 3)):
        set_act(frames[i])
        sim.step_frame(frames[i])
        sim.positions_np()
    stream.synchronize()
    if world > 1:
        torch.distributed.barrier()
    h2d = (sim.n_inst if batched else sim.NT) * 4 + sc.n_bones * 12 * 4
    d2h = sim.NV * 3 * 4
    evs2 = [(ev(), ev()) for _ in range(args.steps)]
    for k, i in enumerate(range(args.warmup, nf)):
        flush_l2()
        evs2[k][0].record(stream)
        set_act(frames[i])
        sim.step_frame(frames[i])
        _ = sim.positions_np()
        evs2[k][1].record(stream)
    stream.synchronize()
    ms_e2e = sum(a.elapsed_time(b) for a, b in evs2) / args.steps
    if world > 1:
        t = torch.tensor([ms_e2e], device=sim.device)
        torch.distributed.all_reduce(t, op=torch.distributed.ReduceOp.MAX)
        ms_e2e = float(t.item())

    # ---- roofline of the dominant kernel, measured inside a real frame: one
    # frame replayed launch by launch with events around its tet passes on the
    # engine stream (the launch of all substeps where the frame is one; else
    # every substep's iterations, or every iteration with its boundary finish).
    L = sim.layout
    flush_l2()
    frame_resident(nf - 1)
    iters = []
    sim._targets_kernel()
    sim.collision_solvers[0].bake() if sim.collision_solvers else None
    pin = capi.OP_PIN if sim._has_pins else 0
    vel = (0 if sim.quasi_static else capi.OP_VELOCITY) | (capi.OP_SDF if sim.collision_solvers else 0)
    whole = False
    if sim.mg is None and sim.fascia is None and not sim.n_m2m and not sim.collision_solvers_iter:
        if pin:
            sim._vstep(capi.OP_PIN)
        sim.apply_pintotarget_all()
        a, b = ev(), ev()
        a.record(stream)
        whole = sim._fused_substeps(sim.nsubsteps, sim.fine_iters, capi.OP_PREDICT | pin,
                                    capi.OP_PREDICT | pin | vel, vel)
        b.record(stream)
        if whole:
            iters.append((a, b, sim.nsubsteps * sim.fine_iters))
    for sub in range(0 if whole else sim.nsubsteps):
        sim._vstep(capi.OP_PREDICT | (capi.OP_PIN if sim._has_pins and sim.mg is None else 0))
        if sim.mg is not None:
            sim.mg.vcycle(pin_fine=sim._has_pins)
        if not sim.collision_solvers_iter:
            a, b = ev(), ev()
            a.record(stream)
            sim._jacobi_iterations(sim.fine_iters)
            b.record(stream)
            iters.append((a, b, sim.fine_iters))
            continue
        for it in range(sim.fine_iters):
            a, b = ev(), ev()
            a.record(stream)
            sim._hook_iteration()
            b.record(stream)
            iters.append((a, b, 1))
            for fn in sim.collision_solvers_iter:
                fn(it)
    stream.synchronize()
    it_ms = float(sum(a.elapsed_time(b) for a, b, _ in iters) / sum(n for _, _, n in iters))
    persistent = bool(sim.use_persistent and sim._persist_fits and not sim.collision_solvers_iter)
    pstatus = sim.persistent_status()
    if pstatus:
        raise RuntimeError(f"persistent pass reported status {pstatus}")
    flags = np.array([int(m["flags"]) for m in L.materials], np.int64)
    n_aniso = int(((flags[L.tet_material] & capi.MAT_ANISO) != 0).sum())
    alg_bytes = L.n_tets * 56 + n_aniso * 20 + L.n_verts * 40
    achieved = alg_bytes / (it_ms * 1e-3) / 1e9
    peak, peak_kind = _peak_hbm()
    traffic = None
    try:  # ncu DRAM bytes per iteration of this workload's tile pass, when captured
        traffic = json.loads(TRAFFIC.read_text()).get(args.config, {}).get("bytes_per_iteration")
    except (OSError, ValueError):
        pass
    hook_persistent = bool(sim._persist_fits and getattr(sim, "persistent_between_hooks", False)
                           and sim.use_persistent)
    per_iter = (1 if hook_persistent else 2) + (2 if getattr(sim, "dcd", None) is not None else 0)
    fine = len(sim._persist) if persistent else sim.fine_iters * per_iter
    coarse = 0
    if sim.mg is not None:
        co = sim.mg.coarse
        coarse = 1 if (co.use_persistent and co._persist_fits) else 2 * sim.mg.iters
    per_sub = 1 + fine + (2 + coarse if sim.mg is not None else 0)
    if getattr(sim, "dcd", None) is not None:  # broadphase on the first iteration
        every = max(1, int(sim.dcd.params.bvh_rebuild_every))
        per_sub += sum(sim.dcd.buf.broadphase_launches(True, refit_only=(k % every) != 0)
                       for k in range(sim.nsubsteps)) / sim.nsubsteps
    frame_kernel = bool(persistent and sim.persistent_sync == "exchange" and sim._exchange is not None
                        and not (sim._prm.tile_variant & ~0x53))
    # one launch per tile range, or the substeps' launches and a vertex step at the end
    launches_per_frame = 1 + (1 if sim.collision_solvers else 0) + (1 if sim._has_pins else 0) + (
        1 if sim.mg is not None else 0) + (len(sim._persist) if whole else sim.nsubsteps * per_sub + 1)
    n_iter = sim.nsubsteps * sim.fine_iters
    line = {
        "metric": "ms/frame", "value": round(ms_frame, 4), "unit": "ms/frame", "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": round(ms_frame, 4), "higher_is_better": False,
        "scaling": "strong" if (batched and world > 1) else "weak",
        "vs_baseline": None, "dtype": "f32", "data": "synthetic",
        "config": {"workload": WORKLOAD,
                   "n_verts": L.n_verts, "n_tets": L.n_tets, "n_tiles": L.n_tiles, "fine_iterations": sim.fine_iters,
                   "nsubsteps": sim.nsubsteps,
                   "parallelism": (f"instance shards x{world}" if batched else f"replicas x{world}"),
                   "l2": "flushed before every timed frame (256 MB write); inside a frame the ~37 MB "
                         "per-iteration working set stays in L2 (126 MB)"},
        "substeps_per_s": round(1e3 * sim.nsubsteps / ms_frame, 1),
        "tets_per_s": round(L.n_tets * n_iter / (ms_frame * 1e-3), 1),
        "e2e": {"value": round(ms_e2e, 4), "unit": "ms/frame", "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h},
        "roofline": {"bound": "hbm", "achieved": round(achieved, 1), "peak": peak, "unit": "GB/s",
                     "frac": round(achieved / peak, 4), "traffic": traffic, "peak_kind": peak_kind,
                     "kernel": ("k_frame_tiles (all substeps' Jacobi iterations and vertex steps in one launch; "
                                "time per iteration, inside a frame)") if whole else
                               (f"{'k_frame_tiles' if frame_kernel else 'k_iterate_persistent'} (all Jacobi iterations "
                                "of a substep in one launch; time per iteration, inside a frame)") if persistent else
                               ("k_iterate_persistent (one launch per iteration, a hook between iterations)"
                                if (sim._persist_fits and getattr(sim, "persistent_between_hooks", False)
                                    and sim.collision_solvers_iter and sim.use_persistent)
                                else "k_project_tiles + k_apply_list (one Jacobi iteration, timed inside a frame)"),
                     "algorithmic_bytes": alg_bytes, "iteration_us": round(it_ms * 1e3, 2),
                     "frame_roofline_ms": round(alg_bytes * n_iter / (peak * 1e9) * 1e3, 4)},
        "clocks": clk.summary(),
        **({"instances": n_inst_total, "instance_substeps_per_s": round(n_inst_total * sim.nsubsteps / (ms_frame * 1e-3), 1),
            "autotune": {k: v for k, v in tuned.items() if k != "tried"}} if batched else {}),
        "gpu_launches": int(round((launches_per_frame + 1) * args.steps)),
    }
    if rank == 0 and world == 1 and not args.no_cpu_baseline and args.config == "humanv2":
        cb = CpuBaseline(cfg, sc)
        line["cpu_baseline"] = cb.describe(cb.run(1, 2), 1, 2)
    sim.release_graphs()
    if world > 1:
        torch.distributed.barrier()
        torch.distributed.destroy_process_group()
    if rank == 0:
        print(json.dumps(line), flush=True)
    return 0


def run_profile_case(args):
    """Small deterministic workloads for ncu (no timing, no output line).

    humanv2: ``--steps`` frames of the benchmark configuration (the frame's
    launches issued eagerly, without the graph); batched: ``--steps`` frames of
    the 256-instance batch on the per-iteration tile pass.  box3m: a 64x64x120-hex box (2.95M tets, ~150 MB of tet
    streams, larger than L2) and ``--steps`` Jacobi iterations of its tet pass."""
    import torch
    if args.profile_case in ("humanv2", "humanv2_mg_dcd"):
        from rlmusclev2_b200.mg import MultiGridSim, load_config
        sim = MultiGridSim(load_config(str(CONFIGS[args.profile_case][0])))
        sim.use_graphs = False  # the same launches, issued eagerly so the profiler lists each kernel
        for f in range(sim.start_frame, sim.start_frame + args.steps):
            sim.set_fiber_activation(sim.scene.activation(f))
            sim.step_frame(f)
        sim.synchronize()
    elif args.profile_case == "batched":
        from rlmusclev2_b200.batch import BatchSim
        from rlmusclev2_b200.mg import load_config
        sim = BatchSim(load_config(str(CONFIGS["batched"][0])))
        sim.use_graphs = False
        sim.use_persistent = False  # the per-iteration tile pass the autotuner picks at 1 iteration per substep
        for f in range(sim.start_frame, sim.start_frame + args.steps):
            sim.step_frame_inputs(f)
        sim.synchronize()
    elif args.profile_case == "box3m":
        from rlmusclev2_b200 import MuscleSim
        from rlmusclev2_b200.meshgen import box_muscle
        m = box_muscle(nx=64, ny=64, nz=120, spacing=0.0025, seed=0)
        cons = [{"type": "tetarapsvd", "name": "arap", "compliance": 1e-7},
                {"type": "volume", "name": "volume", "compliance": 0.0}]
        sim = MuscleSim.from_procedural(m.verts, m.tets, m.fiber_per_tet, constraint_configs=cons,
                                        device="cuda:0", stopped=m.stopped, dts=1 / 24, num_substeps=10,
                                        gravity=-9.8)
        sim.integrate()
        for _ in range(args.steps):
            sim._fused_iteration()
        sim.synchronize()
    torch.cuda.synchronize()
    return 0


def run_box(args):
    """The box muscle (8x8x32 hexes, 2,673 verts / 12,288 tets, ARAP-SVD + volume,
    dt = 1/24 s in 10 substeps of one Jacobi iteration, the end 5 % pinned):
    ms/frame of MuscleSim.step() (one CUDA graph per frame) with the state on
    the GPU, and end to end with the positions read back every frame."""
    import torch

    from rlmusclev2_b200 import MuscleSim
    from rlmusclev2_b200.meshgen import box_muscle

    world, rank, local = _dist_setup()
    torch.cuda.set_device(local)
    m = box_muscle()
    cons = [{"type": "tetarapsvd", "name": "arap", "compliance": 1e-7},
            {"type": "volume", "name": "volume", "compliance": 0.0}]
    sim = MuscleSim.from_procedural(m.verts, m.tets, m.fiber_per_tet, constraint_configs=cons,
                                    device=f"cuda:{local}", stopped=m.stopped, dts=1.0 / 24.0, num_substeps=10,
                                    density=1060.0, veldamping=0.02, gravity=-9.8)
    s = sim._stream
    ev = lambda: torch.cuda.Event(enable_timing=True)  # noqa: E731
    for _ in range(args.warmup):
        sim.step()
    s.synchronize()
    if world > 1:
        torch.distributed.barrier()
    evs = [(ev(), ev()) for _ in range(args.steps)]
    with ClockSampler(torch.cuda.current_device()) as clk:
        for a, b in evs:
            a.record(s)
            sim.step()
            b.record(s)
        s.synchronize()
    ms = sum(a.elapsed_time(b) for a, b in evs) / args.steps
    evs2 = [(ev(), ev()) for _ in range(args.steps)]
    for a, b in evs2:
        a.record(s)
        sim.step()
        sim.positions_np()
        b.record(s)
    s.synchronize()
    ms_e2e = sum(a.elapsed_time(b) for a, b in evs2) / args.steps
    if world > 1:
        t = torch.tensor([ms, ms_e2e], device=sim.device)
        torch.distributed.all_reduce(t, op=torch.distributed.ReduceOp.MAX)
        ms, ms_e2e = (float(x) for x in t.tolist())
    L = sim.layout
    alg = L.n_tets * 56 + L.n_verts * 40
    peak, peak_kind = _peak_hbm()
    it_s = ms * 1e-3 / 10
    one = sim.use_persistent and sim._persist_fits and sim._exchange is not None  # the frame is one launch per range
    line = {
        "metric": "ms/frame", "value": round(ms, 4), "unit": "ms/frame", "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": round(ms, 4), "higher_is_better": False, "scaling": "weak",
        "vs_baseline": None, "dtype": "f32", "data": "synthetic",
        "config": {"workload": WORKLOAD, "n_verts": L.n_verts, "n_tets": L.n_tets, "n_tiles": L.n_tiles,
                   "parallelism": f"replicas x{world}", "l2": "the 0.8 MB working set stays in L2"},
        "substeps_per_s": round(10e3 / ms, 1), "tets_per_s": round(L.n_tets * 10 / (ms * 1e-3), 1),
        "e2e": {"value": round(ms_e2e, 4), "unit": "ms/frame", "h2d_bytes_per_step": 0,
                "d2h_bytes_per_step": L.n_verts * 12},
        "roofline": {"bound": "launch", "achieved": round(alg / it_s / 1e9, 1), "peak": peak, "unit": "GB/s",
                     "frac": round(alg / it_s / 1e9 / peak, 5), "traffic": None, "peak_kind": peak_kind,
                     "kernel": ("k_frame_tiles (a frame's ten substeps in one launch; launch and latency at 12k tets)" if one
                                else "whole substep (prediction, tile pass, boundary finish): launch-bound at 12k tets"),
                     "algorithmic_bytes": alg},
        "clocks": clk.summary(), "gpu_launches": int((len(sim._persist) if one else 21) * args.steps),
    }
    sim.release_graphs()
    if world > 1:
        torch.distributed.barrier()
        torch.distributed.destroy_process_group()
    if rank == 0:
        print(json.dumps(line), flush=True)
    return 0


def run_learned(args):
    """The learned coarse warm start against the plain solver on config 3's
    mesh and cage, measured in this run on held-out motion seed 41 (frames
    1-4): the max error against the 200-iteration solve from the same
    prediction after n fine iterations (n = 10..160) for the plain form, the
    learned form and the ideal form (the substep's true cage correction, what
    a perfect network would give); the iterations each needs to reach 0.1 mm;
    ms/frame of each form (CUDA events); and the resulting gate."""
    import torch

    from rlmusclev2_b200 import learned as LW
    from rlmusclev2_b200.meshgen import reseed_motion
    from rlmusclev2_b200.mg import MultiGridSim

    world, rank, local = _dist_setup()
    torch.cuda.set_device(local)
    sim = MultiGridSim(LW.learned_config(), device=f"cuda:{local}")
    ws = LW.LearnedWarmStart(sim)
    meta = LW.load_weights(ws)
    ns = [10, 20, 40, 80, 120, 160, 180, 200]
    ws.plain_taken.zero_()
    err, rms = LW.evaluate(ws, [41], 4, ns, ideal=True, checked_ns=(10, 20))
    checked_taken = int(ws.plain_taken.item())
    n_to = {form: LW.iterations_to(err[form], 0.1) for form in ("plain", "learned", "ideal")}
    base = sim.scene
    s = sim._stream
    ev = lambda: torch.cuda.Event(enable_timing=True)  # noqa: E731

    def timed(n, learned, fallback=True):
        ws.reset(reseed_motion(base, 41))
        for f in range(1, 1 + args.warmup):
            ws.frame(f, n, learned, fallback)
        times = []
        with ClockSampler(torch.cuda.current_device()) as clk:
            for f in range(1 + args.warmup, 1 + args.warmup + args.steps):
                ws.begin_frame(f)
                a, b = ev(), ev()
                a.record(s)
                for sub in range(sim.nsubsteps):
                    ws.substep(sub, n, learned, fallback)
                b.record(s)
                ws.end_frame()
                b.synchronize()
                times.append(a.elapsed_time(b))
        return float(np.mean(times)), clk.summary()

    n_l, n_p = 10, 20
    t_p10, _ = timed(10, False)
    t_p20, _ = timed(n_p, False)
    t_learn, clocks = timed(n_l, True)
    t_checked, _ = timed(n_l, True, "residual")
    if world > 1:
        t = torch.tensor([t_learn, t_p20, t_p10, t_checked], device=sim.device)
        torch.distributed.all_reduce(t, op=torch.distributed.ReduceOp.MAX)
        t_learn, t_p20, t_p10, t_checked = (float(x) for x in t.tolist())
    t_iter = (t_p20 - t_p10) / (10 * sim.nsubsteps)  # ms per fine iteration
    fixed = (t_learn - t_p10) / sim.nsubsteps  # ms per substep: restriction, features, network, prolongation
    frame_ms = lambda n, extra: sim.nsubsteps * (extra + n * t_iter) + (t_p10 - 10 * t_iter * sim.nsubsteps)  # noqa: E731
    est = {form: (None if n is None else round(frame_ms(n, fixed if form != "plain" else 0.0), 3))
           for form, n in n_to.items()}
    summ = lambda e: dict(max_mm=round(float(e.max()), 4), p95_mm=round(float(np.percentile(e, 95)), 4))  # noqa: E731
    line = {
        "metric": "ms/frame (learned warm start)", "value": round(t_learn, 4), "unit": "ms/frame", "n_gpus": world,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(t_learn, 4), "higher_is_better": False,
        "scaling": "weak", "vs_baseline": None, "dtype": "bf16 network, f32 solver", "data": "synthetic",
        "config": {"workload": WORKLOAD, "n_verts": sim.NV, "n_tets": sim.NT, "cage_verts": ws.nc,
                   "learned_iterations": n_l, "plain_iterations": n_p, "parallelism": f"replicas x{world}"},
        "plain_ms_per_frame": round(t_p20, 4), "speedup_vs_plain": round(t_p20 / t_learn, 3),
        "ms_per_iteration": round(t_iter, 5), "warm_start_ms_per_substep": round(fixed, 5),
        "error_vs_200_iteration_solve": {form: {str(n): summ(err[form][n]) for n in ns}
                                         for form in ("plain", "learned", "ideal")},
        "iterations_to_0.1mm": {k: (None if v is None else round(v, 1)) for k, v in n_to.items()},
        # the fallback rule as stated: every substep also runs the plain solve and
        # keeps it when the learned post-iteration ARAP residual is higher
        "residual_checked_fallback": {
            "ms_per_frame": round(t_checked, 4), "iterations": n_l,
            "error_vs_200_iteration_solve": {str(n): summ(err["checked"][n]) for n in (10, 20)},
            "plain_taken": checked_taken, "checks": int(2 * err["checked"][10].shape[0])},
        "ms_per_frame_at_0.1mm": est,
        "gate_0.1mm_at_2x": bool(est["learned"] is not None and est["plain"] is not None
                                 and est["learned"] <= 0.5 * est["plain"]),
        "frames": "held-out seed 41, frames 1-4", "weights": meta, "clocks": clocks,
    }
    if world > 1:
        torch.distributed.barrier()
        torch.distributed.destroy_process_group()
    if rank == 0:
        print(json.dumps(line), flush=True)
    return 0


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--config", choices=sorted(CONFIGS), default="humanv2",
                    help="workload (default: the 535k-tet configuration the metric is quoted on)")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--profile-case", choices=["humanv2", "humanv2_mg_dcd", "batched", "box3m"], default=None,
                    help="run a small fixed workload for ncu and exit")
    args = ap.parse_args()
    global CONFIG, WORKLOAD
    CONFIG, WORKLOAD = CONFIGS[args.config]
    if args.profile_case:
        return run_profile_case(args)
    if args.warmup < 3:
        ap.error("--warmup must be >= 3")
    if args.impl == "reference":
        return run_reference(args)
    if args.config == "learned":
        return run_learned(args)
    if args.config == "box":
        return run_box(args)
    return run_ours(args)


if __name__ == "__main__":
    sys.exit(main())
