"""Benchmark: ABD body-steps/s at the 1e-5 Newton residual (plus Newton
iterations per step) for one workload, as one JSON line.

Workloads (--workload):
  pile    4096 icospheres landing in a 12x12x40 open box, dt = 1/120, from
          the state after 100 steps (the dense pile-up configuration)
  net16   16x16 chain mail of 256 torus links (288 verts / 576 tris each),
          corner links pinned, dt = 1/240, FP64 (default; the chain-net
          configuration of the benchmark suite)
  chain   the reference's own 144-link chain scene with its constants
  cubes   8 falling unit cubes on a ground plane, dt = 1/120
  batch   512 independent scenes of 4..64 cubes/tori, one handle
A step is one physics time step of the whole workload (Newton to 1e-5 or
16 iterations, with collision detection, assembly, Krylov solve, CCD and
line search).  Inputs are seeded synthetic scenes.

Arms: --impl ours (default) runs libabd_b200.so; --impl reference runs the
CPU restatement of the reference's step (the oracle: the reference itself
is Python + NVIDIA Warp, which is not installable here) on all host cores.

Multi-GPU (torchrun): every rank steps its own replica (seeded by rank) on
its own GPU with no collective in the step ("replicas only" for single-scene
workloads; scenes shard for `batch`); the value is all ranks' body-steps
over the slowest rank's device time.
"""
import argparse
import json
import os
import subprocess
import sys
import threading
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

import numpy as np  # noqa: E402

METRIC = "ABD body-steps/s @1e-5 residual: learned+batched vs plain, same B200; iters/step"
PILE_MAX_ITER = 512


def make_workload(name, rank=0, precision=0, ns_batch=512, world=1):
    from colb_b200 import params as P, scene as S
    if name == "net16":
        from colb_b200 import fixtures
        state, t0, seed = fixtures.load_net16()
        sc = dict(S.config2_chain_net(n=16, seed=seed), state=state)
        p = P.config_params(dt=1.0 / 240.0, precision=precision)
        cfg = dict(workload=f"net16: 16x16 torus chain mail, 256 links (R 1.0, r 0.25, 24x12 -> 288 v / 576 t), "
                   f"4 corners pinned, dt 1/240, log barrier dhat 1e-3 kappa 1e7, k_ortho 1e7, CCD line search; "
                   f"timed from the resting state after {t0} plain FP64 steps (colb_b200/data/net16_t120.npz)",
                   bodies=256, verts=len(sc["xbar"]), tris=len(sc["tris"]), start_step=t0)
        return [sc], p, cfg
    if name == "pile":
        from colb_b200 import fixtures
        state, t0, seed = fixtures.load_pile()
        sc = dict(S.config5_pile(seed=seed), state=state)
        # landing spheres need far more than 64 Newton iterations per step
        # to reach the 1e-5 residual (the cap ends the step unconverged)
        p = P.config_params(precision=precision, newton_max_iter=PILE_MAX_ITER)
        cfg = dict(workload=f"pile: 4096 icospheres (subdivision 1/2, r U(0.2,0.5)) dropped into a 12x12x40 open box "
                   f"(ground + 4 wall half-spaces), dt 1/120, log barrier dhat 1e-3 kappa 1e7, k_ortho 1e7, CCD line "
                   f"search, Newton cap {PILE_MAX_ITER}; timed from step {t0} while the spheres land "
                   f"(colb_b200/data/pile_t100.npz)", bodies=4096, verts=len(sc["xbar"]), tris=len(sc["tris"]),
                   start_step=t0)
        return [sc], p, cfg
    if name == "net16c":
        sc = S.config2_chain_net(n=16, seed=rank, pitch=1.5 - 5e-4)
        p = P.config_params(dt=1.0 / 240.0, precision=precision)
        cfg = dict(workload="net16c: the net16 chain mail at pitch 1.4995, every interlocked pair within dhat at t=0 "
                   "(contact-rich from the first step)", bodies=256, verts=len(sc["xbar"]), tris=len(sc["tris"]))
        return [sc], p, cfg
    if name == "chain":
        sc = S.load_npz_scene(os.path.join(ROOT, "tests", "golden", "chains_scene.npz"))
        p = P.reference_params(precision=precision)
        cfg = dict(workload="chain: reference assets/chains.json, 144 links of link.ma, reference constants "
                   "(dt 8e-3, kappa 4e8, cubic barrier dhat 0.095, EE contact)", bodies=144, verts=len(sc["xbar"]))
        return [sc], p, cfg
    if name == "cubes":
        sc = S.config1_cubes(seed=rank)
        p = P.config_params(precision=precision)
        cfg = dict(workload="cubes: 8 unit cubes 2x2x2, ground plane, dt 1/120", bodies=8)
        return [sc], p, cfg
    if name == "batch":
        # ns_batch scenes per GPU: world * ns_batch seeded scenes partitioned
        # across ranks by primitive count (colb_b200/shard.py)
        from colb_b200 import shard
        allsc = S.config3_batch(n_scenes=ns_batch * world, seed=0)
        scenes, _ = shard.shard(allsc, rank, world)
        p = P.config_params(precision=precision)
        nb = sum(len(s["mass"]) for s in scenes)
        cfg = dict(workload=f"batch: {ns_batch} scenes per GPU of 4..64 cubes/tori (log-uniform), ground, dt 1/120",
                   bodies=nb, scenes=len(scenes), scenes_total=len(allsc))
        return scenes, p, cfg
    raise SystemExit(f"unknown workload {name}")


def dynamic_bodies(scenes):
    return int(sum((s["mass"] > 0).sum() for s in scenes))


class ClockSampler:
    """SM clocks and clock-event (throttle) reasons while the timed region
    runs, read in-process through NVML every 0.25 s (reading only; spawning
    nvidia-smi instead stalls the host-synchronous step loop).  Falls back to
    nvidia-smi when NVML cannot be loaded."""

    def __init__(self, device=0, period=0.25):
        self.device = device
        self.period = period
        self.rows = []           # (sm_mhz, sm_max_mhz, reasons bitmask)
        self._stop = threading.Event()
        self._t = threading.Thread(target=self._run, daemon=True)
        self._nv = None

    def _sample_nvml(self, h):
        nv = self._nv
        sm = nv.nvmlDeviceGetClockInfo(h, nv.NVML_CLOCK_SM)
        mx = nv.nvmlDeviceGetMaxClockInfo(h, nv.NVML_CLOCK_SM)
        try:
            rs = nv.nvmlDeviceGetCurrentClocksEventReasons(h)
        except Exception:
            rs = nv.nvmlDeviceGetCurrentClocksThrottleReasons(h)
        self.rows.append((float(sm), float(mx), int(rs)))

    def _sample_smi(self):
        fields = "clocks.sm,clocks.max.sm,clocks_event_reasons.active"
        out = subprocess.run(["nvidia-smi", "-i", str(self.device), "--query-gpu=" + fields,
                              "--format=csv,noheader,nounits"], capture_output=True, text=True, timeout=5)
        if out.returncode == 0 and out.stdout.strip():
            c = [x.strip() for x in out.stdout.strip().split(",")]
            self.rows.append((float(c[0]), float(c[1]), int(c[2], 16)))

    def _run(self):
        h = None
        try:
            import pynvml as nv
            nv.nvmlInit()
            self._nv = nv
            h = nv.nvmlDeviceGetHandleByIndex(self.device)
        except Exception:
            self._nv = None
        while not self._stop.is_set():
            try:
                if self._nv is not None:
                    self._sample_nvml(h)
                else:
                    self._sample_smi()
            except Exception:
                pass
            self._stop.wait(self.period)

    def __enter__(self):
        self._t.start()
        return self

    def __exit__(self, *a):
        self._stop.set()
        self._t.join(timeout=10)

    def summary(self):
        if not self.rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["clock sampling unavailable"], "samples": 0}
        bits = {"hw_slowdown": 0x8, "sw_thermal_slowdown": 0x20, "hw_thermal_slowdown": 0x40, "sw_power_cap": 0x4}
        reasons = sorted({name for r in self.rows for name, bit in bits.items() if r[2] & bit})
        return {"sm_mhz": float(np.median([r[0] for r in self.rows])), "sm_max_mhz": max(r[1] for r in self.rows),
                "reasons": reasons, "samples": len(self.rows), "source": "nvml" if self._nv is not None else "nvidia-smi"}


def measured_peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            d = json.load(f)
        return float(d["hbm_gbs"]), "measured"
    except Exception:
        return 6650.0, "fallback"


def traffic_from_profiles(kernel, workload):
    """Per-launch DRAM bytes of `kernel` from the committed ncu summary, if any."""
    try:
        with open(os.path.join(ROOT, "profiles", "traffic.json")) as f:
            d = json.load(f)
        return d.get(workload, {}).get(kernel)
    except Exception:
        return None


def cpu_baseline(scenes, params, cfg, budget_s=20.0, threads=None):
    """The oracle (CPU restatement of the reference step) on all host cores,
    on a bounded sample of the same workload: the full scene for as many
    steps as fit in about `budget_s`."""
    from oracle import oracle as O
    threads = threads or os.cpu_count()
    O.set_threads(threads)
    w = O.OracleWorld(params, scenes)
    nb = dynamic_bodies(scenes)
    steps, t0 = 0, time.perf_counter()
    iters = 0
    by_step = []
    while True:
        rc, st = w.step(1)
        steps += 1
        iters += st.newton_iters
        by_step.append(int(st.newton_iters))
        el = time.perf_counter() - t0
        if el > budget_s or steps >= 200:
            break
    value = nb * steps / el
    return {"value": value, "unit": "body-steps/s", "cores": threads, "kind": "port",
            "sample": f"{steps} full steps of {cfg['workload'].split(':')[0]} from step {cfg.get('start_step', 0)} ({el:.1f} s, "
                      f"{iters / max(1, steps * len(scenes)):.2f} Newton iters/step/scene), oracle/abd_oracle.c with OpenMP",
            "start_step": cfg.get("start_step", 0), "newton_iters_by_step": by_step}


def flush_l2(buf):
    buf.add_(1.0)   # writes 256 MB (> 126 MB L2)


def run_ours(args, rank, world):
    import torch
    from colb_b200.engine import Engine
    dev = int(os.environ.get("LOCAL_RANK", 0))
    torch.cuda.set_device(dev)
    scenes, p, cfg = make_workload(args.workload, rank, args.precision, world=world)
    if args.ls_graph is not None:
        p.ls_graph = args.ls_graph
    cfg = dict(cfg, line_search="one CUDA graph per Newton iteration" if p.ls_graph else "host loop per trial")
    if args.ls_groups:
        p.ls_groups = 1
        cfg = dict(cfg, line_search="one step length per contact group")
    if args.warm_start:
        p.warm_start = args.warm_start
        cfg = dict(cfg, warm_start={2: "inertial", 3: "learned (colb_b200/data/warmstart_net16.npz)"}[args.warm_start])
    eng = Engine(p, scenes, device=dev)
    if args.warm_start == 3:
        from colb_b200 import learned as Lr
        params, norm, _ = Lr.load()
        eng.set_mlp(params, norm)
    nb = dynamic_bodies(scenes)
    flush = torch.empty(64 * 1024 * 1024, dtype=torch.float32, device="cuda")
    # the warm-up steps settle the autotuner, the line-search graph and the
    # buffer sizes; the timed steps then start again from the workload's
    # start state, the same state the CPU arms start from
    state0 = eng.get_state()
    for _ in range(args.warmup):
        eng.step(1)
    eng.set_state(state0)
    # ---- timed: device time of K steps, L2 flushed before each step
    if world > 1:
        import torch.distributed as dist
        dist.barrier()
    torch.cuda.synchronize()
    gpu_ms, launches, iters, unconv, lin, graphs, syncs = 0.0, 0, 0, 0, 0, 0, 0
    by_step, xs = [], []
    keep_x = args.workload == "net16" and not args.profile
    with ClockSampler(dev) as clk:
        for _ in range(args.steps):
            flush_l2(flush)
            torch.cuda.synchronize()
            rc, st = eng.step(1)
            gpu_ms += st.gpu_ms
            launches += st.kernel_launches
            iters += st.newton_iters
            unconv += st.unconverged
            lin += st.lin_iters
            graphs += st.ls_graph_launches
            syncs += st.host_syncs
            by_step.append(int(st.newton_iters))
            if keep_x and len(xs) < 10:
                xs.append(eng.vertices())       # after the device-timed step: FP64 positions for the forms' error
    torch.cuda.synchronize()
    t = torch.tensor([gpu_ms], dtype=torch.float64, device="cuda")
    if world > 1:
        import torch.distributed as dist
        dist.barrier()
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
    max_ms = float(t.item())
    # bodies over all ranks (scene shards differ in size)
    nbt = torch.tensor([float(nb)], dtype=torch.float64, device="cuda")
    if world > 1:
        import torch.distributed as dist
        dist.all_reduce(nbt)
    nb = int(nbt.item()) if world > 1 else nb
    if args.profile:
        return dict(scenes=scenes, p=p, cfg=cfg, nb=nb, max_ms=max_ms, launches=launches, iters=iters, unconv=unconv,
                    lin=lin, e2e_s=float("nan"), clocks=clk.summary(), phases=None, n_timing=0, bytes_state=48 * 8 * eng.nb,
                    graphs=graphs, syncs=syncs, by_step=by_step, state0=state0, xs=xs)
    # ---- e2e through the public API with host buffers: the same K steps
    # from the same state, with H2D of the state, one step and D2H of the
    # state every step
    eng.set_state(state0)
    try:
        pinned = torch.from_numpy(state0.copy()).pin_memory().numpy()
    except Exception:
        pinned = state0.copy()
    e2e_iters = 0
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    for _ in range(args.steps):
        eng.set_state(pinned)
        rc, st = eng.step(1)
        e2e_iters += st.newton_iters
        eng.get_state(out=pinned)
    e2e_s = time.perf_counter() - t0
    e2e_t = torch.tensor([e2e_s], dtype=torch.float64, device="cuda")
    if world > 1:
        import torch.distributed as dist
        dist.all_reduce(e2e_t, op=dist.ReduceOp.MAX)
    # ---- per-phase device timers (separate pass over the first timed steps,
    # from the same state)
    eng.set_state(state0)
    eng.set_timing(True, True)
    n_timing = max(2, min(args.steps, 5))
    for _ in range(n_timing):
        eng.step(1)
    phases = eng.timing()
    eng.set_timing(False, True)
    return dict(scenes=scenes, p=p, cfg=cfg, nb=nb, max_ms=max_ms, launches=launches, iters=iters, unconv=unconv,
                lin=lin, e2e_s=float(e2e_t.item()), clocks=clk.summary(), phases=phases, n_timing=n_timing,
                bytes_state=48 * 8 * eng.nb, graphs=graphs, e2e_iters=e2e_iters, syncs=syncs, by_step=by_step,
                state0=state0, xs=xs)


def run_forms(args, scenes, p, ref_xs=None, dev=0):
    """The three forms beside the plain FP64 solver on the same workload:
    mixed precision, the learned warm start, and 8 scenes batched in one
    handle (alone and all together).  Each form warms up for 2 steps, then
    times min(K, 10) steps from the workload's start state (the plain
    solver's timed start).  Forms in mixed precision report, for every
    timed step, the largest vertex position error of the first scene copy
    against the plain FP64 run's positions after the same step (`ref_xs`),
    relative to the scene extent."""
    import torch
    from colb_b200 import learned as Lr
    from colb_b200._abi import params_to_dict, params_from_dict
    from colb_b200.engine import Engine
    params, norm, meta = Lr.load()
    steps = max(1, min(args.steps, 10))
    base = params_to_dict(p)
    forms = {"mixed": (dict(precision=1), 1, False), "learned": (dict(warm_start=3), 1, True),
             "batched_x8": ({}, 8, False), "batched_x8+mixed": (dict(precision=1), 8, False),
             "learned+batched_x8+mixed": (dict(precision=1, warm_start=3), 8, True)}
    if args.workload == "pile":
        # one scene of 4096 bodies: the batched form steps its contact groups
        # as independent units (one step length per group, ls_groups)
        forms = {"mixed": (dict(precision=1), 1, False), "contact_groups": (dict(ls_groups=1), 1, False),
                 "learned": (dict(warm_start=3), 1, True),
                 "learned+contact_groups+mixed": (dict(precision=1, warm_start=3, ls_groups=1), 1, True)}
    out = {}
    allow = (-5, -6, -7)
    for name, (over, copies, learned) in forms.items():
        e = None
        try:
            e = Engine(params_from_dict(dict(base, **over)), list(scenes) * copies, device=dev)
            if learned:
                e.set_mlp(params, norm)
            nb = dynamic_bodies(scenes) * copies
            start = e.get_state()
            for _ in range(2):
                e.step(1, allow=allow)
            e.set_state(start)
            torch.cuda.synchronize()
            ms = it = unconv = syncs = 0
            errs = []
            nv1 = len(scenes[0]["xbar"])
            for k in range(steps):
                rc, st = e.step(1, allow=allow)
                ms += st.gpu_ms; it += st.newton_iters; unconv += st.unconverged; syncs += st.host_syncs
                if over.get("precision") == 1 and ref_xs is not None and k < len(ref_xs):
                    x = e.vertices()[:nv1]
                    errs.append(float(np.abs(x - ref_xs[k]).max() / np.abs(ref_xs[k]).max()))
            out[name] = {"value": nb * steps / (ms / 1000.0), "unit": "body-steps/s",
                         "newton_iters_per_step": it / (steps * len(scenes) * copies), "unconverged_steps": unconv,
                         "steps": steps, "intersections": e.count_intersections(),
                         "host_syncs_per_step": syncs / steps}
            if errs:
                out[name]["max_rel_pos_err_per_step"] = errs
                out[name]["max_rel_pos_err_vs_fp64"] = max(errs)
        except Exception as ex:                      # report the form as failed, keep the line
            out[name] = {"error": str(ex)}
        finally:
            if e is not None:
                e.close()
    out["learned_model"] = dict(meta, file="colb_b200/data/warmstart_net16.npz")
    return out


def run_batch512(args, dev=0):
    """The batched-scenes configuration: 512 scenes of 4..64 cubes / tori in
    one handle, mixed precision and FP64, device time of min(K, 10) steps
    after 2 warm-up steps from the scenes' initial state."""
    import torch
    from colb_b200 import params as P, scene as S
    from colb_b200.engine import Engine
    scenes = S.config3_batch(n_scenes=512, seed=0)
    nb = dynamic_bodies(scenes)
    steps = max(1, min(args.steps, 10))
    out = {"scenes": len(scenes), "bodies": nb}
    for name, prec in (("fp64", 0), ("mixed", 1)):
        e = None
        try:
            e = Engine(P.config_params(precision=prec), scenes, device=dev)
            start = e.get_state()
            for _ in range(2):
                e.step(1, allow=(-5, -6, -7))
            e.set_state(start)
            torch.cuda.synchronize()
            ms = it = unconv = 0
            for _ in range(steps):
                rc, st = e.step(1, allow=(-5, -6, -7))
                ms += st.gpu_ms; it += st.newton_iters; unconv += st.unconverged
            out[name] = {"value": nb * steps / (ms / 1000.0), "unit": "body-steps/s",
                         "newton_iters_per_step": it / (steps * len(scenes)), "unconverged_steps": unconv,
                         "steps": steps, "intersections": e.count_intersections()}
        except Exception as ex:
            out[name] = {"error": str(ex)}
        finally:
            if e is not None:
                e.close()
    return out


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--workload", default="net16", choices=["net16", "net16c", "chain", "cubes", "batch", "pile"])
    ap.add_argument("--ls-groups", type=int, default=0, choices=[0, 1], help="1: one step length per contact group")
    ap.add_argument("--ls-graph", type=int, default=None, choices=[0, 1],
                    help="1: line search as one CUDA graph per Newton iteration, 0: host loop (default: the workload's)")
    ap.add_argument("--precision", type=int, default=0, help="0 FP64, 1 mixed FP32/FP64")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--warm-start", type=int, default=0, choices=[0, 2, 3], help="0 plain, 2 inertial, 3 learned network")
    ap.add_argument("--no-forms", action="store_true", help="skip the mixed / learned / batched measurements")
    ap.add_argument("--profile", action="store_true",
                    help="timed steps only (no end-to-end, phase-timer, forms or CPU passes): the command to run under ncu")
    args = ap.parse_args()
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))

    if args.impl == "reference":
        if rank != 0:
            return
        if args.workload == "pile":
            print(json.dumps({"impl": "reference", "metric": METRIC,
                              "unavailable": "one CPU oracle step of the 4096-body pile takes longer than 15 min on 8 cores"}))
            return
        scenes, p, cfg = make_workload(args.workload, 0, args.precision)
        cb = cpu_baseline(scenes, p, cfg, budget_s=max(10.0, 6.0 * args.steps))
        line = {"metric": METRIC, "value": cb["value"], "unit": "body-steps/s", "n_gpus": args.gpus,
                "steps": args.steps, "warmup": args.warmup, "higher_is_better": True, "impl": "reference",
                "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
                "config": cfg, "cpu_baseline": cb,
                "e2e": {"value": cb["value"], "unit": "body-steps/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
                "note": "reference = CPU restatement of abd.py's step (the reference needs NVIDIA Warp, not installable here)"}
        print(json.dumps(line))
        return

    if world > 1:
        import torch
        import torch.distributed as dist
        torch.cuda.set_device(int(os.environ.get("LOCAL_RANK", 0)))
        dist.init_process_group("nccl", timeout=__import__("datetime").timedelta(seconds=120))
    r = run_ours(args, rank, world)
    nb_total = r["nb"]
    if args.profile:
        if rank == 0:
            print(json.dumps({"metric": METRIC, "value": nb_total * args.steps / (r["max_ms"] / 1000.0),
                              "unit": "body-steps/s", "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
                              "profile_run": True, "gpu_launches": r["launches"],
                              "newton_iters_per_step": r["iters"] / (args.steps * len(r["scenes"]))}))
        return
    value = nb_total * args.steps / (r["max_ms"] / 1000.0)
    e2e = nb_total * args.steps / r["e2e_s"]
    peak, peak_kind = measured_peaks()
    ph = r["phases"]
    # dominant kernel of this library among the phases that bracket one kernel
    # launch each (cuSOLVER's factorization, when the direct solver runs, is
    # reported separately as phases_ms_per_step.dense; the swept-candidate
    # phase brackets several kernels, a sort and a host read-back, so it
    # appears only in phases_ms_per_step)
    kernel_names = {"asm_contact": "k_contact_assemble", "energy_list": "k_ls_energy",
                    "spmv": "k_bi_scene / k_pcg_spmv / k_bi_spmv", "energy_query": "k_ee/pt_energy", "band": "k_band_solve"}
    dom = max(kernel_names, key=lambda k: ph[k]["ms"])
    avg_ms = ph[dom]["ms"] / max(1, ph[dom]["launches"])
    avg_bytes = ph[dom]["bytes"] / max(1, ph[dom]["launches"])
    achieved = avg_bytes / (avg_ms / 1000.0) / 1e9 if avg_ms > 0 else 0.0
    line = {
        "metric": METRIC, "value": value, "unit": "body-steps/s", "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": r["max_ms"] / args.steps, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f64" if args.precision == 0 else "f32+f64",
        "data": "synthetic",
        "config": dict(r["cfg"], parallelism=f"replicas x{world}" if args.workload != "batch" else f"scenes sharded x{world}",
                       l2="flushed before every timed step (256 MB write)", precision="fp64" if args.precision == 0 else "mixed"),
        "newton_iters_per_step": r["iters"] / (args.steps * len(r["scenes"])),
        "krylov_iters_per_step": r["lin"] / args.steps,
        "newton_iters_by_step": r["by_step"],
        "timed_steps_start": r["cfg"].get("start_step", 0),
        "unconverged_steps": r["unconv"],
        "gpu_launches": r["launches"],
        "ls_graph_launches": r["graphs"],
        "host_syncs_per_newton_iter": r["syncs"] / max(1, r["iters"]),
        "e2e": {"value": e2e, "unit": "body-steps/s", "h2d_bytes_per_step": r["bytes_state"],
                "d2h_bytes_per_step": r["bytes_state"],
                "newton_iters_per_step": r["e2e_iters"] / (args.steps * len(r["scenes"])),
                "note": "the timed steps again from the same state, host copies of the state in and out every step"},
        "roofline": {"bound": "hbm", "kernel": kernel_names[dom], "phase": dom, "achieved": achieved, "peak": peak, "unit": "GB/s",
                     "frac": achieved / peak, "peak_source": peak_kind,
                     "traffic": traffic_from_profiles(kernel_names[dom].split(" ")[0], args.workload),
                     "algorithmic_bytes_per_launch": avg_bytes, "avg_launch_ms": avg_ms},
        "phases_ms_per_step": {k: v["ms"] / r["n_timing"] for k, v in ph.items()},
        "phases_note": (f"separate pass over the first {r['n_timing']} timed steps from the same state; every phase "
                        "is bracketed by events and the line search runs as the host loop, so phases overlap "
                        "(solve contains dense and band) and their sum exceeds ms_per_step"),
        "clocks": r["clocks"],
    }
    if rank == 0 and world == 1 and args.workload in ("net16", "pile") and not args.no_forms:
        forms = {"plain_fp64": {"value": value, "unit": "body-steps/s",
                                "newton_iters_per_step": line["newton_iters_per_step"], "steps": args.steps}}
        forms.update(run_forms(args, r["scenes"], r["p"], ref_xs=r["xs"]))
        if args.workload == "net16":
            forms["batch512"] = run_batch512(args)
        plain = forms["plain_fp64"]["value"]
        lbm = forms.get("learned+batched_x8+mixed", {})
        if "value" in lbm:
            # the benchmark's headline comparison: learned + batched + mixed
            # against the plain FP64 solver on the same net, same B200
            forms["learned+batched_x8+mixed_vs_plain"] = {
                "speedup": lbm["value"] / plain,
                "newton_iter_cut": 1.0 - lbm["newton_iters_per_step"] / forms["plain_fp64"]["newton_iters_per_step"]}
        line["forms"] = forms
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        if args.workload == "pile":
            line["cpu_baseline"] = {"value": None, "unit": "body-steps/s", "cores": os.cpu_count(), "kind": "port",
                                    "sample": "none: one oracle step of the 4096-body pile takes longer than 15 min on "
                                              "8 host cores, beyond a bounded sample"}
        else:
            cb = cpu_baseline(r["scenes"], r["p"], r["cfg"])
            # both arms start their timed steps from the same state: put the
            # GPU's Newton iterations of the same steps beside the oracle's
            cb["gpu_newton_iters_by_step"] = r["by_step"][:len(cb["newton_iters_by_step"])]
            line["cpu_baseline"] = cb
    if rank == 0:
        print(json.dumps(line))
    if world > 1:
        import torch.distributed as dist
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
