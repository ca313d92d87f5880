"""Benchmark: ms per electronic step of the 512-atom Si-like cell on one B200.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

Workload (si512): 512-atom diamond-lattice cell a=41.04 bohr of the synthetic
Si-like species, atoms displaced by U(-0.05,0.05) bohr (seed 5), Gamma point,
25 Ry, 1024 bands, PBE; coefficients complex N(0,1) from seed 5, then
orthonormalised.  A step is one SCF iteration with nite=0: update_density,
update_vhxc, energy(true) (H*psi), eigenvalue_sum and one PSDA update with
ortho_align.  The wavefunctions (1.2 GB) are larger than L2, so no flush is
needed between steps.

The headline `value` is the mixed-precision path (FP32 staged FFTs); the FP64
path is timed in the same run (`fp64_ms_per_step`), and `dE_per_atom` is the
total-energy difference between the two after the same steps.  `e2e` runs
the same step through the C ABI with the wavefunctions in pinned host memory:
each step uploads C, runs the step and downloads C and the energies.

Under torchrun each rank runs an independent replica on its own GPU (the
electronic step of one cell does not shard in this build).  `--impl
reference` times one full electronic step of the same cell (all 1024 bands)
on the reference's own CPU build (oracle/_ref) with every host thread; one
step takes minutes there, so it is timed once whatever --steps says.  The
`cpu_baseline` leg of this arm reuses that measurement when the reference arm
ran on this machine since its last boot, and otherwise models the step from a
32-band sample (the line's `cpu_baseline.sample` says which).
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import tempfile
import time

# The 32-system batch runs one stream per system: let the device give each its
# own hardware queue (the default of 8 serialises streams onto shared queues).
# Read once, when this process creates its CUDA context.
os.environ.setdefault("CUDA_DEVICE_MAX_CONNECTIONS", "32")

ROOT = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(ROOT, "qbox-public_b200")
for p in (PKG, ROOT):
    if p not in sys.path:
        sys.path.insert(0, p)

METRIC = ("ms per electronic step, mixed vs FP64 on GPU, 512-atom Si-like, "
          "ΔE≤1e-6 Ha/atom")
WORKLOAD = ("si512: 512-atom Si-like diamond cell a=41.04 bohr, Gamma, 25 Ry, "
            "1024 bands, PBE, 140^3 grid, 72919 PW/band")


def dist_env():
    from qbx import replicas
    return replicas.dist_env()


# ---------------------------------------------------------------- clocks
class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled every 200 ms."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device: int):
        self.device = device
        self.proc = None
        self.out = tempfile.NamedTemporaryFile("w+", suffix=".csv", delete=False)

    def start(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.device), f"--query-gpu={self.FIELDS}",
                 "--format=csv,noheader,nounits", "-lms", "200"],
                stdout=self.out, stderr=subprocess.DEVNULL)
        except OSError:
            self.proc = None

    def stop(self):
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        self.out.flush()
        self.out.seek(0)
        sm, smax, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in self.out.read().splitlines():
            f = [x.strip() for x in line.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                smax.append(float(f[2]))
            except ValueError:
                continue
            for name, val in zip(names, f[5:9]):
                if val.lower() == "active":
                    reasons.add(name)
        os.unlink(self.out.name)
        return {"sm_mhz": statistics.median(sm) if sm else None,
                "sm_max_mhz": max(smax) if smax else None,
                "reasons": sorted(reasons), "samples": len(sm)}


# ---------------------------------------------------------- reference arm
def reference_step_ms(nsteps: int, nbands_sample: int, threads: int):
    """Time the reference (oracle/_ref) on a band sample of si512 and scale
    each phase to 1024 bands: density and H*psi linearly in the bands (FFTs
    and nonlocal projections), the PSDA update quadratically (band-band
    GEMMs), update_vhxc not at all."""
    from qbx import systems
    from oracle import inputs
    full = systems.si512()
    s = full.band_sample(nbands_sample)
    with tempfile.TemporaryDirectory() as td:
        out = inputs.run_reference(s, td, nsteps, threads=threads)
    e = out["energies"]
    k = max(1, nsteps - 1)              # the first step carries warm-up costs
    tc = statistics.median(e["t_charge"][-k:])
    tv = statistics.median(e["t_vhxc"][-k:])
    te = statistics.median(e["t_energy"][-k:])
    tw = statistics.median(e["t_wf_update"][-k:])
    f = full.nbands / nbands_sample
    ms = 1e3 * (tc * f + tv + te * f + tw * f * f)
    sample = (f"{nbands_sample} of {full.nbands} bands of si512 for {nsteps} steps, "
              f"median of the last {k}; per-phase scaling to 1024 bands "
              f"(density {tc:.2f}s, vhxc {tv:.2f}s, energy {te:.2f}s, "
              f"wf_update {tw:.2f}s per sample step)")
    return ms, sample


def host_threads() -> int:
    try:
        return len(os.sched_getaffinity(0))
    except AttributeError:
        return os.cpu_count() or 1


def _full_step_cache() -> str:
    """Where the reference arm leaves its full-step measurement for the
    cpu_baseline leg of the next run on the same machine boot."""
    try:
        boot = open("/proc/sys/kernel/random/boot_id").read().strip()
    except OSError:
        boot = "unknown"
    return os.path.join(tempfile.gettempdir(), f"qbx_reference_si512_step_{boot}.json")


def reference_full_step(threads: int):
    """One electronic step of the whole si512 workload (all 1024 bands) on
    the reference's own CPU build (oracle/_ref/ref_driver): the sum of its
    timers for update_density, update_vhxc, energy(true) and the PSDA update
    (src/BOSampleStepper.cpp:795-977 with nite=0).  Measured, not scaled."""
    from qbx import systems
    from oracle import inputs
    s = systems.si512()
    t0 = time.time()
    with tempfile.TemporaryDirectory() as td:
        out = inputs.run_reference(s, td, 1, threads=threads)
    wall = time.time() - t0
    e = out["energies"]
    phases = {k: float(e[k][0]) for k in ("t_charge", "t_vhxc", "t_energy", "t_wf_update")}
    ms = 1e3 * sum(phases.values())
    return ms, phases, wall


def run_reference_arm(args):
    rank, world, _ = dist_env()
    if rank != 0:
        return
    threads = host_threads()
    ref = os.path.join(ROOT, "oracle", "_ref", "ref_driver")
    if not os.path.exists(ref):
        print(json.dumps({"impl": "reference",
                          "unavailable": "oracle/_ref/ref_driver not built (make -C oracle)"}))
        return
    ms, phases, wall = reference_full_step(threads)
    try:
        with open(_full_step_cache(), "w") as f:
            json.dump({"ms": ms, "cores": threads, "phases_s": phases}, f)
    except OSError:
        pass
    sample = (f"one full electronic step of si512 (all 1024 bands, 140^3 grid, PBE): "
              f"update_density {phases['t_charge']:.1f} s, update_vhxc {phases['t_vhxc']:.1f} s, "
              f"energy {phases['t_energy']:.1f} s, PSDA update {phases['t_wf_update']:.1f} s; "
              f"{wall:.0f} s with set-up; one step only (--steps {args.steps} not repeated: "
              f"a step takes minutes)")
    line = {
        "metric": METRIC, "value": ms, "unit": "ms", "n_gpus": world, "steps": 1,
        "warmup": 0, "ms_per_step": ms, "higher_is_better": False,
        "scaling": "strong" if args.shard else "weak", "vs_baseline": None, "dtype": "f64",
        "data": "synthetic",
        "impl": "reference",
        "config": bench_config(world, args.shard),
        "precision": "FP64 (the reference's CPU build, single task, OpenMP + OpenBLAS threads)",
        "steps_requested": args.steps, "warmup_requested": args.warmup,
        "cpu_baseline": {"value": ms, "unit": "ms", "cores": threads, "kind": "reference",
                         "sample": sample},
        "e2e": {"value": ms, "unit": "ms", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line))


def bench_config(world: int, shard: bool = False) -> dict:
    """The workload both arms run (identical in both JSON lines)."""
    par = "single GPU"
    if world > 1:
        par = f"band pairs sharded over {world} GPUs" if shard else "replicas"
    return {"workload": WORKLOAD,
            "l2": "inputs larger than L2 (1.19 GB wavefunctions per step)",
            "parallelism": par}


# ------------------------------------------------------------ our arm
def algorithmic_bytes_xy_vpsi(ctx, npairs: int, nlaunch: float, cbytes: int, vbytes: int) -> float:
    """Per H*psi, the x pass (pen::xv: x transform, times V(r), x transform
    back, in place): every band pair's tile of occupied columns read once and
    written once, and the potential read once per launch (N v bytes)."""
    n0, n1, n2 = ctx.grid
    ncol = 2 * int(max(h for h, _, _ in ctx.miller())) + 1
    return npairs * 2.0 * ncol * n1 * n2 * cbytes + nlaunch * float(vbytes) * n0 * n1 * n2


def run_ours(args):
    import numpy as np
    import torch
    from qbx import capi, systems

    from qbx import replicas
    rank, world, local = dist_env()
    torch.cuda.set_device(local)
    replicas.init("nccl")
    dev = local

    s = systems.si512()
    hkl = s.miller()
    c0 = s.coefficients(hkl)
    natoms = len(s.atoms)

    def timed(ctx, nsteps, profile=False, e2e_bufs=None):
        stream = torch.cuda.ExternalStream(ctx.stream(), device=dev)
        start = torch.cuda.Event(enable_timing=True)
        end = torch.cuda.Event(enable_timing=True)
        replicas.barrier(device=f"cuda:{dev}")
        torch.cuda.synchronize()
        if profile:
            ctx.profile(True)
        n0 = ctx.launch_count()
        start.record(stream)
        r = None
        if e2e_bufs is not None:
            # the streamed SlaterDet: each step uploads its input from pinned
            # host memory and downloads its result, the copies on their own
            # streams overlapping the neighbouring steps' compute
            for _ in range(nsteps):
                ctx.stream_in(e2e_bufs[0])
                ctx.scf_step_async()
                ctx.stream_out(e2e_bufs[1])
            r = ctx.stream_wait()
        else:
            for _ in range(nsteps):
                r = ctx.scf_step()
        end.record(stream)
        end.synchronize()
        torch.cuda.synchronize()
        replicas.barrier(device=f"cuda:{dev}")
        ms = start.elapsed_time(end) / nsteps
        launches = ctx.launch_count() - n0
        return ms, r, launches

    def max_over_ranks(x):
        return replicas.max_over_ranks(x, device=f"cuda:{dev}")

    sharded = args.shard and world > 1

    def maybe_shard(ctx):
        # --shard: the band pairs of the one cell split over the ranks (NCCL
        # allreduce of the density, broadcast of the H*psi blocks); the
        # sharded step runs eagerly
        if sharded:
            from qbx import sharding
            sharding.shard_band_pairs(ctx, device=f"cuda:{dev}")
        else:
            ctx.set_step_graph(True)

    # ---- mixed precision (headline)
    mix = capi.from_system(s, device=dev, precision=capi.MIXED, coeffs=c0)
    mix.scf_step()
    tuning_mix = mix.autotune()
    # the step runs as a captured CUDA graph (captured during the warm-up)
    maybe_shard(mix)
    for _ in range(args.warmup):
        mix.scf_step()
    clocks = ClockSampler(dev)
    clocks.start()
    ms_mix, r_mix, launches = timed(mix, args.steps)
    clk = clocks.stop()
    graphs, graph_launches, graph_note = mix.step_graph_info()
    # per-region breakdown: the same step eagerly under the CUDA-event profiler
    ms_mix_eager, _, _ = timed(mix, args.steps, profile=True)
    prof = {}
    for name in ("update_density", "update_vhxc", "energy", "vpsi", "psda_update",
                 "xy_vpsi", "xy_density", "zfft_bwd", "zfft_fwd", "grid_fft",
                 "gemm_nl_project", "gemm_nl_apply", "gemm_residual", "overlap_cholesky",
                 "gemm_overlap_last", "gemm_rotate", "polar"):
        t, n = mix.profile_get(name)
        prof[name] = {"ms_per_step": t / args.steps, "launches_per_step": n / args.steps}
    mix.profile(False)
    npairs = (s.nbands + 1) // 2
    # the x pass takes all band pairs in one launch
    t_xy, n_xy = prof["xy_vpsi"]["ms_per_step"], prof["xy_vpsi"]["launches_per_step"]
    bytes_hpsi = algorithmic_bytes_xy_vpsi(mix, npairs, n_xy, 8, 8)
    per_launch_bytes = bytes_hpsi / max(1e-9, n_xy)
    per_launch_ms = t_xy / max(1e-9, n_xy)
    peaks = {}
    try:
        peaks = json.load(open(os.path.join(ROOT, "MEASURED_PEAKS.json")))
    except (OSError, ValueError):
        pass
    hbm_peak = peaks.get("hbm_gbs", 6650.0)
    achieved = per_launch_bytes / (per_launch_ms * 1e-3) / 1e9
    roofline = {"kernel": "pen::xv<float, 140> (H*psi x pass: x transform of the tiles kept "
                          "from the density pass, times V, transform back in place)",
                "bound": "issue",   # 60 % of the slots; DRAM at 31 % (profiles/)
                "achieved": achieved, "peak": hbm_peak, "unit": "GB/s",
                "frac": achieved / hbm_peak,
                "peak_source": "measured" if "hbm_gbs" in peaks else "fallback",
                # DRAM bytes of the ncu capture (profiles/fft_pencil_si512.md:
                # 645.7 MB for 32 band pairs) scaled by the band pairs
                "traffic": 645.7e6 / 32.0 * (npairs / max(1e-9, n_xy)),
                "algorithmic_bytes_per_launch": per_launch_bytes,
                "launch_ms": per_launch_ms}
    # GEMM share: the split-precision products of the mixed step (BF16 and
    # TF32 splits on the tcgen05 kernel) and the FP64 Cholesky
    gemm_ms = sum(prof[k]["ms_per_step"] for k in
                  ("gemm_nl_project", "gemm_nl_apply", "gemm_residual", "overlap_cholesky",
                   "gemm_overlap_last", "gemm_rotate"))
    K = 2 * mix.ngw
    n = s.nbands
    npj = 4 * natoms
    gemm_flop = 2 * (2.0 * K * npj * n) + 2 * (2.0 * K * n * n) + K * n * n + 2 * (2.0 * K * n * n)

    # ---- FP64 path on the same start
    f64 = capi.from_system(s, device=dev, precision=capi.FP64, coeffs=c0)
    f64.scf_step()
    f64.autotune()
    maybe_shard(f64)
    for _ in range(args.warmup):
        f64.scf_step()
    ms_f64, r_f64, _ = timed(f64, args.steps)
    de_traj = abs(r_mix["etotal"] - r_f64["etotal"]) / natoms
    # the error of one mixed step: both paths evaluate the same coefficients
    # (the FP64 trajectory's current ones)
    c_ref = f64.get_coeffs()
    mix.set_coeffs(c_ref)
    e_mix_same = mix.scf_step()["etotal"]
    e_f64_same = f64.scf_step()["etotal"]
    de_atom = abs(e_mix_same - e_f64_same) / natoms
    f64.close()

    # ---- end to end through the C ABI with pinned host buffers
    nb = 2 * mix.ngw * s.nbands * 8
    pin_in = torch.empty(nb // 8, dtype=torch.float64, pin_memory=True)
    pin_out = torch.empty(nb // 8, dtype=torch.float64, pin_memory=True)
    cur = mix.get_coeffs()
    pin_in.numpy()[:] = cur.view(np.float64).ravel()
    # two streamed steps per timed step, at most 40: the first upload and the
    # last download have no neighbouring step to overlap (about 43 ms in
    # all), and over more steps that fill and drain weighs less per step
    ne2e = max(2, min(2 * args.steps, 40))
    # warm-up of the streamed path: its first call allocates the device
    # staging buffers (2 x 1.19 GB) and the copy streams
    for _ in range(2):
        mix.stream_in(pin_in.numpy())
        mix.scf_step_async()
        mix.stream_out(pin_out.numpy())
    mix.stream_wait()
    ms_e2e, _, _ = timed(mix, ne2e, e2e_bufs=(pin_in.numpy(), pin_out.numpy()))
    # the host link alone: one copy of the same bytes each way (the end-to-end
    # step cannot be faster than the slower direction)
    link = {}
    dev_buf = torch.empty(nb // 8, dtype=torch.float64, device=f"cuda:{dev}")
    for name, (dst, src) in (("h2d_gbs", (dev_buf, pin_in)), ("d2h_gbs", (pin_out, dev_buf))):
        c0 = torch.cuda.Event(enable_timing=True)
        c1 = torch.cuda.Event(enable_timing=True)
        dst.copy_(src, non_blocking=True)
        c0.record()
        dst.copy_(src, non_blocking=True)
        c1.record()
        c1.synchronize()
        link[name] = nb / (c0.elapsed_time(c1) * 1e-3) / 1e9
    # both directions at once, as the streamed steps run them
    dev_buf2 = torch.empty_like(dev_buf)
    s_up, s_down = torch.cuda.Stream(), torch.cuda.Stream()
    c0 = torch.cuda.Event(enable_timing=True)
    c1 = torch.cuda.Event(enable_timing=True)
    c0.record()
    s_up.wait_event(c0)
    s_down.wait_event(c0)
    with torch.cuda.stream(s_up):
        dev_buf.copy_(pin_in, non_blocking=True)
    with torch.cuda.stream(s_down):
        pin_out.copy_(dev_buf2, non_blocking=True)
    torch.cuda.current_stream().wait_stream(s_up)
    torch.cuda.current_stream().wait_stream(s_down)
    c1.record()
    c1.synchronize()
    both_ms = c0.elapsed_time(c1)
    link["both_directions_gbs"] = 2 * nb / (both_ms * 1e-3) / 1e9
    del dev_buf, dev_buf2

    # ---- molecular dynamics of the same cell (dt = 20 a.u., forces every
    # ionic step, captured electronic steps): ms per ionic step, and the same
    # ionic steps in FP64 from the same coefficients and positions
    md = None
    if args.md_steps > 0:
        masses = [sp.mass for sp in s.species]
        c_md = mix.get_coeffs()
        mix.psda_reset()          # both runs start without PSDA history

        def md_leg(ctx):
            w = ctx.md_run(1, args.md_nitscf, 20.0, masses)          # warm-up (captures)
            st = torch.cuda.ExternalStream(ctx.stream(), device=dev)
            e0 = torch.cuda.Event(enable_timing=True)
            e1 = torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            e0.record(st)
            o = ctx.md_run(args.md_steps, args.md_nitscf, 20.0, masses, vel=w["velocities"])
            e1.record(st)
            e1.synchronize()
            return e0.elapsed_time(e1) / args.md_steps, o

        ms_md, out_md = md_leg(mix)
        f64md = capi.from_system(s, device=dev, precision=capi.FP64, coeffs=c_md, gram=False)
        maybe_shard(f64md)
        ms_md64, out_md64 = md_leg(f64md)
        f64md.close()
        ec = out_md["ionic"][:, 2]
        ec64 = out_md64["ionic"][:, 2]
        md = {"ionic_steps": args.md_steps, "scf_steps_per_ionic_step": args.md_nitscf,
              "dt_au": 20.0, "ms_per_ionic_step": ms_md,
              "fp64_ms_per_ionic_step": ms_md64,
              "econst": [float(x) for x in ec],
              "econst_fp64": [float(x) for x in ec64],
              "econst_drift_per_atom": float(ec[-1] - ec[0]) / natoms,
              "econst_drift_per_atom_fp64": float(ec64[-1] - ec64[0]) / natoms,
              "max_dE_mixed_vs_fp64_per_atom": float(np.abs(ec - ec64).max()) / natoms,
              "max_dtau_mixed_vs_fp64_bohr": float(np.abs(out_md["positions"]
                                                          - out_md64["positions"]).max()),
              "profile_ms_one_ionic_step": None,
              "what": ("per ionic step: density, potential, energy and forces; velocity "
                       "Verlet; atoms_moved; linear wavefunction extrapolation (align, "
                       "lowdin); scf_steps_per_ionic_step captured electronic steps. Both "
                       "runs start from the same coefficients and positions (one untimed "
                       "ionic step each, then the timed steps); with one electronic step "
                       "per ionic step from unconverged wavefunctions econst is not "
                       "conserved, and the FP64 run shows the drift that is not precision")}
        # where one (eager, profiled) ionic step goes
        mix.profile(True)
        mix.md_run(1, args.md_nitscf, 20.0, masses)
        md["profile_ms_one_ionic_step"] = {
            k: mix.profile_get(k)[0] for k in ("md_forces", "md_move_atoms", "md_extrapolate",
                                               "update_density", "energy", "psda_update")}
        mix.profile(False)
    mix.close()

    # ---- the 32-system batch (small cells of uneven size), split over the
    # ranks, captured steps launched together (qbx_scf_step_batch)
    batch = None
    if args.batch_steps > 0:
        systs = systems.batch()
        mine = [systs[i] for i in replicas.shard(len(systs), rank, world)]
        bctx = [capi.from_system(x, device=dev, precision=capi.MIXED) for x in mine]
        for c in bctx:
            c.set_step_graph(True)
        for _ in range(3):
            capi.scf_step_batch(bctx)          # first use, capture, warm
        torch.cuda.synchronize()
        replicas.barrier(device=f"cuda:{dev}")
        b0 = torch.cuda.Event(enable_timing=True)
        b1 = torch.cuda.Event(enable_timing=True)
        b0.record()
        for _ in range(args.batch_steps):
            capi.scf_step_batch(bctx)          # returns when every system is done
        b1.record()
        b1.synchronize()
        bms = b0.elapsed_time(b1) / args.batch_steps
        seq0 = torch.cuda.Event(enable_timing=True)
        seq1 = torch.cuda.Event(enable_timing=True)
        seq0.record()
        for c in bctx:
            c.scf_step()
        seq1.record()
        seq1.synchronize()
        batch = {"systems": len(systs), "systems_this_rank": len(mine),
                 "ms_per_batched_step": bms,
                 "ms_one_after_another": seq0.elapsed_time(seq1),
                 "what": ("one mixed electronic step of each system (8-64 atoms, 20-30 Ry, "
                          "bands = 2 x atoms), captured steps launched on one stream each")}
        for c in bctx:
            c.close()
        replicas.barrier(device=f"cuda:{dev}")

    # ---- k points off Gamma: si64 at two k points (complex bases, FP64),
    # ms per electronic step, beside the reference's own time for one step
    kpts = None
    if args.kpoint_steps > 0:
        sk = systems.si64k2()
        kc = capi.from_system(sk, device=dev, precision=capi.FP64)
        for _ in range(2):
            kc.scf_step()
        stream = torch.cuda.ExternalStream(kc.stream(), device=dev)
        k0 = torch.cuda.Event(enable_timing=True)
        k1 = torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        k0.record(stream)
        for _ in range(args.kpoint_steps):
            ek = kc.scf_step()
        k1.record(stream)
        k1.synchronize()
        kpts = {"system": "si64 (PBE, 30 Ry, 128 bands) at k = (1/4,1/4,1/4), (-1/4,1/4,1/4), "
                          "weights 1/2",
                "ngw_per_kpoint": list(kc.kngw), "precision": "fp64",
                "ms_per_step": max_over_ranks(k0.elapsed_time(k1) / args.kpoint_steps),
                "etotal_last": ek["etotal"], "reference_ms_per_step": None}
        kc.close()

    ms_mix = max_over_ranks(ms_mix)
    ms_f64 = max_over_ranks(ms_f64)
    ms_e2e = max_over_ranks(ms_e2e)
    if batch is not None:
        batch["ms_per_batched_step"] = max_over_ranks(batch["ms_per_batched_step"])
        batch["ms_one_after_another"] = max_over_ranks(batch["ms_one_after_another"])

    if rank == 0:
        cpu = None
        if os.environ.get("QBX_BENCH_NO_CPU") != "1":
            ref = os.path.join(ROOT, "oracle", "_ref", "ref_driver")
            threads = host_threads()
            cached = None
            try:
                cached = json.load(open(_full_step_cache()))
            except (OSError, ValueError):
                pass
            if cached and cached.get("cores") == threads:
                # the reference arm ran on this machine since its last boot:
                # its measured full step (all 1024 bands) is the baseline
                cpu = {"value": cached["ms"], "unit": "ms", "cores": threads,
                       "kind": "reference",
                       "sample": "one full 1024-band si512 step of the reference's CPU build, "
                                 "measured by `bench.py --impl reference` on this machine"}
            elif os.path.exists(ref):
                cms, sample = reference_step_ms(2, 32, threads)
                cpu = {"value": cms, "unit": "ms", "cores": threads, "kind": "reference",
                       "sample": "modelled (no full-step measurement on this machine): " + sample}
        if kpts is not None and cpu is not None:
            # the reference's own k-point step on the host cores (one step,
            # the sum of its timed phases)
            from oracle import inputs
            with tempfile.TemporaryDirectory() as td:
                out = inputs.run_reference(systems.si64k2(), td, 1, threads=cpu["cores"])
            e = out["energies"]
            kpts["reference_ms_per_step"] = 1e3 * float(
                e["t_charge"][0] + e["t_vhxc"][0] + e["t_energy"][0] + e["t_wf_update"][0])
            kpts["reference_cores"] = cpu["cores"]
        line = {
            "metric": METRIC, "value": ms_mix, "unit": "ms", "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms_mix,
            "higher_is_better": False, "scaling": "strong" if sharded else "weak",
            "vs_baseline": None,
            "dtype": ("mixed: FP32 FFTs and real-space work; BF16x3 (inner products) and "
                      "TF32x3 (rotation) split products on tcgen05 with FP32 accumulation; "
                      "FP64 Cholesky, polar, phases and reductions"),
            "data": "synthetic",
            "config": bench_config(world, sharded),
            "precision": "mixed",
            "step_graph": {"captured": graphs, "launches": graph_launches, "note": graph_note,
                           "eager_ms_per_step": ms_mix_eager},
            "md": md,
            "batch": batch,
            "kpoints": kpts,
            "dE_definition": ("|E_mixed - E_fp64| / atoms for one electronic step of both paths "
                              "from the same coefficients (the FP64 trajectory's after "
                              "warm-up + timed steps)"),
            "etotal_mixed": e_mix_same, "etotal_fp64": e_f64_same,
            "dE_trajectory_per_atom": de_traj,
            "roofline": roofline,
            "gemm": {"ms_per_step": gemm_ms, "flop_per_step": gemm_flop,
                     "tflops": gemm_flop / (gemm_ms * 1e-3) / 1e12 if gemm_ms else None,
                     "precision": "mixed: split BF16 (inner products) and TF32 (tall updates) "
                                  "on tcgen05, FP64 Cholesky/polar (cuSOLVER/cuBLAS)"},
            "profile": prof,
            "fft_tuning": tuning_mix.strip().splitlines()[-1],
            "cpu_baseline": cpu,
            "e2e": {"value": ms_e2e, "unit": "ms", "h2d_bytes_per_step": nb,
                    "d2h_bytes_per_step": nb,
                    "host_link": {k: round(v, 1) for k, v in link.items()},
                    # a step's upload and download over the link, run together
                    "copy_floor_ms": max(nb / (min(link["h2d_gbs"], link["d2h_gbs"]) * 1e9),
                                         2 * nb / (link["both_directions_gbs"] * 1e9)) * 1e3},
            "gpu_launches": launches,
            "clocks": clk,
        }
        # the headline comparison last, where a truncated log keeps it
        line["fp64_ms_per_step"] = ms_f64
        line["mixed_vs_fp64_speedup"] = ms_f64 / ms_mix
        line["dE_per_atom"] = de_atom
        line["dE_ok"] = bool(de_atom <= 1e-6)
        print(json.dumps(line))
    replicas.finalize()


def run_profile_case(args):
    """A case for ncu: the 512-atom cell with a band sample (all 1024 bands
    for the launch list of the headline step; 64 for full captures, whose
    kernels do the same work per band pair while the device holds a few
    GB), mixed precision.  Warm-up steps run before cudaProfilerStart, so
    `ncu --profile-from-start off` sees exactly one electronic step."""
    import torch
    from qbx import capi, systems
    s = systems.si512()
    if args.profile_bands < s.nbands:
        s = s.band_sample(args.profile_bands)
    ctx = capi.from_system(s, precision=capi.MIXED)
    ctx.scf_step()
    if args.profile_tune:
        ctx.autotune()
    if args.profile_graph:
        ctx.set_step_graph(True)     # the profiled step is the captured graph
    for _ in range(args.warmup):
        ctx.scf_step()
    ctx.synchronize()
    torch.cuda.profiler.start()
    ctx.scf_step()
    ctx.synchronize()
    torch.cuda.profiler.stop()
    ctx.close()


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--md-steps", type=int, default=10,
                    help="ionic steps of the molecular-dynamics measurement (0: skip)")
    ap.add_argument("--md-nitscf", type=int, default=1,
                    help="electronic steps per ionic step in the MD measurement")
    ap.add_argument("--batch-steps", type=int, default=3,
                    help="timed steps of the 32-system batch measurement (0: skip)")
    ap.add_argument("--kpoint-steps", type=int, default=3,
                    help="timed steps of the two-k-point si64 measurement (0: skip)")
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--shard", action="store_true",
                    help="with several GPUs: split the band pairs of the one cell over them "
                         "(strong scaling) instead of running independent replicas")
    ap.add_argument("--profile-bands", type=int, default=0,
                    help="run only warm-up + one mixed step of si512 with this many bands "
                         "(a case for profilers); prints nothing")
    ap.add_argument("--profile-tune", action="store_true",
                    help="with --profile-bands: autotune the FFT configuration first")
    ap.add_argument("--profile-graph", action="store_true",
                    help="with --profile-bands: profile the captured step (graph launch)")
    args = ap.parse_args()
    if args.profile_bands:
        run_profile_case(args)
        return
    if args.warmup < 3:
        args.warmup = 3
    if args.impl == "reference":
        run_reference_arm(args)
    else:
        run_ours(args)


if __name__ == "__main__":
    main()
