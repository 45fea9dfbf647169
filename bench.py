"""Benchmark: w-projection gridding + degridding throughput (Mvis/s) on one GB300.

Workload (default): the 4,177,920-visibility w-projection observation
(256 log-radial antennas, 32,640 baselines x 128 time samples, 4096^2
complex64 grid, 32 w-planes with supports 8..64, oversample 8, w-kernels
generated on the GPU in FP64 and cast to complex64), seeded synthetic data.

One step = one gridding pass (zero the grid, grid every visibility) plus one
degridding pass (predict every visibility from a model grid) through the
FP32 tiled adjoint pair, replayed from a CUDA graph, inputs resident in HBM,
L2 flushed (a 256 MiB write) before every step.  Reported next to it: the
plain FP64 GPU path, the FP32 error against it, the HBM roofline of the
dominant kernel, an end-to-end figure with host buffers, and the CPU
restatement of the reference's gridder timed on the host cores.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
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

METRIC = "Mvis/s grid+degrid, FP32 batched vs FP64 plain at stated err; % HBM roofline"
L2_BYTES = 129 * 1024 * 1024

# The roofline's algorithmic bytes follow the unfused per-tap model (a record
# per visibility, and per tap one GCF element plus the grid element read and
# written, or read): the tiled kernels reuse the staged tile and GCF on chip,
# so frac can exceed 1; `traffic` is the kernel's measured DRAM bytes.
ROOFLINE_MODEL = ("unfused per-tap bytes (grid 32 + 24 S^2, degrid 40 + 16 S^2 per visibility); "
                  "on-chip reuse not credited; DRAM bytes per launch in traffic")


def measured_peaks():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    try:
        d = json.load(open(p))
        return float(d["hbm_gbs"]), "measured"
    except Exception:
        return 6800.0, "fallback"


class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled during the timed region."""

    Q = ("clocks.sm,clocks.max.sm,clocks_event_reasons.hw_slowdown,"
         "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
         "clocks_event_reasons.sw_power_cap")

    def __init__(self, index=0):
        self.index = index
        self.proc = None
        self.lines = []

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.index), f"--query-gpu={self.Q}",
                 "--format=csv,noheader,nounits", "-lms", "20"],
                stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except Exception:
            self.proc = None
        return self

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def __exit__(self, *a):
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                self.proc.kill()

    def summary(self):
        sm, mx, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            f = [x.strip() for x in ln.split(",")]
            if len(f) < 6:
                continue
            try:
                sm.append(float(f[0]))
                mx.append(float(f[1]))
            except ValueError:
                continue
            for k, nm in enumerate(names):
                if f[2 + k].lower().startswith("active"):
                    reasons.add(nm)
        if not sm:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": [], "samples": 0}
        return {"sm_mhz": float(np.median(sm)), "sm_max_mhz": float(max(mx)),
                "reasons": sorted(reasons), "samples": len(sm)}


# ---------------------------------------------------------------- workload
def load_workload(name):
    from rc_gb300 import synth

    return synth.config(name)


def cpu_leg(ob, supports, gcf128_np, offs, sample_n, nthreads):
    """The reference's CPU gridder semantics (the oracle's FP64 restatement,
    multi-plane, per-thread grids as MS4's OpenMP gridder does) on the first
    sample_n visibilities: grid, then degrid from the gridded result."""
    from oracle import oracle as O

    n = ob.n if sample_n <= 0 else min(sample_n, ob.n)
    uvw = np.ascontiguousarray(ob.uvw[:n])
    vis = np.ascontiguousarray(ob.vis[:n])
    plane = O.wbin(uvw, ob.w_low, ob.w_high, ob.n_planes)
    G = ob.grid_size
    grid = np.zeros((G, G), np.complex128)
    t0 = time.perf_counter()
    used = O.scatter_planes(ob.scale, G, int(supports.max()), uvw, vis, plane, supports,
                            gcf128_np, offs, grid, nthreads=nthreads)
    t1 = time.perf_counter()
    O.degrid_planes(ob.scale, G, int(supports.max()), uvw, plane, supports, gcf128_np, offs, grid,
                    mode=0, nthreads=nthreads)
    t2 = time.perf_counter()
    return n, (t2 - t0), used, (t1 - t0), (t2 - t1)


_CPU_CHILD = r"""
import json, os, sys, time
import numpy as np
sys.path.insert(0, sys.argv[1])
from oracle import oracle as O
d = np.load(sys.argv[2])
uvw, vis, sup, gcf, offs = d["uvw"], d["vis"], d["sup"], d["gcf"], d["offs"]
scale, G, lo, hi, npl = float(d["scale"]), int(d["G"]), float(d["lo"]), float(d["hi"]), int(d["npl"])
nth = os.cpu_count() or 1
plane = O.wbin(uvw, lo, hi, npl)
def leg(n):
    grid = np.zeros((G, G), np.complex128)
    t0 = time.perf_counter()
    used = O.scatter_planes(scale, G, int(sup.max()), uvw[:n], vis[:n], plane[:n], sup, gcf, offs,
                            grid, nthreads=nth)
    O.degrid_planes(scale, G, int(sup.max()), uvw[:n], plane[:n], sup, gcf, offs, grid, mode=0,
                    nthreads=nth)
    return time.perf_counter() - t0, used
leg(min(len(vis), 50000))
runs = [leg(len(vis)) for _ in range(2)]
print(json.dumps({"n": int(len(vis)), "dt": float(np.mean([r[0] for r in runs])),
                  "used": int(runs[0][1])}))
"""


def cpu_leg_isolated(ob, gcf128_np, offs, sample_n):
    """cpu_leg in a fresh interpreter that loads only numpy and the oracle:
    inside the bench process the CUDA and torch runtimes compete with the
    oracle's OpenMP threads for the host cores."""
    import tempfile

    n = ob.n if sample_n <= 0 else min(sample_n, ob.n)
    with tempfile.TemporaryDirectory() as d:
        path = os.path.join(d, "sample.npz")
        np.savez(path, uvw=np.ascontiguousarray(ob.uvw[:n]), vis=np.ascontiguousarray(ob.vis[:n]),
                 sup=ob.supports, gcf=gcf128_np, offs=offs, scale=ob.scale, G=ob.grid_size,
                 lo=ob.w_low, hi=ob.w_high, npl=ob.n_planes)
        r = subprocess.run([sys.executable, "-c", _CPU_CHILD, ROOT, path], capture_output=True,
                           text=True, check=True)
    out = json.loads(r.stdout.strip().splitlines()[-1])
    return out["n"], out["dt"], out["used"]


def _oracle_taps(ob, n):
    """Sum of S_v^2 over the first n visibilities that the reference's bounds
    rule keeps, by the oracle's index rule (for the reference arm's line)."""
    from oracle import oracle as O

    plane = O.wbin(ob.uvw[:n], ob.w_low, ob.w_high, ob.n_planes)
    taps = 0
    for p, S in enumerate(ob.supports):
        m = plane == p
        if not m.any():
            continue
        rec = np.zeros((int(m.sum()), 5))
        rec[:, :3] = ob.uvw[:n][m]
        idx = O.index(rec, ob.scale, ob.grid_size, int(S), int(ob.supports.max()),
                      ext_x=ob.grid_size, ext_y=ob.grid_size)
        taps += int(idx[:, 4].sum()) * int(S) * int(S)
    return taps


def reference_arm(args):
    """--impl reference: the reference's CPU gridding path (its semantics
    restated in C, FP64, all host threads) on this workload's whole
    observation; the reference's own kernels are Halide generators that cannot
    be built here."""
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return 0
    from rc_gb300 import gcf as Gm

    ob = load_workload(args.config)
    offs, total = Gm.layout(ob.supports)
    gcf = _gcf_host(ob)
    nthreads = os.cpu_count() or 1
    sample_n = args.cpu_sample
    if args.warmup > 0:
        cpu_leg(ob, ob.supports, gcf, offs, min(ob.n, 50000), nthreads)
    times = []
    for _ in range(args.steps):
        n, dt, used, _, _ = cpu_leg(ob, ob.supports, gcf, offs, sample_n, nthreads)
        times.append(dt)
    t = float(np.mean(times))
    val = n / t / 1e6
    taps = _oracle_taps(ob, n)
    what = "the whole observation" if n == ob.n else f"first {n} of {ob.n} visibilities"
    line = {
        "metric": METRIC, "impl": "reference", "value": round(val, 3), "unit": "Mvis/s",
        "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": round(1e3 * t, 3), "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f64", "data": "synthetic (seeded)",
        "config": {"workload": _workload_desc(ob), "sample_visibilities": n, "taps": taps},
        "cpu_baseline": {"value": round(val, 3), "unit": "Mvis/s", "cores": used, "kind": "port",
                         "taps": taps, "gtaps_per_s": round(2 * taps / t / 1e9, 3),
                         "sample": f"{what}, grid + degrid, FP64"},
        "e2e": {"value": round(val, 3), "unit": "Mvis/s", "h2d_bytes_per_step": 0,
                "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line))
    return 0


def _workload_desc(ob):
    return (f"{ob.name}: {ob.n} vis, {ob.grid_size}^2 grid, {ob.n_planes} w-planes "
            f"S {int(ob.supports.min())}-{int(ob.supports.max())}, oversample 8")


_GCF_CACHE = {}


def _gcf_host(ob):
    """complex128 GCFs for the reference arm, from the numpy restatement of the
    reference's generator (no engine code on that arm)."""
    key = ob.name
    if key in _GCF_CACHE:
        return _GCF_CACHE[key]
    from oracle import oracle as O
    from rc_gb300 import gcf as Gm

    tp = Gm.pswf_taper(ob.max_support)
    out = np.concatenate([O.gcf_layers(w, int(S), ob.max_support, ob.scale / 2, taper=tp).ravel()
                          for w, S in zip(ob.w_planes, ob.supports)])
    _GCF_CACHE[key] = out
    return out


# ---------------------------------------------------------------- our arm
def abi_e2e(ob, steps, warmup):
    """Config 1 through the reference's own host-buffer symbols, the way the
    MS6 Haskell gridder calls them (MS6/programs/Kernel/Gridder.hs:58-71,
    Degrid.hs:146-155): one kern_scatter_gpu1 and one kern_degrid_gpu1 per
    (tile, w-bin), and config 1 has one of each.  FP64 5-double records, the
    7 x 7 PSWF in S = 8, a complex128 grid in pageable host memory; every copy
    is inside the call.  Each step grids into a zeroed grid (zeroed outside the
    timer) and degrids from the result.  Returns the e2e object."""
    from rc_gb300 import compat
    from rc_gb300 import gcf as Gm

    vis5 = ob.vis5()
    S, G = 8, ob.grid_size
    gcf = Gm.pswf_uv_gcf(S, 7)
    grid = np.zeros((G, G), np.complex128)
    out = np.zeros_like(vis5)
    times = []
    for i in range(warmup + steps):
        grid.fill(0)
        t0 = time.perf_counter()
        rc1 = compat.call_scatter("kern_scatter_gpu1", ob.scale, G, S, vis5, gcf, grid)
        rc2 = compat.call_degrid("kern_degrid_gpu1", ob.scale, G, S, gcf, grid, vis5, out)
        t1 = time.perf_counter()
        assert rc1 == 0 and rc2 == 0, (rc1, rc2)
        if i >= warmup:
            times.append(t1 - t0)
    t = float(np.mean(times))
    n, gcf_b, grid_b = ob.n, gcf.size * 16, G * G * 16
    return {"value": round(n / t / 1e6, 3), "unit": "Mvis/s", "ms_per_step": round(1e3 * t, 3),
            "h2d_bytes_per_step": 2 * (40 * n + gcf_b + grid_b),
            "d2h_bytes_per_step": grid_b + 40 * n,
            "path": "kern_scatter_gpu1 + kern_degrid_gpu1 on pageable host buffer_t (FP64), "
                    "host wall clock per step, mean of K after W"}


def abi_strategy_e2e(ob, args, model64):
    """Config 2 through the reference's own host-buffer symbols, driven the
    way the MS6 gridding strategy drives them (MS6/programs/gridding.hs:40-103;
    one C call per region, Flow/Halide.hs:309-322): the C++ host layer's
    binSizer + binner over the uv-tile (uv-tiles 1, the reference default,
    MS6/programs/Kernel/Config.hs:101) and ob.n_planes w-bins, one
    kern_scatter_gpu1 per w-bin into the tile with its gcfMaxSize margin,
    detiling into the full grid; then one kern_degrid_gpu1 per w-bin against
    the full model grid.  FP64 5-double records in pageable host memory; GCF
    files of supports 16 / 32 / 64 (the reference's own set,
    MS6/cfg/continuum.yaml) at the w where the workload's support rule passes
    16 and 32, generated on the GPU and chosen per bin by gcfGet; the model is
    the FP64 dirty grid.  Binning and GCF reads happen once per observation
    and are reported apart; a pass is one gridding plus one degridding of every
    visibility, host wall clock, mean of K after W."""
    import tempfile

    from rc_gb300 import build as B
    from rc_gb300 import gcf as Gm

    exe = B.strategy_program()
    G, n = ob.grid_size, ob.n
    from rc_gb300 import synth

    files = synth.abi_gcf_files(ob)
    ws = np.array([w for w, _ in files])
    sup = np.array([S for _, S in files], np.int32)
    g64, _, offs = Gm.generate(ws, sup, 64, ob.scale / 2, taper=Gm.pswf_taper(64),
                               want32=False)
    g64 = g64.cpu().numpy()
    with tempfile.TemporaryDirectory() as d:
        lines = []
        for i, ((w, S), o) in enumerate(zip(files, offs)):
            path = os.path.join(d, "gcf%d.dat" % i)
            g64[o:o + 64 * S * S].tofile(path)
            lines.append("%s %d %.17g" % (path, S, w))
        with open(os.path.join(d, "params.txt"), "w") as f:
            f.write("%d %d %.17g %d %d %d %d %d\n" % (G, G, ob.scale, 1, ob.n_planes, len(files),
                                                      1, 1))
            f.write("\n".join(lines) + "\n")
        np.ascontiguousarray(ob.vis5(), np.float64).tofile(os.path.join(d, "vis.bin"))
        np.ascontiguousarray(model64, np.complex128).tofile(os.path.join(d, "model.bin"))
        with open(os.path.join(d, "time.txt"), "w") as f:
            f.write("%d %d\n" % (args.warmup, args.steps))
        r = subprocess.run([exe, d, "time"], capture_output=True, text=True, timeout=3600)
        if r.returncode != 0:
            raise RuntimeError("gridding_strategy time: " + r.stderr)
        out = json.loads(r.stdout.strip().splitlines()[-1])
    tg, td = float(np.mean(out["grid_ms"])), float(np.mean(out["degrid_ms"]))
    return {"value": round(n / ((tg + td) * 1e-3) / 1e6, 3), "unit": "Mvis/s",
            "ms_per_step": round(tg + td, 3), "grid_ms": round(tg, 3),
            "degrid_ms": round(td, 3), "binning_ms_once": round(out["bin_ms"], 1),
            "gcf_read_ms_once": round(out["gcf_read_ms"], 1),
            "calls_per_direction": out["calls_per_direction"],
            "records": out["records"],
            "gcf_files": [{"w": round(w, 3), "size": S} for w, S in files],
            "path": "rc_gb300/host/gridding_strategy.cpp `time` on include/rc_kernels.hpp: "
                    "binSizer + binner, kern_scatter_gpu1 per w-bin, kern_detile, "
                    "kern_degrid_gpu1 per w-bin; pageable host buffers, every copy inside "
                    "the calls; host wall clock per pass, mean of K after W"}


def _explicit_params(args):
    return {k: v for k, v in (("tile", args.tile), ("threads", args.threads),
                              ("period_cap", args.cap), ("bundles_per_cta", args.bpc)) if v}


def _tuned_params(args, make_plan, vis32, g32, grid, n_supports):
    """Tunables: explicit flags, else the autotuner (cached per workload key)."""
    import torch

    from rc_gb300 import autotune as AT

    explicit = _explicit_params(args)
    tune_info = {"source": "flags" if explicit else "autotune"}
    if explicit or args.no_tune:
        tune_info["source"] = "flags" if explicit else "defaults"
        return dict(AT.DEFAULT, **explicit), tune_info
    probe = make_plan(**AT.DEFAULT)
    planes = probe.export_index()
    kept_mask = planes[:, 4] == 1
    counts = torch.bincount(planes[kept_mask, 3].long(), minlength=n_supports).cpu()
    key = AT.plan_signature(probe, counts.numpy())
    probe.close()
    cached = AT._load().get(key)
    if cached:
        params = dict(cached["params"])
        tune_info["cached"] = True
    else:
        t0 = time.perf_counter()
        params, best_ms, table = AT.tune(make_plan, vis32, g32, grid, key=key)
        tune_info.update(cached=False, candidates=len(table),
                         seconds=round(time.perf_counter() - t0, 2), best_ms=round(best_ms, 3))
    tune_info["key"] = key
    return params, tune_info


def _ncu_figures(config, kernel):
    """ncu figures of one launch of `kernel` on `config`, from
    profiles/traffic.json: (DRAM bytes read + written, the binding pipe)."""
    tpath = os.path.join(ROOT, "profiles", "traffic.json")
    try:
        d = json.load(open(tpath)).get(config, {}).get(kernel)
    except Exception:
        return None, None
    if d is None:
        return None, None
    if isinstance(d, (int, float)):
        return int(d), None
    bind = {k: d[k] for k in ("pipe", "pct", "source") if k in d}
    return d.get("dram_bytes"), (bind or None)


def roofline_of(config, kept, taps, tg, td, peak, peak_kind):
    """Roofline of the dominant FP32 kernel: the per-tap byte model's fraction
    of the measured HBM peak (frac), the DRAM bytes ncu counts per launch
    (traffic) and their fraction of the peak (hbm_frac_dram), and the pipe
    that binds the kernel with its ncu utilisation (binding)."""
    bytes_grid = 32 * kept + 24 * taps
    bytes_deg = 40 * kept + 16 * taps
    if tg >= td:
        dom, b_dom, t_dom = "k_grid_tiled", bytes_grid, tg
    else:
        dom, b_dom, t_dom = "k_degrid_tiled", bytes_deg, td
    achieved = b_dom / (t_dom * 1e-3) / 1e9
    traffic, binding = _ncu_figures(config, dom)
    per_kernel = {}
    for name, b, t in (("k_grid_tiled", bytes_grid, tg), ("k_degrid_tiled", bytes_deg, td)):
        tr, bd = _ncu_figures(config, name)
        per_kernel[name] = {
            "ms": round(t, 4), "frac_model": round(b / (t * 1e-3) / 1e9 / peak, 4),
            "hbm_frac_dram": round(tr / (t * 1e-3) / 1e9 / peak, 4) if tr else None,
            "binding": bd}
    return {"bound": "hbm", "kernel": dom, "achieved": round(achieved, 1), "peak": peak,
            "unit": "GB/s", "frac": round(achieved / peak, 4), "peak_kind": peak_kind,
            "traffic": traffic, "algorithmic_bytes_per_launch": int(b_dom),
            "hbm_frac_dram": (round(traffic / (t_dom * 1e-3) / 1e9 / peak, 4)
                              if traffic else None),
            "binding": binding, "kernels": per_kernel, "model": ROOFLINE_MODEL}


def device_pair(ob, args, dev, flush, clock_index=0, steps=None, fp64_reps=None):
    """Everything measured with the inputs resident in HBM, for one workload:
    GCFs generated on the GPU (first call and warm), the plan (tuned), the
    FP32 pair timed per kernel and as a CUDA-graph step (L2 flushed before
    each), the plain FP64 pair on the same step, and the FP32 error against
    it.  Returns a dict of the tensors and figures."""
    import torch

    from rc_gb300 import gcf as Gm
    from rc_gb300.engine import Plan

    steps = args.steps if steps is None else steps
    s = torch.cuda.current_stream(dev)
    G = ob.grid_size
    tp = Gm.pswf_taper(ob.max_support)
    gen = []
    for _ in range(2):  # the first call loads the library
        t0 = time.perf_counter()
        g64, g32, offs = Gm.generate(ob.w_planes, ob.supports, ob.max_support, ob.scale / 2,
                                     taper=tp, device=dev)
        torch.cuda.synchronize()
        gen.append(1e3 * (time.perf_counter() - t0))

    h_uvw = torch.tensor(ob.uvw).pin_memory()
    d_uvw = torch.empty_like(h_uvw, device=dev)
    e_up = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    e_up[0].record(s)
    d_uvw.copy_(h_uvw, non_blocking=True)
    e_up[1].record(s)
    e_up[1].synchronize()
    uvw_up_ms = e_up[0].elapsed_time(e_up[1])
    vis32 = torch.tensor(ob.vis, dtype=torch.complex64, device=dev)
    vis64 = torch.tensor(ob.vis, dtype=torch.complex128, device=dev)
    grid = torch.zeros((G, G), dtype=torch.complex64, device=dev)

    def make_plan(**p):
        return Plan(d_uvw, scale=ob.scale, grid_size=G, grid_shape=(G, G), supports=ob.supports,
                    w_range=(ob.w_low, ob.w_high), **p)

    params, tune_info = _tuned_params(args, make_plan, vis32, g32, grid, len(ob.supports))
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    plan = make_plan(**params)
    torch.cuda.synchronize()
    plan_ms = 1e3 * (time.perf_counter() - t0)
    st = plan.stats()
    pred = torch.empty(ob.n, dtype=torch.complex64, device=dev)

    # model grid for degridding: the FP64 dirty grid of the observation
    grid64 = torch.zeros((G, G), dtype=torch.complex128, device=dev)
    plan.grid64(vis64, g64, grid64)
    model32 = grid64.to(torch.complex64)
    pred64 = plan.degrid64(g64, grid64)
    torch.cuda.synchronize()

    # accuracy of the FP32 pair against the plain FP64 path (itself pinned to
    # the oracle at 1e-12 by the tests)
    grid.zero_()
    plan.grid(vis32, g32, grid)
    plan.degrid(g32, model32, out=pred)
    torch.cuda.synchronize()
    err_grid = float(torch.linalg.vector_norm(grid.to(torch.complex128) - grid64) /
                     torch.linalg.vector_norm(grid64))
    err_deg = float(torch.linalg.vector_norm(pred.to(torch.complex128) - pred64) /
                    torch.linalg.vector_norm(pred64))

    def step():
        grid.zero_()
        plan.grid(vis32, g32, grid)
        plan.degrid(g32, model32, out=pred)

    use_graph = not args.no_graph
    if use_graph:
        side = torch.cuda.Stream(dev)
        side.wait_stream(s)
        with torch.cuda.stream(side):
            step()
        s.wait_stream(side)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            step()
        run = graph.replay
    else:
        run = step

    # per-kernel timing (eager, events on the launching stream)
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(3)]
    kg, kd = [], []
    for i in range(args.warmup + steps):
        flush.fill_(float(i))
        grid.zero_()
        ev[0].record(s)
        plan.grid(vis32, g32, grid)
        ev[1].record(s)
        plan.degrid(g32, model32, out=pred)
        ev[2].record(s)
        ev[2].synchronize()
        if i >= args.warmup:
            kg.append(ev[0].elapsed_time(ev[1]))
            kd.append(ev[1].elapsed_time(ev[2]))

    # timed steps: W warm-up replays, then K, each after an L2 flush
    for i in range(args.warmup):
        flush.fill_(float(i))
        run()
    torch.cuda.synchronize()
    world = int(os.environ.get("WORLD_SIZE", "1"))
    if world > 1:
        import torch.distributed as dist

        dist.barrier()
    torch.cuda.synchronize()
    starts = [torch.cuda.Event(enable_timing=True) for _ in range(steps)]
    ends = [torch.cuda.Event(enable_timing=True) for _ in range(steps)]
    with ClockSampler(clock_index) as clk:
        wall0 = time.perf_counter()
        for i in range(steps):
            flush.fill_(float(i + 7))
            starts[i].record(s)
            run()
            ends[i].record(s)
        torch.cuda.synchronize()
        wall = time.perf_counter() - wall0
    t_step = float(np.mean([a.elapsed_time(b) for a, b in zip(starts, ends)]))

    # plain FP64 GPU path, same step
    k64 = []
    reps = (0 if args.quick else 2 + max(2, steps // 4)) if fp64_reps is None else fp64_reps
    for i in range(reps):
        flush.fill_(float(i))
        grid64.zero_()
        ev[0].record(s)
        plan.grid64(vis64, g64, grid64)
        plan.degrid64(g64, grid64, out=pred64)
        ev[1].record(s)
        ev[1].synchronize()
        if i >= 2:
            k64.append(ev[0].elapsed_time(ev[1]))
    return dict(plan=plan, params=params, tune_info=tune_info, st=st, kept=st["kept"],
                taps=st["taps"], tg=float(np.mean(kg)), td=float(np.mean(kd)), t_step=t_step,
                fp64_ms=float(np.mean(k64)) if k64 else None, err_grid=err_grid,
                err_deg=err_deg, grid=grid, pred=pred, vis32=vis32, model32=model32, g32=g32,
                g64=g64, grid64=grid64, d_uvw=d_uvw, plan_ms=plan_ms, gcf_ms=gen[1], gcf_first_ms=gen[0],
                uvw_up_ms=uvw_up_ms, uvw_bytes=h_uvw.numel() * 8, use_graph=use_graph,
                clk=clk, wall=wall)


def target_c4(args, dev, flush):
    """The least-squares layout (2,064,384 visibilities, 2048^2, 16 w-planes
    S 8-62): the FP32 pair against the plain FP64 pair, the error, and both
    roofline figures, next to the stated target (>= 60 % of the HBM roofline,
    >= 3x the plain FP64 gridder, rel-L2 <= 1e-5 against FP64)."""
    ob = load_workload("c4")
    R = device_pair(ob, args, dev, flush, steps=max(5, args.steps // 2), fp64_reps=5)
    peak, peak_kind = measured_peaks()
    rl = roofline_of("c4", R["kept"], R["taps"], R["tg"], R["td"], peak, peak_kind)
    value = ob.n / (R["t_step"] * 1e-3) / 1e6
    fp64 = ob.n / (R["fp64_ms"] * 1e-3) / 1e6
    ratio = value / fp64
    fr = min(rl["kernels"]["k_grid_tiled"]["frac_model"],
             rl["kernels"]["k_degrid_tiled"]["frac_model"])
    err = max(R["err_grid"], R["err_deg"])
    out = {"workload": _workload_desc(ob), "visibilities": ob.n, "taps": R["taps"],
           "value": round(value, 3), "unit": "Mvis/s", "ms_per_step": round(R["t_step"], 4),
           "fp64_plain": {"value": round(fp64, 3), "ms_per_step": round(R["fp64_ms"], 3)},
           "ratio_f32_over_f64": round(ratio, 2),
           "rel_l2_vs_fp64": {"grid": R["err_grid"], "degrid": R["err_deg"]},
           "roofline": {k: {kk: v[kk] for kk in ("ms", "frac_model", "hbm_frac_dram",
                                                  "binding")}
                        for k, v in rl["kernels"].items()},
           "tuning": dict(R["params"], **R["tune_info"]), "clocks": R["clk"].summary(),
           "target": {"roofline_frac_min": 0.6, "ratio_min": 3.0, "rel_l2_max": 1e-5},
           "met": bool(fr >= 0.6 and ratio >= 3.0 and err <= 1e-5),
           "note": "roofline_frac_min is met on the per-tap byte model (frac_model); "
                   "hbm_frac_dram is the DRAM traffic ncu counts, and binding the pipe "
                   "that limits the kernel"}
    R["plan"].close()
    return out


def our_arm(args):
    import torch

    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if world > 1:
        import torch.distributed as dist

        torch.cuda.set_device(local)
        dist.init_process_group("nccl", device_id=torch.device("cuda", local))
    dev = torch.device("cuda", local)

    from rc_gb300 import gcf as Gm
    from rc_gb300 import lib as L

    L.load()
    ob = load_workload(args.config)
    # shard by replica: each rank grids its own observation of the same size
    if world > 1 and rank > 0:
        from rc_gb300 import synth

        ob = synth.config(args.config, seed=synth.SEED0 + 1000 * rank)
    G = ob.grid_size
    s = torch.cuda.current_stream(dev)
    flush = torch.empty(2 * L2_BYTES // 4, dtype=torch.float32, device=dev)
    R = device_pair(ob, args, dev, flush, clock_index=local)
    plan, grid, pred, model32, g32 = R["plan"], R["grid"], R["pred"], R["model32"], R["g32"]
    kept, taps, st = R["kept"], R["taps"], R["st"]
    t_step = R["t_step"]
    if world > 1:
        import torch.distributed as dist

        tt = torch.tensor([t_step], device=dev)
        dist.all_reduce(tt, op=dist.ReduceOp.MAX)
        t_step = float(tt.item())
        dist.barrier()
    value = world * ob.n / (t_step * 1e-3) / 1e6
    fp64_mvis = ob.n / (R["fp64_ms"] * 1e-3) / 1e6 if R["fp64_ms"] else float("nan")
    peak, peak_kind = measured_peaks()
    tg, td = R["tg"], R["td"]
    roofline = roofline_of(args.config, kept, taps, tg, td, peak, peak_kind)

    # end to end through the public API: every step uploads its visibilities
    # and model grid from pinned host memory and downloads its grid and
    # predictions, inside the timed region.  Device and host buffers are
    # double-buffered and the copies run on their own streams, so step i+1's
    # uploads overlap step i's degridding, step i's grid download overlaps its
    # degridding and its prediction download overlaps step i+1's gridding: in
    # steady state a step costs its kernels plus what the copies cannot hide.
    # The per-step working set (about 300 MB) is larger than L2.
    h_vis = torch.tensor(ob.vis, dtype=torch.complex64).pin_memory()
    h_model = model32.cpu().pin_memory()
    h_grid = [torch.empty((G, G), dtype=torch.complex64).pin_memory() for _ in range(2)]
    h_pred = [torch.empty(ob.n, dtype=torch.complex64).pin_memory() for _ in range(2)]
    d_vis_e = [torch.empty_like(R["vis32"]) for _ in range(2)]
    d_model_e = [torch.empty_like(model32) for _ in range(2)]
    d_grid_e = [grid, torch.empty_like(grid)]
    d_pred_e = [pred, torch.empty_like(pred)]
    s_up, s_down = torch.cuda.Stream(dev), torch.cuda.Stream(dev)

    def pipeline(k, start):
        mk = [[torch.cuda.Event() for _ in range(k)] for _ in range(6)]
        vis_up, model_up, grid_done, deg_done, grid_down, pred_down = mk
        s_up.wait_event(start)
        for i in range(k):
            b = i % 2
            with torch.cuda.stream(s_up):
                if i >= 2:
                    s_up.wait_event(grid_done[i - 2])
                d_vis_e[b].copy_(h_vis, non_blocking=True)
                vis_up[i].record(s_up)
                if i >= 2:
                    s_up.wait_event(deg_done[i - 2])
                d_model_e[b].copy_(h_model, non_blocking=True)
                model_up[i].record(s_up)
            s.wait_event(vis_up[i])
            if i >= 2:
                s.wait_event(grid_down[i - 2])
            d_grid_e[b].zero_()
            plan.grid(d_vis_e[b], g32, d_grid_e[b])
            grid_done[i].record(s)
            s.wait_event(model_up[i])
            if i >= 2:
                s.wait_event(pred_down[i - 2])
            plan.degrid(g32, d_model_e[b], out=d_pred_e[b])
            deg_done[i].record(s)
            with torch.cuda.stream(s_down):
                s_down.wait_event(grid_done[i])
                h_grid[b].copy_(d_grid_e[b], non_blocking=True)
                grid_down[i].record(s_down)
                s_down.wait_event(deg_done[i])
                h_pred[b].copy_(d_pred_e[b], non_blocking=True)
                pred_down[i].record(s_down)
        s.wait_stream(s_up)
        s.wait_stream(s_down)

    e2e_ms = e2e_lat = None
    if not args.quick:
        st0 = torch.cuda.Event()
        st0.record(s)
        pipeline(args.warmup, st0)
        torch.cuda.synchronize()
        t0e, t1e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        t0e.record(s)
        pipeline(args.steps, t0e)
        t1e.record(s)
        t1e.synchronize()
        e2e_ms = t0e.elapsed_time(t1e) / args.steps
        # the last step's results are the step's own
        assert torch.equal(h_pred[(args.steps - 1) % 2], d_pred_e[(args.steps - 1) % 2].cpu())
        # latency of one step on its own (no neighbour to overlap with): the
        # same copies and kernels, each step bracketed by events and waited on
        lat = []
        for i in range(args.warmup + args.steps):
            t0e.record(s)
            pipeline(1, t0e)
            t1e.record(s)
            t1e.synchronize()
            if i >= args.warmup:
                lat.append(t0e.elapsed_time(t1e))
        e2e_lat = float(np.median(lat))
    e2e_mvis = world * ob.n / (e2e_ms * 1e-3) / 1e6 if e2e_ms else float("nan")
    h2d = h_vis.numel() * 8 + h_model.numel() * 8
    d2h = h_grid[0].numel() * 8 + h_pred[0].numel() * 8
    # the per-observation costs (uvw upload, plan, GCF generation) spread over
    # the major cycles that reuse them
    once_ms = R["uvw_up_ms"] + R["plan_ms"] + R["gcf_ms"]
    amortised = None
    if e2e_ms:
        amortised = {str(c): round(world * ob.n / ((e2e_ms + once_ms / c) * 1e-3) / 1e6, 3)
                     for c in (1, 5)}

    abi = None
    if not args.quick and world == 1:
        if args.config == "c1":
            abi = abi_e2e(ob, args.steps, args.warmup)
        elif args.config == "c2" and not args.no_abi:
            abi = abi_strategy_e2e(ob, args, R["grid64"].cpu().numpy())

    # CPU baseline (rank 0, N = 1 only): the oracle port on the host cores
    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu and not args.quick:
        offs_np, _ = Gm.layout(ob.supports)
        n, dt, used = cpu_leg_isolated(ob, R["g64"].cpu().numpy(), offs_np, args.cpu_sample)
        cpu = {"value": round(n / dt / 1e6, 3), "unit": "Mvis/s", "cores": used, "kind": "port",
               "taps": taps if n == ob.n else None,
               "gtaps_per_s": round(2 * taps / dt / 1e9, 3) if n == ob.n else None,
               "sample": (f"{'the whole observation' if n == ob.n else f'first {n} of {ob.n}'} "
                          f"visibilities, grid + degrid, FP64, {used} threads, mean of 2 runs "
                          f"after a warm-up, {dt:.3f} s each, in a child interpreter without "
                          "the GPU runtime")}

    c4 = None
    if args.config == "c2" and not args.quick and world == 1 and not args.no_target:
        plan_keep = plan  # the headline plan stays alive; c4 has its own
        c4 = target_c4(args, dev, flush)
        del plan_keep

    if rank == 0:
        line = {
            "metric": METRIC, "value": round(value, 3), "unit": "Mvis/s", "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(t_step, 4),
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
            "data": "synthetic (seeded); no public dataset",
            "config": {"workload": _workload_desc(ob), "visibilities": ob.n, "kept": kept,
                       "taps": taps, "grid": f"{G}x{G} complex64",
                       "l2": "flushed (256 MiB write) before every step",
                       "tile": st["tile"], "threads": st["threads"], "graph": R["use_graph"],
                       "tuning": dict(R["params"], **R["tune_info"]),
                       "parallelism": f"replicas x{world}"},
            "roofline": roofline,
            "kernels_ms": {"grid_f32": round(tg, 4), "degrid_f32": round(td, 4),
                           "grid_frac_of_roofline": roofline["kernels"]["k_grid_tiled"][
                               "frac_model"],
                           "degrid_frac_of_roofline": roofline["kernels"]["k_degrid_tiled"][
                               "frac_model"],
                           "plan_ms": round(R["plan_ms"], 2),
                           "gcf_generate_ms": round(R["gcf_ms"], 2),
                           "gcf_generate_first_call_ms": round(R["gcf_first_ms"], 2),
                           "uvw_upload_ms": round(R["uvw_up_ms"], 3)},
            "fp64_plain": {"value": round(fp64_mvis, 3), "unit": "Mvis/s",
                           "ms_per_step": round(R["fp64_ms"], 3) if R["fp64_ms"] else None,
                           "speedup_f32_over_f64": round(value / world / fp64_mvis, 2)},
            "rel_l2_vs_fp64": {"grid": R["err_grid"], "degrid": R["err_deg"], "bar": 1e-5},
            "e2e": {"value": round(e2e_mvis, 3), "unit": "Mvis/s", "h2d_bytes_per_step": h2d,
                    "d2h_bytes_per_step": d2h,
                    "ms_per_step": round(e2e_ms, 3) if e2e_ms else None,
                    "timing": "K steps pipelined (double-buffered, copies on their own "
                              "streams) between two events, / K",
                    "single_step_latency_ms": round(e2e_lat, 3) if e2e_lat else None,
                    "amortised_per_observation": {
                        "value_by_major_cycles": amortised,
                        "once_ms": round(once_ms, 2),
                        "once": "uvw upload (pinned) + plan (index math, w-binning, sort/bin) "
                                "+ GCF generation, once per observation, spread over 1 or 5 "
                                "major cycles of one grid + one degrid step each"}},
            "e2e_reference_abi": abi,
            "cpu_baseline": cpu,
            "target_c4": c4,
            "clocks": R["clk"].summary(),
            "gpu_launches": 2 * args.steps,
            "wall_s_timed_region": round(R["wall"], 4),
        }
        print(json.dumps(line))
    if world > 1:
        import torch.distributed as dist

        dist.destroy_process_group()
    return 0


def our_arm_batch(args):
    """config 3: 64 channel grids + 9 facet grids (1024^2-4096^2, 48 shared
    w-planes, S 8-96, ~32 M vis) gridded and degridded by ONE batched launch each."""
    import torch

    from rc_gb300 import gcf as Gm
    from rc_gb300 import lib as L
    from rc_gb300 import synth
    from rc_gb300.engine import Batch

    L.load()
    dev = torch.device("cuda", 0)
    s = torch.cuda.current_stream(dev)
    t0 = time.perf_counter()
    members, scale, supports, w_planes, wlo, whi = synth.config3(n_t=args.c3_nt)
    n_ch_members = 64  # the channel grids come first, then the facets
    gen_s = time.perf_counter() - t0
    smax = int(supports.max())
    g64, g32, offs = Gm.generate(w_planes, supports, smax, scale / 2,
                                 taper=Gm.pswf_taper(smax), device=dev)
    uvws = [torch.tensor(m.uvw, device=dev) for m in members]
    vis32 = [torch.tensor(m.vis, dtype=torch.complex64, device=dev) for m in members]
    grids = [torch.zeros((m.grid_size, m.grid_size), dtype=torch.complex64, device=dev)
             for m in members]
    preds = [torch.empty(m.n, dtype=torch.complex64, device=dev) for m in members]

    def make_batch(**p):
        return Batch([dict(uvw=u, scale=scale, grid_size=m.grid_size,
                           grid_shape=(m.grid_size, m.grid_size), supports=supports,
                           gcf_offsets=offs, w_range=(wlo, whi))
                      for u, m in zip(uvws, members)], **p)

    # tunables: explicit flags, else the autotuner on the heaviest member (the
    # highest channel: a 4096^2 grid and the largest w-supports), whose
    # choice then runs the whole batch (every member shares the w-planes)
    from rc_gb300 import autotune as AT
    from rc_gb300.engine import Plan

    explicit = {k: v for k, v in (("tile", args.tile), ("threads", args.threads),
                                  ("period_cap", args.cap), ("bundles_per_cta", args.bpc)) if v}
    tune_info = {"source": "flags" if explicit else "autotune"}
    if explicit or args.no_tune:
        params = dict(AT.DEFAULT, **explicit)
        tune_info["source"] = "flags" if explicit else "defaults"
    else:
        k = n_ch_members - 1
        m = members[k]

        def make_plan(**p):
            return Plan(uvws[k], scale=scale, grid_size=m.grid_size,
                        grid_shape=(m.grid_size, m.grid_size), supports=supports,
                        gcf_offsets=offs, w_range=(wlo, whi), **p)

        t0 = time.perf_counter()
        params, best_ms, table = AT.tune(make_plan, vis32[k], g32, grids[k])
        tune_info.update(member=k, candidates=len(table), seconds=round(time.perf_counter() - t0, 2),
                         best_ms=round(best_ms, 3))
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    B = make_batch(**params)
    torch.cuda.synchronize()
    plan_ms = 1e3 * (time.perf_counter() - t0)
    st = B.stats()
    n_vis = sum(m.n for m in members)

    def step():
        for g in grids:
            g.zero_()
        B.grid(vis32, g32, grids)
        B.degrid(g32, grids, preds=preds)

    side = torch.cuda.Stream(dev)
    side.wait_stream(s)
    with torch.cuda.stream(side):
        step()
    s.wait_stream(side)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        step()
    flush = torch.empty(2 * L2_BYTES // 4, dtype=torch.float32, device=dev)
    for i in range(args.warmup):
        flush.fill_(float(i))
        graph.replay()
    torch.cuda.synchronize()
    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True))
          for _ in range(args.steps)]
    with ClockSampler(0) as clk:
        for i in range(args.steps):
            flush.fill_(float(i + 3))
            ev[i][0].record(s)
            graph.replay()
            ev[i][1].record(s)
        torch.cuda.synchronize()
    t_step = float(np.mean([a.elapsed_time(b) for a, b in ev]))
    value = n_vis / (t_step * 1e-3) / 1e6
    # per-kernel times (eager)
    e = [torch.cuda.Event(enable_timing=True) for _ in range(3)]
    kg, kd = [], []
    for i in range(3):
        flush.fill_(float(i))
        for g in grids:
            g.zero_()
        e[0].record(s)
        B.grid(vis32, g32, grids)
        e[1].record(s)
        B.degrid(g32, grids, preds=preds)
        e[2].record(s)
        e[2].synchronize()
        kg.append(e[0].elapsed_time(e[1]))
        kd.append(e[1].elapsed_time(e[2]))
    # FP64 plain comparison and the FP32 error against it
    vis64 = [torch.tensor(m.vis, dtype=torch.complex128, device=dev) for m in members]
    grids64 = [torch.zeros((m.grid_size, m.grid_size), dtype=torch.complex128, device=dev)
               for m in members]
    preds64 = [torch.empty(m.n, dtype=torch.complex128, device=dev) for m in members]
    e[0].record(s)
    B.grid64(vis64, g64, grids64)
    B.degrid64(g64, grids64, preds64)
    e[1].record(s)
    e[1].synchronize()
    t64 = e[0].elapsed_time(e[1])
    for g in grids:
        g.zero_()
    B.grid(vis32, g32, grids)
    models = [g.to(torch.complex64) for g in grids64]
    B.degrid(g32, models, preds=preds)
    torch.cuda.synchronize()
    num = sum(float(torch.linalg.vector_norm(a.to(torch.complex128) - b) ** 2)
              for a, b in zip(grids, grids64))
    den = sum(float(torch.linalg.vector_norm(b) ** 2) for b in grids64)
    nump = sum(float(torch.linalg.vector_norm(a.to(torch.complex128) - b) ** 2)
               for a, b in zip(preds, preds64))
    denp = sum(float(torch.linalg.vector_norm(b) ** 2) for b in preds64)
    peak, peak_kind = measured_peaks()
    bytes_grid = 32 * st["kept"] + 24 * st["taps"]
    bytes_deg = 40 * st["kept"] + 16 * st["taps"]
    tg, td = float(np.mean(kg)), float(np.mean(kd))
    dom = ("k_grid_tiled", bytes_grid, tg) if tg >= td else ("k_degrid_tiled", bytes_deg, td)
    achieved = dom[1] / (dom[2] * 1e-3) / 1e9
    line = {
        "metric": METRIC, "value": round(value, 3), "unit": "Mvis/s", "n_gpus": 1,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(t_step, 4),
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
        "data": "synthetic (seeded); no public dataset",
        "config": {"workload": f"c3: {len(members)} grids (64 channels 100-200 MHz + 9 facets, "
                               f"1024^2-4096^2), {n_vis} vis, 48 w-planes S 8-{smax}, one "
                               f"persistent launch per direction", "visibilities": n_vis,
                   "kept": st["kept"], "taps": st["taps"], "bundles": st["bundles"],
                   "tuning": dict(params, **tune_info), "graph": True,
                   "generate_s": round(gen_s, 1),
                   "l2": "flushed (256 MiB write) before every step"},
        "roofline": {"bound": "hbm", "kernel": dom[0], "achieved": round(achieved, 1),
                     "peak": peak, "unit": "GB/s", "frac": round(achieved / peak, 4),
                     "peak_kind": peak_kind, "traffic": None,
                     "algorithmic_bytes_per_launch": int(dom[1]), "model": ROOFLINE_MODEL},
        "kernels_ms": {"grid_f32": round(tg, 3), "degrid_f32": round(td, 3),
                       "plan_ms": round(plan_ms, 1)},
        "fp64_plain": {"value": round(n_vis / (t64 * 1e-3) / 1e6, 3), "unit": "Mvis/s",
                       "ms_per_step": round(t64, 2),
                       "speedup_f32_over_f64": round(t64 / t_step, 2)},
        "rel_l2_vs_fp64": {"grid": (num / den) ** 0.5, "degrid": (nump / denp) ** 0.5,
                           "bar": 1e-5},
        "e2e": None, "cpu_baseline": None, "clocks": clk.summary(),
        "gpu_launches": 2 * args.steps,
    }
    print(json.dumps(line))
    return 0


def our_arm_major_cycle(args):
    """config 5: 512 stations to 40 km, 130,816 bl x 64 t x 4 ch = 33.5 M vis,
    8192^2 grid, 64 w-planes S 8-128; 5 major cycles of grid -> FFT -> Hogbom
    (gain 0.1, 1000 iterations) -> FFT -> degrid -> subtract, all on the GPU."""
    import torch

    from rc_gb300 import gcf as Gm
    from rc_gb300 import lib as L
    from rc_gb300 import synth
    from rc_gb300.engine import Plan
    from rc_gb300.major_cycle import MajorCycle

    L.load()
    dev = torch.device("cuda", 0)
    t0 = time.perf_counter()
    ob = synth.config("c5", n_t=args.c5_nt)
    gen_s = time.perf_counter() - t0
    n = ob.grid_size
    _, g32, _ = Gm.generate(ob.w_planes, ob.supports, ob.max_support, ob.scale / 2,
                            taper=Gm.pswf_taper(ob.max_support), want64=False, device=dev)
    uvw = torch.tensor(ob.uvw, device=dev)
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    plan = Plan(uvw, scale=ob.scale, grid_size=n, grid_shape=(n, n), supports=ob.supports,
                w_range=(ob.w_low, ob.w_high), tile=args.tile or 24, threads=args.threads or 256,
                period_cap=args.cap or 40)
    torch.cuda.synchronize()
    plan_ms = 1e3 * (time.perf_counter() - t0)
    st = plan.stats()
    t_img = torch.tensor(Gm.w0_correction(ob.max_support, ob.scale / 2,
                                          Gm.pswf_taper(ob.max_support), n, device=dev),
                         dtype=torch.float32, device=dev)
    mc = MajorCycle(plan, g32, t_img)
    vis = torch.tensor(ob.vis, dtype=torch.complex64, device=dev)
    # warm-up: one short cycle
    mc.run(vis, n_major=1, n_minor=10)
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    with ClockSampler(0) as clk:
        e0.record()
        model, resid, stats = mc.run(vis, n_major=5, n_minor=1000, gain=0.1)
        e1.record()
        torch.cuda.synchronize()
    total_ms = e0.elapsed_time(e1)
    # one grid + degrid pass timed alone, for the Mvis/s of the adjoint pair
    grid = torch.zeros((n, n), dtype=torch.complex64, device=dev)
    a, b, c = (torch.cuda.Event(enable_timing=True) for _ in range(3))
    a.record()
    plan.grid(vis, g32, grid)
    b.record()
    plan.degrid(g32, grid)
    c.record()
    c.synchronize()
    tg, td = a.elapsed_time(b), b.elapsed_time(c)
    peak, peak_kind = measured_peaks()
    bytes_grid = 32 * st["kept"] + 24 * st["taps"]
    line = {
        "metric": METRIC, "value": round(ob.n / ((tg + td) * 1e-3) / 1e6, 3), "unit": "Mvis/s",
        "n_gpus": 1, "steps": 5, "warmup": 1, "ms_per_step": round(total_ms / 5, 2),
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
        "data": "synthetic (seeded); no public dataset",
        "config": {"workload": f"c5: {ob.n} vis, {n}^2 grid, {ob.n_planes} w-planes S "
                               f"{int(ob.supports.min())}-{int(ob.supports.max())}; step = one "
                               f"major cycle (grid, FFT, Hogbom 1000 it., FFT, degrid)",
                   "kept": st["kept"], "taps": st["taps"], "generate_s": round(gen_s, 1),
                   "plan_ms": round(plan_ms, 1), "major_cycles": stats},
        "roofline": {"bound": "hbm", "kernel": "k_grid_tiled",
                     "achieved": round(bytes_grid / (tg * 1e-3) / 1e9, 1), "peak": peak,
                     "unit": "GB/s", "frac": round(bytes_grid / (tg * 1e-3) / 1e9 / peak, 4),
                     "peak_kind": peak_kind, "traffic": None,
                     "algorithmic_bytes_per_launch": int(bytes_grid), "model": ROOFLINE_MODEL},
        "kernels_ms": {"grid_f32": round(tg, 3), "degrid_f32": round(td, 3),
                       "major_cycle_total_ms": round(total_ms, 1)},
        "e2e": None, "cpu_baseline": None, "clocks": clk.summary(),
    }
    print(json.dumps(line))
    return 0


# ---------------------------------------------------------------- OSKAR ingest
OSKAR_METRIC = "Mvis/s OSKAR .vis ingest (read, CRC-32C check, reshuffle to [bl][t][ch], u,v,w to wavelengths)"


def _oskar_file(ob, path, writer):
    """The config-2 observation as an OSKAR 2.6 file (blocks of 8 times)."""
    t0 = time.perf_counter()
    if writer == "ours":
        from rc_gb300 import synth
        size = synth.write_oskar_vis(path, ob, max_times_per_block=8)
    else:  # the reference arm runs none of the engine's code
        from oracle import oskar as K
        B, T = ob.n_bl, ob.n_t
        S = int(round((1 + (1 + 8 * B) ** 0.5) / 2))
        vis = ob.vis.reshape(B, T).T
        amps = np.zeros((T, 1, B, 4), np.complex128)
        amps[:, 0, :, 0] = vis
        amps[:, 0, :, 3] = vis
        m = (ob.uvw * (299792458.0 / 150e6)).reshape(B, T, 3).transpose(2, 1, 0)
        lay = K.layout(S, T, 1, 8, freq_start_hz=150e6, freq_inc_hz=0.0)
        assert K.write(path, lay, amps, m[0], m[1], m[2]) == 0
        size = os.path.getsize(path)
    return size, time.perf_counter() - t0


def our_arm_oskar(args):
    """OSKAR ingest: the config-2 observation (256 stations, 32,640 baselines x
    128 times x 1 channel = 4,177,920 points) stored as an OSKAR 2.6 .vis file
    in blocks of 8 times (367 MB), in the page cache.  One step = open + index +
    read every block: small tags on the host; payloads by parallel pread into
    pinned slots and copies to HBM; CRC-32C of every payload and the reshuffle
    [t][c][b] -> [b][t][c] with the wavelength scaling and extrema on the GPU.
    value: outputs left in HBM (gb_oskar_read_device); e2e: the reference ABI
    (mkFromFile + readAndReshuffle) into host arrays; cpu_baseline: the C
    restatement of the reference reader (single thread, as the reference)."""
    import ctypes as C
    import tempfile

    import torch

    from rc_gb300 import lib as Lm
    from rc_gb300 import synth

    L = Lm.load()
    dev = torch.device("cuda", 0)
    ob = synth.config("c2")
    tmpdir = tempfile.mkdtemp(prefix="rc_oskar_")
    path = os.path.join(tmpdir, "c2.vis")
    fsize, write_s = _oskar_file(ob, path, "ours")
    pb = path.encode()
    vd = Lm.VisData()
    Lm.check(L.mkFromFile(C.byref(vd), pb), "mkFromFile")
    P, B = vd.num_points, vd.num_baselines
    L.freeBinHandler(C.byref(vd))
    d_amps = torch.empty((P, 4), dtype=torch.complex128, device=dev)
    d_uvw = torch.empty((P, 3), dtype=torch.float64, device=dev)
    mx = Lm.Metrix()
    blw = (Lm.WMaxMin * B)()
    stream = torch.cuda.current_stream().cuda_stream
    tm = (C.c_double * 4)()

    def dev_step():
        v = Lm.VisData()
        Lm.check(L.mkFromFile(C.byref(v), pb), "mkFromFile")
        try:
            Lm.check(L.gb_oskar_read_device(C.byref(v), d_amps.data_ptr(), d_uvw.data_ptr(),
                                            C.byref(mx), blw, stream), "gb_oskar_read_device")
        finally:
            L.freeBinHandler(C.byref(v))
        L.gb_oskar_last_timings(tm)
        return list(tm)

    for _ in range(args.warmup):
        dev_step()
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    per = []
    with ClockSampler(0) as clk:
        e0.record()
        for _ in range(args.steps):
            per.append(dev_step())
        e1.record()
        torch.cuda.synchronize()
    ms = e0.elapsed_time(e1) / args.steps
    per = np.array(per)
    stage_ms, crc_ms, resh_ms = (float(np.median(per[:, k])) for k in range(3))
    # e2e through the reference ABI with host arrays (what the Haskell reader calls)
    amps_h = np.empty((P, 4), np.complex128)
    uvw_h = np.empty((P, 3), np.float64)
    mx_h = Lm.Metrix()
    blw_h = (Lm.WMaxMin * B)()

    def host_step():
        v = Lm.VisData()
        Lm.check(L.mkFromFile(C.byref(v), pb), "mkFromFile")
        try:
            Lm.check(L.readAndReshuffle(C.byref(v), amps_h.ctypes.data, uvw_h.ctypes.data,
                                        C.byref(mx_h), blw_h), "readAndReshuffle")
        finally:
            L.freeBinHandler(C.byref(v))

    host_step()
    t0 = time.perf_counter()
    for _ in range(args.steps):
        host_step()
    e2e_ms = 1e3 * (time.perf_counter() - t0) / args.steps
    same_dev = bool(np.array_equal(d_amps.cpu().numpy().view(np.uint8), amps_h.view(np.uint8))
                    and np.array_equal(d_uvw.cpu().numpy().view(np.uint8), uvw_h.view(np.uint8)))
    cpu = None
    parity = None
    if not args.no_cpu:
        from oracle import oskar as K
        reps = max(1, min(3, args.steps))
        t0 = time.perf_counter()
        for _ in range(reps):
            st, h, a_o, uvw_o, mx_o, bl_o = K.read(path)
        cpu_s = (time.perf_counter() - t0) / reps
        parity = bool(st == 0 and np.array_equal(a_o.view(np.uint8), amps_h.view(np.uint8)) and
                      np.array_equal(uvw_o.view(np.uint8), uvw_h.view(np.uint8)))
        cpu = {"value": round(P / cpu_s / 1e6, 3), "unit": "Mvis/s", "cores": 1, "kind": "port",
               "sample": f"the whole {fsize / 1e6:.0f} MB file ({P} points), C restatement of "
                         "mkFromFile + readAndReshuffle (fread, CRC-32C slicing-by-8, reshuffle)",
               "ms": round(1e3 * cpu_s, 1)}
    os.remove(path)
    os.rmdir(tmpdir)
    peak, peak_kind = measured_peaks()
    payload = P * 88  # per point: 64 B of 4-pol amplitudes + 24 B of u,v,w (one channel)
    dom = "k_crc32c" if crc_ms >= resh_ms else "k_oskar_reshuffle"
    dom_bytes = payload if dom == "k_crc32c" else 2 * payload
    dom_ms = max(crc_ms, resh_ms)
    traffic = None
    tpath = os.path.join(ROOT, "profiles", "traffic.json")
    if os.path.exists(tpath):
        traffic = json.load(open(tpath)).get("oskar", {}).get(dom)
    line = {
        "metric": OSKAR_METRIC, "value": round(P / (ms * 1e-3) / 1e6, 3), "unit": "Mvis/s",
        "n_gpus": 1, "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(ms, 3),
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
        "data": "synthetic (seeded) config-2 observation written as an OSKAR 2.6 file",
        "config": {"workload": f"OSKAR .vis of c2: {B} baselines x {vd.num_times} times x 1 "
                               f"channel = {P} points, blocks of 8 times, {fsize} bytes, file "
                               "in the page cache; inputs larger than L2",
                   "file_write_s": round(write_s, 1), "outputs_bitexact_device_vs_host": same_dev,
                   "parity_vs_oracle_bitexact": parity},
        "roofline": {"bound": "hbm", "kernel": dom,
                     "achieved": round(dom_bytes / (dom_ms * 1e-3) / 1e9, 1), "peak": peak,
                     "unit": "GB/s", "frac": round(dom_bytes / (dom_ms * 1e-3) / 1e9 / peak, 4),
                     "peak_kind": peak_kind, "traffic": traffic,
                     "algorithmic_bytes_per_launch": int(dom_bytes)},
        "kernels_ms": {"host_staging_ms": round(stage_ms, 3), "k_crc32c": round(crc_ms, 4),
                       "k_oskar_reshuffle": round(resh_ms, 4)},
        "e2e": {"value": round(P / (e2e_ms * 1e-3) / 1e6, 3), "unit": "Mvis/s",
                "ms_per_step": round(e2e_ms, 2), "h2d_bytes_per_step": int(payload),
                "d2h_bytes_per_step": int(P * 88)},
        "cpu_baseline": cpu, "gpu_launches": 3 * args.steps, "clocks": clk.summary(),
    }
    print(json.dumps(line))
    return 0


def reference_arm_oskar(args):
    """--impl reference --config oskar: the reference reader's semantics (its C
    restatement, single thread as the reference) on the same file."""
    import tempfile

    from oracle import oskar as K
    from rc_gb300 import synth

    if int(os.environ.get("RANK", "0")) != 0:
        return 0
    ob = synth.config("c2")
    tmpdir = tempfile.mkdtemp(prefix="rc_oskar_ref_")
    path = os.path.join(tmpdir, "c2.vis")
    fsize, _ = _oskar_file(ob, path, "reference")
    for _ in range(min(args.warmup, 1)):
        K.read(path)
    t0 = time.perf_counter()
    for _ in range(args.steps):
        st, h, *_ = K.read(path)
    dt = (time.perf_counter() - t0) / args.steps
    os.remove(path)
    os.rmdir(tmpdir)
    P = h.num_points
    val = P / dt / 1e6
    line = {
        "metric": OSKAR_METRIC, "impl": "reference", "value": round(val, 3), "unit": "Mvis/s",
        "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": round(1e3 * dt, 2), "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f64", "data": "synthetic (seeded)",
        "config": {"workload": f"OSKAR .vis of c2: {P} points, {fsize} bytes, page cache",
                   "status": st},
        "cpu_baseline": {"value": round(val, 3), "unit": "Mvis/s", "cores": 1, "kind": "port",
                         "sample": "whole file, C restatement of mkFromFile + readAndReshuffle"},
        "e2e": {"value": round(val, 3), "unit": "Mvis/s", "h2d_bytes_per_step": 0,
                "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line))
    return 0


def main(argv=None):
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--config", default="c2")
    ap.add_argument("--tile", type=int, default=0)
    ap.add_argument("--threads", type=int, default=0)
    ap.add_argument("--cap", type=int, default=0)
    ap.add_argument("--bpc", type=int, default=0, help="bundles per CTA (0: tuned)")
    ap.add_argument("--no-graph", action="store_true")
    ap.add_argument("--no-tune", action="store_true", help="built-in defaults, no autotuning")
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--quick", action="store_true",
                    help="FP32 step, kernel times and error only (tuning sweeps)")
    ap.add_argument("--cpu-sample", type=int, default=0,
                    help="visibilities of the CPU legs (0: the whole observation)")
    ap.add_argument("--no-abi", action="store_true",
                    help="skip the reference-ABI strategy leg (config 2)")
    ap.add_argument("--no-target", action="store_true",
                    help="skip the config-4 target leg (config 2)")
    ap.add_argument("--c3-nt", type=int, default=216, help="time samples per baseline in c3")
    ap.add_argument("--c5-nt", type=int, default=64, help="time samples per baseline in c5")
    args = ap.parse_args(argv)
    if args.warmup < 3 and args.impl == "ours":
        args.warmup = 3
    if args.impl == "reference":
        return reference_arm_oskar(args) if args.config == "oskar" else reference_arm(args)
    if args.config == "oskar":
        return our_arm_oskar(args)
    if args.config == "c3":
        return our_arm_batch(args)
    if args.config == "c5":
        return our_arm_major_cycle(args)
    return our_arm(args)


if __name__ == "__main__":
    sys.exit(main())
