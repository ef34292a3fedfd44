"""GLST energy+force throughput on B200 (one JSON line on rank 0).

Workload (N=1): 10,000 TIP3P-like waters (30,000 atoms), cubic box L = 66.9 A,
cutoff 10 A, splitting alpha = 0.31 1/A (tol = erfc(3.1)/10), the default
cubature order; mixed precision.  A step = one energy+force solve of that
system (glst_compute: assignment, near field, structure factors, shell sums,
long-range gather, combine).  Metric: atom-evals/s = atoms solved / second.

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

For N > 1 (torchrun, one rank per GPU) every rank solves its own copy of the
system (independent systems, no collective on the data path): weak scaling,
value = all ranks' atoms / max-over-ranks time.
--impl reference times the FP64 CPU restatement of the reference's GLST sum
(the reference ships no CPU implementation; its own code is CUDA) on the
host's cores: every timed step one complete solve of the same workload.
"""
import argparse
import json
import os
import statistics
import subprocess
import sys
import threading
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

import numpy as np  # noqa: E402

import __graft_entry__  # noqa: E402

METRIC = "atom-evals/s at <=1e-5 force RMS err vs FP64"
UNIT = "atom-evals/s"
WORKLOAD = "water10k"


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--workload", default=WORKLOAD)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-batch", action="store_true")
    ap.add_argument("--no-serve", action="store_true")
    ap.add_argument("--profile-batch", default=None, choices=["branches", "plain", "worklist"],
                    help="only create the 256-box batch and solve it twice in this mode (a short process "
                         "for an ncu launch list of the batch's kernels), then exit")
    ap.add_argument("--reference-log", default=None, metavar="PATH",
                    help="also write the flagship run as a log in the reference driver's layout "
                         "(test/full_example.cu), which utils/parse_glst_results.py reads")
    return ap.parse_args()


class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled during the timed region."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index):
        self.index = index
        self.proc = None
        self.lines = []

    def start(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.index), "--query-gpu=" + self.FIELDS,
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
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        sm, smax, reasons = [], None, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            parts = [p.strip() for p in ln.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                smax = float(parts[2])
            except ValueError:
                continue
            for nm, v in zip(names, parts[5:9]):
                if v.lower() == "active":
                    reasons.add(nm)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": smax,
                "reasons": sorted(reasons), "samples": len(sm)}


def dist_setup(args):
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    pg = None
    if world > 1:
        import datetime

        import torch.distributed as dist
        dist.init_process_group("nccl" if args.impl == "ours" else "gloo",
                                timeout=datetime.timedelta(seconds=120))
        pg = dist
    return world, rank, local, pg


def cpu_baseline_run(sysd, full=True, K_sample_div=32):
    """FP64 oracle on the host cores: one complete solve of the workload
    (assignment, structure factors, shell sums and gather over all K nodes,
    near field), timed by the wall clock.  full=False solves the near field
    and 1/K_sample_div of the nodes only (a warm-up that touches every code
    path in a fraction of the time)."""
    from oracle import oracle, planner
    g = __graft_entry__.load_package()
    store = planner.TDesignStore(g.TDESIGN_STORE)
    x, y, z, q = sysd["x"], sysd["y"], sysd["z"], sysd["q"]
    p = planner.make_plan(len(x), sysd["tol"], sysd["box"], sysd["rcut"], store)
    k1 = p.K if full else max(1, p.K // K_sample_div)
    t0 = time.perf_counter()
    oracle.glst(x, y, z, q, p, k0=0, k1=k1)
    t = time.perf_counter() - t0
    return dict(seconds_per_solve=t, cores=oracle.num_threads(), K=p.K, K_used=k1)


def run_reference(args, world, rank):
    """The reference's GLST sum on the host cores (the reference ships no CPU
    path; this is the FP64 oracle, a kernel-by-kernel restatement of its
    double path, OpenMP over all cores).  Warm-up steps solve the near field
    and 1/32 of the nodes; every timed step is one complete solve."""
    __graft_entry__.load_package()
    from glst_b200 import systems
    if rank != 0:
        return
    sysd = systems.config_system(args.workload, seed=0)
    n = len(sysd["x"])
    for _ in range(args.warmup):
        cpu_baseline_run(sysd, full=False)
    times = []
    info = None
    for _ in range(args.steps):
        info = cpu_baseline_run(sysd, full=True)
        times.append(info["seconds_per_solve"])
    sec = statistics.mean(times)
    val = n / sec
    sample = "every timed step one complete FP64 solve of the workload (all %d atoms, all %d nodes), wall clock" % (
        n, info["K"])
    line = {
        "impl": "reference", "metric": METRIC, "value": val, "unit": UNIT, "n_gpus": args.gpus,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": sec * 1e3, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic (seeded TIP3P-like water)",
        "config": {"workload": args.workload, "atoms": n, "nodes": info["K"], "sample": sample,
                   "warmup_steps": "near field + 1/32 of the nodes"},
        "cpu_baseline": {"value": val, "unit": UNIT, "cores": info["cores"], "kind": "port", "sample": sample},
        "e2e": {"value": val, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


def weak_throughput(local_ms, local_atoms, dist=None, device=None):
    """Whole-job throughput of independent per-rank work: every rank
    processed `local_atoms` in `local_ms`; the job takes the slowest rank's
    time (max over ranks) and processed world x local_atoms.  Returns
    (max_ms, atoms per second)."""
    world = 1
    if dist is not None and dist.is_initialized():
        import torch
        world = dist.get_world_size()
        t = torch.tensor([float(local_ms)], dtype=torch.float64, device=device)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        local_ms = float(t.item())
    return local_ms, world * local_atoms / (local_ms * 1e-3)


def series_fma(inf, nodes, n, gather):
    """FP32 fused multiply-adds of the far field's Chebyshev series for n atoms:
    per (atom, direction) P terms in the structure factors and two series of P
    terms in the gather, per (cell, node) a product over P terms.  P as the
    engine chooses it (planner.cpp, series_terms): the tail of the Bessel
    coefficients at the largest node, or weighted by the quadrature's w kappa."""
    if not inf.has_far_field:
        return 0.0
    kx, ky, kz, w, group = nodes
    tau = (np.arange(512) + 0.5) * np.pi / 512
    p_idx = np.arange(88)
    ops = 0.0
    for gi in range(inf.ngroup):
        m = group == gi
        n_rad = inf.group_gl_degree[gi] // 2
        n_dir = inf.group_nodes[gi] / n_rad
        kap = np.sqrt(kx[m] ** 2 + ky[m] ** 2 + kz[m] ** 2).reshape(n_rad, -1)[:, 0]
        z = kap * 1.02 * 0.5 * np.sqrt(3.0) * inf.cell_dim
        bes = np.abs(np.mean(np.cos(p_idx[None, :, None] * tau - z[:, None, None] * np.sin(tau)), axis=-1))
        wz = w[m].reshape(n_rad, -1)[:, 0] * z if gather else (z == z.max()).astype(float)
        tail = np.cumsum((2.0 * wz[:, None] * bes).sum(0)[::-1])[::-1]
        P = int(np.count_nonzero(tail > (1e-8 if gather else 2e-7) * wz.sum()))
        every = (2 if P <= 36 else 8) if gather else (2 if P <= 48 else 4)
        P = max(4, -(-P // every) * every)
        ops += n_dir * P * (float(n) * (2.0 if gather else 1.0) + float(inf.ncell_total) * n_rad)
    return ops


def run_batch(g, torch, dev, stream, fma_peak, n_steps=4, n_sys=256, seed=0):
    """256 independent water boxes of uneven size (300-30,000 atoms, two
    cubature orders): one captured graph over all systems vs the same systems
    solved one after another (one launch sequence each).  Also: the FP32
    floor of the pass (the series' FMAs of both passes over atoms at the
    measured FMA peak), and the same comparison per system-size class."""
    from glst_b200 import systems
    sy = systems.batch_uneven(n_sys, seed=seed)
    ops, per_grid = [], {}
    for s in sy:
        inf = g.plan(s["natom"], s["tol"], s["box"], s["rcut"], with_nodes=False)[0]
        key = (s["tol"], tuple(inf.ncell))
        if key not in per_grid:  # linear in the atoms
            inf, nodes = g.plan(s["natom"], s["tol"], s["box"], s["rcut"])
            per_grid[key] = [sum(series_fma(inf, nodes, n, gather) for gather in (False, True)) for n in (0, 1)]
        at0, at1 = per_grid[key]
        ops.append(at0 + s["natom"] * (at1 - at0))

    def floor_ms(idx):
        return sum(ops[i] for i in idx) / fma_peak * 1e3

    def timed(idx, steps):
        sub = [sy[i] for i in idx]
        ins = [torch.tensor(np.concatenate([s[k] for s in sub]), dtype=torch.float64, device=dev)
               for k in ("x", "y", "z", "q")]
        n = ins[0].numel()
        outs = [torch.empty(n, dtype=torch.float64, device=dev) for _ in range(4)]
        t0 = time.perf_counter()
        b = g.GlstBatch(sub, nstreams=16)
        t_create = time.perf_counter() - t0
        res = {}
        for name, mode in (("batched", "branches"), ("worklist", "worklist"), ("plain", "plain")):
            for _ in range(2):
                b.compute(*ins, *outs, mode=mode, stream=stream)
            torch.cuda.synchronize()
            e0 = torch.cuda.Event(enable_timing=True)
            e1 = torch.cuda.Event(enable_timing=True)
            e0.record(stream)
            for _ in range(steps):
                b.compute(*ins, *outs, mode=mode, stream=stream)
            e1.record(stream)
            torch.cuda.synchronize()
            ms = e0.elapsed_time(e1) / steps
            res[name] = {"ms_per_step": ms, "value": n / (ms * 1e-3)}
        b.close()
        del ins, outs
        torch.cuda.empty_cache()
        return n, res, t_create

    all_idx = list(range(len(sy)))
    n, res, t_create = timed(all_idx, n_steps)
    fl = floor_ms(all_idx)
    out = {"workload": "%d uneven water boxes, %d atoms (300-30,000 each), 2 cubature orders" % (n_sys, n),
           "unit": UNIT, "batched": res["batched"], "plain": res["plain"],
           "batched_definition": "one captured graph: every system's launch sequence on 16 parallel branches",
           "worklist": res["worklist"],
           "worklist_definition": "one captured graph: one launch per phase over the (system, block) work list",
           "ratio": res["plain"]["ms_per_step"] / res["batched"]["ms_per_step"],
           "floor_ms": fl, "batched_over_floor": res["batched"]["ms_per_step"] / fl,
           "plain_over_floor": res["plain"]["ms_per_step"] / fl,
           "floor_definition": "FP32 FMAs of the far field's series / measured FMA peak (%.3g/s)" % fma_peak,
           "create_s": t_create, "steps": n_steps}
    classes = {"small (< 3,000 atoms)": [i for i in all_idx if sy[i]["natom"] < 3000],
               "medium (3,000-19,999 atoms)": [i for i in all_idx if 3000 <= sy[i]["natom"] < 20000],
               "large (>= 20,000 atoms)": [i for i in all_idx if sy[i]["natom"] >= 20000]}
    out["by_size"] = {}
    for name, idx in classes.items():
        if not idx:
            continue
        nc, rc, _ = timed(idx, n_steps)
        out["by_size"][name] = {"systems": len(idx), "atoms": nc, "floor_ms": floor_ms(idx),
                                "batched_ms": rc["batched"]["ms_per_step"], "worklist_ms": rc["worklist"]["ms_per_step"],
                                "plain_ms": rc["plain"]["ms_per_step"],
                                "ratio": rc["plain"]["ms_per_step"] / rc["batched"]["ms_per_step"]}
    # The reference library's plain path on the same 256 systems (one solve
    # after another, calc_ener_force only), recorded earlier on a B200 with
    # the reference harness into the batch256 golden fixture: a recorded
    # figure, not measured in this run.
    gold = os.path.join(ROOT, "tests", "golden", "batch256_double.npz")
    if n_sys == 256 and seed == 0 and os.path.exists(gold):
        ref_ms = float(np.load(gold)["ms_host"].sum())
        out["reference_plain_recorded_not_measured_here"] = {
            "ms_per_step": ref_ms, "value": n / (ref_ms * 1e-3),
            "batched_ratio": ref_ms / res["batched"]["ms_per_step"],
            "source": "tests/golden/batch256_double.npz (reference harness, one B200, recorded)"}
    return out


def run_serve(g, n_requests=120, loads=(0.5, 0.8, 1.1), budget=150 << 30, nslots=8, seed=0):
    """Served request stream: requests of 1,000-200,000 atoms (log-uniform),
    60 % continuing a resident system with every atom displaced by
    N(0, 0.01 A); HBM budget 150 GB.  Capacity = requests/s with every
    request queued at once; then Poisson arrivals at 3 offered loads (fractions
    of that capacity), continuous batching (8 slots) vs one request at a time
    (1 slot).  Latency = submit to completion.  Each figure is the median
    (by throughput) of three runs; every run starts a new server, so its new
    systems are planned and allocated inside the run."""
    from glst_b200 import systems
    reqs = systems.request_stream(n_requests, seed=seed)
    atoms = sum(len(r["x"]) for r in reqs)

    def serve(nslots_, arrivals):
        with g.GlstServer(budget, nslots=nslots_) as srv:
            tickets = []
            t0 = time.perf_counter()
            for r, ta in zip(reqs, arrivals):
                dt = ta - (time.perf_counter() - t0)
                if dt > 0:
                    time.sleep(dt)
                tickets.append(srv.submit(r["key"], r["x"], r["y"], r["z"], r["q"], r["tol"], r["box"], r["rcut"]))
            lat = [srv.wait(t, timeout_ms=300000)[5] * 1e-3 for t in tickets]
            span = time.perf_counter() - t0
            st = srv.stats()
        lat.sort()
        return {"p50_ms": lat[len(lat) // 2], "p99_ms": lat[min(len(lat) - 1, int(0.99 * len(lat)))],
                "value": atoms / span, "requests_per_s": len(lat) / span,
                "evictions": int(st.evictions), "systems_created": int(st.systems_created)}

    def median_of(runs, nslots_, arrivals):
        # shared-box timing of ~1 s runs is noisy: the run with the median span
        res = sorted((serve(nslots_, arrivals) for _ in range(runs)), key=lambda r: r["requests_per_s"])
        out = dict(res[len(res) // 2])
        out["runs"] = runs
        return out

    zero = [0.0] * len(reqs)
    serve(nslots, zero)  # warm-up pass: plans, pinned staging, first kernel launches
    cap = median_of(3, nslots, zero)
    cap_plain = median_of(3, 1, zero)
    rng = np.random.default_rng(seed + 1)
    out = {"workload": "%d requests, %d atoms, 1,000-200,000 atoms each, 60%% continue a resident system"
                       % (len(reqs), atoms), "unit": UNIT, "budget_bytes": budget,
           "capacity": {"continuous_batching": cap, "one_at_a_time": cap_plain}, "loads": []}
    for f in loads:
        rate = f * cap["requests_per_s"]
        arr = np.cumsum(rng.exponential(1.0 / rate, len(reqs))).tolist()
        out["loads"].append({"offered": f, "rate_per_s": rate, "continuous_batching": median_of(3, nslots, arr),
                             "one_at_a_time": median_of(3, 1, arr)})
    return out


def write_reference_log(path, workload, g, f, inf, sysd, d, stream, dev, torch, iters=20):
    """The flagship system as the reference's driver reports it: per-phase
    times over `iters` solves (phases one after another, each bracketed by
    CUDA events), direct Coulomb on the GPU, error report vs Coulomb."""
    from glst_b200 import reports
    names = ["assign", "near_field", "structure_factors", "shell_sums", "long_range", "combine"]
    calls = [lambda: f.assign_atoms(*d, stream=stream), lambda: f.calc_sr_ef(stream=stream),
             lambda: f.calc_sf(stream=stream), lambda: f.sum_rmt_sf(stream=stream),
             lambda: f.calc_lr_ef(stream=stream), lambda: f.comm_ef(stream=stream)]
    per = {k: [] for k in names}
    for _ in range(iters):
        ev = [torch.cuda.Event(enable_timing=True) for _ in range(len(calls) + 1)]
        ev[0].record(stream)
        for i, c in enumerate(calls):
            c()
            ev[i + 1].record(stream)
        torch.cuda.synchronize()
        for i, k in enumerate(names):
            per[k].append(ev[i].elapsed_time(ev[i + 1]))
    glst = f.get_ef()
    n = len(sysd["x"])
    co = [torch.empty(n, dtype=torch.float64, device=dev) for _ in range(4)]
    c0, c1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    c0.record(stream)
    g.direct_coulomb(*d, *co, stream=stream)
    c1.record(stream)
    torch.cuda.synchronize()
    coul = [t.cpu().numpy() for t in co]
    L = sysd["box"]
    meta = {"sweep": "bench", "sys": workload, "tol": "%g" % sysd["tol"],
            "box_dim": "%g,%g,%g" % tuple(L), "cut": "%g" % sysd["rcut"], "requested_gpus": "1"}
    text = reports.format_run_log(meta, inf, L, per, c0.elapsed_time(c1), reports.error_stats(glst, coul),
                                  sysd["tol"])
    with open(path, "w") as fh:
        fh.write(text)


def run_ours(args, world, rank, local, dist):
    import torch
    g = __graft_entry__.load_package()
    from glst_b200 import systems
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    sysd = systems.config_system(args.workload, seed=0)
    n = len(sysd["x"])
    L = sysd["box"][0]
    f = g.GlstForce(n, sysd["tol"], L, L, L, rcut=sysd["rcut"])
    inf = f.info()
    d = [torch.tensor(sysd[k], dtype=torch.float64, device=dev) for k in ("x", "y", "z", "q")]
    stream = torch.cuda.current_stream(dev)
    flush = torch.empty(256 * 1024 * 1024, dtype=torch.uint8, device=dev)  # > 126 MB L2

    for _ in range(args.warmup):
        f.calc_ener_force(*d, stream=stream)
    torch.cuda.synchronize()
    f.check(stream=stream)

    # per-phase times of one instrumented step (same stream, CUDA events)
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(7)]
    flush.zero_()
    ev[0].record(stream)
    f.assign_atoms(*d, stream=stream)
    ev[1].record(stream)
    f.calc_sr_ef(stream=stream)
    ev[2].record(stream)
    f.calc_sf(stream=stream)
    ev[3].record(stream)
    f.sum_rmt_sf(stream=stream)
    ev[4].record(stream)
    f.calc_lr_ef(stream=stream)
    ev[5].record(stream)
    f.comm_ef(stream=stream)
    ev[6].record(stream)
    torch.cuda.synchronize()
    names = ["assign", "near_field", "structure_factors", "shell_sums", "long_range", "combine"]
    phases = {nm: ev[i].elapsed_time(ev[i + 1]) for i, nm in enumerate(names)}

    # timed region: K steps, L2 flushed between steps (outside the step events)
    starts = [torch.cuda.Event(enable_timing=True) for _ in range(args.steps)]
    ends = [torch.cuda.Event(enable_timing=True) for _ in range(args.steps)]
    clocks = ClockSampler(local)
    if dist:
        dist.barrier()
    torch.cuda.synchronize()
    clocks.start()
    time.sleep(0.3)
    wall0 = time.perf_counter()
    for i in range(args.steps):
        flush.zero_()
        starts[i].record(stream)
        f.calc_ener_force(*d, stream=stream)
        ends[i].record(stream)
    torch.cuda.synchronize()
    wall = time.perf_counter() - wall0
    clk = clocks.stop()
    step_ms = [s.elapsed_time(e) for s, e in zip(starts, ends)]
    total_ms, value = weak_throughput(sum(step_ms), n * args.steps, dist, dev)
    f.check(stream=stream)

    # end to end through the public API from pinned host memory
    hx = [torch.tensor(sysd[k], dtype=torch.float64).pin_memory() for k in ("x", "y", "z", "q")]
    ho = [torch.empty(n, dtype=torch.float64).pin_memory() for _ in range(4)]
    lib = g.load_library()

    def host_step():
        st = lib.glst_compute_host(f._h, *[t.data_ptr() for t in hx], *[t.data_ptr() for t in ho],
                                   stream.cuda_stream)
        if st:
            raise g.GlstError(st, lib.glst_last_error().decode())

    for _ in range(2):
        host_step()
    e_steps = max(3, args.steps // 2)
    torch.cuda.synchronize()
    if dist:
        dist.barrier()
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for _ in range(e_steps):
        host_step()
    e1.record(stream)
    torch.cuda.synchronize()
    e2e_ms, e2e_val = weak_throughput(e0.elapsed_time(e1), n * e_steps, dist, dev)

    # roofline of the dominant far-field kernel: FP32 FMAs of its Chebyshev series
    sfu_peak, fma_peak = g.measure_pipe_peaks()
    K = inf.num_nodes
    dom = max(("structure_factors", "long_range"), key=lambda k: phases[k])
    fma_ops = series_fma(inf, f.nodes(), n, dom == "long_range")
    fma_ach = fma_ops / (phases[dom] * 1e-3)
    roofline = {
        "bound": "fp32", "kernel": dom, "achieved": fma_ach / 1e9, "peak": fma_peak / 1e9,
        "unit": "G FP32 FMA/s", "frac": fma_ach / fma_peak, "ops_per_launch": fma_ops,
        "peak_source": "measured on this GPU by glst_measure_pipe_peaks (FP32 FMA loop)",
        "traffic": 2.991e8 if dom == "long_range" else 2.260e8,
        "traffic_source": "dram__bytes_read.sum + dram__bytes_write.sum of one ncu capture of this "
                          "kernel on this workload (profiles/water10k_solve_kernels.md)",
        "pairs_per_launch": float(n) * K,
        "sfu_peak_per_s": sfu_peak,
    }
    # The same kernel against the HBM roofline (MEASURED_PEAKS.json): its
    # algorithmic bytes are the cross-cell operand it streams once (R read
    # for the gather, S written for the structure factors: C x K float2).
    C = inf.ncell_total
    hbm_bytes = C * K * 8.0
    hbm_peak, hbm_src = 6650.0, "fallback (no MEASURED_PEAKS.json)"
    mp = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(mp):
        try:
            hbm_peak, hbm_src = float(json.load(open(mp))["hbm_gbs"]), "MEASURED_PEAKS.json hbm_gbs (measured)"
        except (ValueError, KeyError):
            pass
    hbm_ach = hbm_bytes / (phases[dom] * 1e-3) / 1e9
    roofline["hbm"] = {"achieved": hbm_ach, "peak": hbm_peak, "unit": "GB/s", "frac": hbm_ach / hbm_peak,
                       "bytes_per_launch": hbm_bytes, "peak_source": hbm_src,
                       "reading": "not the bound: the kernel is bound by FP32 work, HBM carries its operand once"}

    line = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": total_ms / args.steps, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f32 phase series + f64 cell-relative/shell/energy",
        "data": "synthetic (seeded TIP3P-like water, no dataset)",
        "config": {"workload": args.workload, "atoms": n, "box_A": L, "rcut_A": sysd["rcut"],
                   "tol": sysd["tol"], "cells": list(inf.ncell), "groups": inf.ngroup, "nodes": K,
                   "node_stages": inf.node_stages, "device_bytes": int(inf.device_bytes),
                   "parallelism": "dp%d (independent systems)" % world,
                   "l2": "flushed (256 MB write) between timed steps"},
        "clocks": clk,
        "e2e": {"value": e2e_val, "unit": UNIT, "h2d_bytes_per_step": 4 * 8 * n, "d2h_bytes_per_step": 4 * 8 * n,
                "path": "glst_compute_host (pinned host buffers, H2D + solve + D2H per step)"},
        "gpu_launches": int(inf.kernels_per_compute) * args.steps,
        "phases_ms": phases,
        "phases_note": ("phase by phase through the reference's phase methods; with several node stages "
                        "calc_sf runs the whole staged far field" if inf.node_stages > 1 else
                        "phase by phase through the reference's phase methods"),
        "roofline": roofline,
        "wall_s_timed": wall,
    }
    if rank == 0 and args.reference_log:
        write_reference_log(args.reference_log, args.workload, g, f, inf, sysd, d, stream, dev, torch, iters=20)
    if world == 1 and not args.no_batch:
        line["batched_vs_plain"] = run_batch(g, torch, dev, stream, fma_peak, n_steps=max(2, args.steps // 5))
    if world == 1 and not args.no_serve:
        f.close()
        torch.cuda.empty_cache()
        line["served"] = run_serve(g)
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        cb = cpu_baseline_run(sysd, full=True)
        line["cpu_baseline"] = {"value": n / cb["seconds_per_solve"], "unit": UNIT, "cores": cb["cores"],
                                "kind": "port",
                                "sample": "one complete FP64 oracle solve of the workload (%d atoms, %d nodes): "
                                          "%.1f s wall clock" % (n, cb["K"], cb["seconds_per_solve"])}
    if rank == 0:
        print(json.dumps(line), flush=True)
    f.close()


def profile_batch(mode):
    import torch
    g = __graft_entry__.load_package()
    from glst_b200 import systems
    dev = torch.device("cuda", 0)
    sy = systems.batch_uneven(256, seed=0)
    ins = [torch.tensor(np.concatenate([s[k] for s in sy]), dtype=torch.float64, device=dev)
           for k in ("x", "y", "z", "q")]
    outs = [torch.empty(ins[0].numel(), dtype=torch.float64, device=dev) for _ in range(4)]
    with g.GlstBatch(sy, nstreams=16) as b:
        for _ in range(2):
            b.compute(*ins, *outs, mode=mode)
        torch.cuda.synchronize()


def main():
    args = parse()
    if args.profile_batch:
        profile_batch(args.profile_batch)
        return
    world, rank, local, dist = dist_setup(args)
    try:
        if args.impl == "reference":
            run_reference(args, world, rank)
        else:
            run_ours(args, world, rank, local, dist)
    finally:
        if dist:
            dist.destroy_process_group()


if __name__ == "__main__":
    main()
