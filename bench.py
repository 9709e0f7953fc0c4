"""Throughput of the B200 Ros2 step (atmosphere-Ros2-steps per second).

Workload (one "step" = one Ros2 step of every atmosphere of the batch):
config-0-shaped atmospheres - a seeded element-balanced C/H/O/N network with
ni=69 species and 700+700 reactions, nz=120 layers, rate constants
log-uniform in [1e-40, 1e-8], mixing ratios log-uniform in [1e-20, 1],
dt = 1e-6 s - batched B atmospheres per GPU (default two per SM, 296 on a
B200; seeded per atmosphere and per rank), FP64. The same inputs are stepped
repeatedly (as the reference's benchmarks/bench_step.py does). Per-step
inputs (rates 398 MB, solver workspace 1.47 GB at B=296) exceed the 126 MB L2.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--batch B] [--impl b200|reference]

Multi-GPU: one process per GPU (torchrun); each rank steps its own batch
(weak scaling, no collective on the data path; the max over ranks of the
device time is taken with one all-reduce after the timed region).
"""
from __future__ import annotations

import argparse
import importlib
import json
import os
import statistics
import subprocess
import tempfile
import sys
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "atmosphere-Ros2-steps/s: batched mixed vs plain FP64, 1 B200, ≤1e-6 rel err"
UNIT = "atmosphere-steps/s"


def pkg(name):
    return importlib.import_module("jax-vulcan_b200." + name)


def rank_seeds(B, rank):
    """Seeds of the atmospheres a rank steps: disjoint across ranks (replicas
    over independent atmospheres, no data-path collective)."""
    return [1000 * rank + b for b in range(B)]


def max_over_ranks(x, dist, world, device):
    """The max of a per-rank timing over all ranks (one all-reduce)."""
    if world <= 1:
        return float(x)
    import torch
    t = torch.tensor([float(x)], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def job_value(world, B, ms):
    """Whole-job throughput: atmospheres of all ranks per second of the slowest rank."""
    return world * B / (ms * 1e-3)


def make_batch(B, rank, nz=120, mild=False):
    """The timed batch: config-0-shaped atmospheres seeded per rank. mild=False
    is the specified draw (k log-uniform in [1e-40, 1e-8]); mild=True divides
    each rate constant by n_max^(order-1), so the pseudo-first-order rates are
    log-uniform in [1e-40, 1e4] s^-1 (the well-conditioned draw)."""
    syn = pkg("synthetic")
    net = syn.make_network(0, 69, 700)
    kw = dict(mild=True, k_range=(-40.0, 4.0)) if mild else {}
    cases = [syn.make_case(seed=(sd,), net=net, nz=nz, **kw) for sd in rank_seeds(B, rank)]
    Y = np.stack([c.y for c in cases])
    K = np.stack([c.k for c in cases])
    DT = np.array([c.dt for c in cases])
    A = {}
    for key, v in cases[0].atm.items():
        A[key] = v if isinstance(v, bool) else np.stack([c.atm[key] for c in cases])
    return net, cases, Y, K, DT, A


class ClockSampler:
    """nvidia-smi clock/throttle sampling during the timed region."""

    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index):
        self.index = index
        self.proc = None
        self.path = os.path.join(tempfile.gettempdir(), f"vb_clocks_{os.getpid()}_rank{index}.csv")

    def start(self):
        try:
            os.makedirs(os.path.dirname(self.path), exist_ok=True)
            self.f = open(self.path, "w")
            self.proc = subprocess.Popen(["nvidia-smi", f"--id={self.index}", f"--query-gpu={self.Q}",
                                          "--format=csv,noheader,nounits", "-lms", "100"],
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
        sm, mx, reasons = [], None, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in open(self.path):
            parts = [p.strip() for p in line.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                mx = float(parts[2])
            except ValueError:
                continue
            for n, v in zip(names, parts[5:9]):
                if v.lower() == "active":
                    reasons.add(n)
        if not sm:
            return None
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": mx, "reasons": sorted(reasons),
                "samples": len(sm)}


def cpu_baseline_port(seconds=12.0, max_steps=40):
    """The oracle (NumPy/SciPy restatement of the reference step) on one
    config-0 atmosphere, single-threaded, bounded to ~`seconds`."""
    from threadpoolctl import threadpool_limits

    from oracle import ros2 as orc
    syn = pkg("synthetic")
    case = syn.config0()
    with threadpool_limits(1):
        orc.ros2_step(case.y, case.k, case.dt, case.atm, case.net.tables)
        n, t0 = 0, time.perf_counter()
        while n < max_steps and time.perf_counter() - t0 < seconds:
            orc.ros2_step(case.y, case.k, case.dt, case.atm, case.net.tables)
            n += 1
        el = time.perf_counter() - t0
    return {"value": n / el, "unit": UNIT, "cores": 1, "kind": "port",
            "sample": f"{n} single-atmosphere config-0 steps (ni=69, nr=1400, nz=120) of the NumPy/SciPy "
                      f"restatement of jax_step.jax_ros2_step, 1 thread, {el:.1f} s"}


_REF_CASE = None


def _ref_init():
    """Pool initializer: each worker builds the network and its own
    config-0-shaped atmosphere once (seeded by the worker's index), so the
    timed tasks run only the step."""
    global _REF_CASE
    import multiprocessing as mp
    syn = importlib.import_module("jax-vulcan_b200.synthetic")
    idx = mp.current_process()._identity[0] if mp.current_process()._identity else 0
    net = syn.make_network(0, 69, 700)
    _REF_CASE = syn.make_case(seed=(idx,), net=net)


def _ref_task(_):
    """One Ros2 step of this worker's atmosphere; returns its duration (s)."""
    from oracle import ros2 as orc
    c = _REF_CASE
    t0 = time.perf_counter()
    orc.ros2_step(c.y, c.k, c.dt, c.atm, c.net.tables)
    return time.perf_counter() - t0


def run_reference(args):
    """Reference arm: the reference's step restated on NumPy/SciPy (JAX is not
    installed) on all host cores, one single-threaded process per core; each
    timed step is a sample of the benchmark batch, one atmosphere per core."""
    import multiprocessing as mp
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    cores = len(os.sched_getaffinity(0))
    for v in ("OMP_NUM_THREADS", "OPENBLAS_NUM_THREADS", "MKL_NUM_THREADS"):
        os.environ[v] = "1"
    ctx = mp.get_context("spawn")
    B = args.batch or 296
    with ctx.Pool(cores, initializer=_ref_init) as pool:
        for _ in range(args.warmup):
            pool.map(_ref_task, range(cores), chunksize=1)
        task_s = []
        t0 = time.perf_counter()
        for _ in range(args.steps):
            task_s += pool.map(_ref_task, range(cores), chunksize=1)
        el = time.perf_counter() - t0
    value = cores * args.steps / el
    one = 1.0 / statistics.median(task_s)
    line = {"metric": METRIC, "value": value, "unit": UNIT, "n_gpus": args.gpus, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": 1e3 * el / args.steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f64", "impl": "reference",
            "data": "synthetic (seeded config-0-shaped atmospheres; stiff k log-uniform 1e-40..1e-8)",
            "config": {"workload": f"batched Ros2 step, {B} config-0-shaped atmospheres per GPU "
                                   f"(ni=69, nr=1400, nz=120, dt=1e-6)",
                       "batch_per_gpu": B, "ni": 69, "nr": 1400, "nz": 120, "precision": "fp64",
                       "sample_per_step": cores},
            "cpu_baseline": {"value": value, "unit": UNIT, "cores": cores, "kind": "port",
                             "sample": f"each step: {cores} of the batch's atmospheres x 1 Ros2 step, one "
                                       f"single-threaded process per core, network and atmosphere built "
                                       f"before timing (NumPy/SciPy restatement of jax_step.jax_ros2_step; "
                                       f"JAX absent)"},
            "single_thread": {"value": one, "unit": UNIT,
                              "note": "median single-atmosphere step time of the timed tasks"},
            "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


def oracle_check(net, cases, sol, delta, status, k1, k2, samples):
    """Correctness of a timed batch step, outside the timed region: status
    words and finiteness of every atmosphere, and for the sampled atmospheres
    the relative error of sol against the oracle (max and per species, floor
    1e-30), the normwise backward errors of both stage solves (k1, k2 read
    back from the workspace) and the largest Schur block condition number."""
    from oracle import ros2 as orc
    import torch
    st = status.cpu().numpy()
    finite = bool(torch.isfinite(sol).all().item()) and bool(torch.isfinite(delta).all().item())
    sol_h, k1_h, k2_h = sol.cpu().numpy(), k1.cpu().numpy(), k2.cpu().numpy()
    per_species, bwd, conds = None, 0.0, 0.0
    for b in samples:
        c = cases[b]
        sref, _, parts = orc.ros2_step(c.y, c.k, c.dt, c.atm, net.tables, return_parts=True)
        rel = (np.abs(sol_h[b] - sref) / np.maximum(np.abs(sref), 1e-30)).max(axis=0)
        per_species = rel if per_species is None else np.maximum(per_species, rel)
        bwd = max(bwd, *orc.stage_backward_errors(c.y, c.k, c.dt, c.atm, net.tables, k1_h[b], k2_h[b]))
        conds = max(conds, float(orc.schur_block_conditions(parts["diag"], parts["sup_neg"],
                                                            parts["sub_neg"]).max()))
    return {"status_ok": bool((st == 0).all()) and finite, "nonzero_status": int((st != 0).sum()),
            "finite": finite, "samples": list(samples),
            "max_rel_err_vs_oracle": float(per_species.max()),
            "per_species_max_rel_err_vs_oracle": [float(v) for v in per_species],
            "species_within_1e-10": int((per_species <= 1e-10).sum()),
            "stage_backward_error_max": bwd, "schur_block_cond_max": conds}


def kernel_launches(torch, fn):
    """Kernel launches of one fn() on the current stream's device, counted in a
    capture of it (a captured step holds the package's kernels and memory sets)."""
    from cuda.bindings import runtime as rt
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph, capture_error_mode="thread_local"):
        fn()
    handle = rt.cudaGraph_t(init_value=graph.raw_cuda_graph())

    def ok(res):
        if res[0] != rt.cudaError_t.cudaSuccess:
            raise RuntimeError(f"graph query: {res[0]}")
        return res[1:]

    n = ok(rt.cudaGraphGetNodes(handle))[-1]
    nodes = ok(rt.cudaGraphGetNodes(handle, n))[0]
    return sum(ok(rt.cudaGraphNodeGetType(v))[0] == rt.cudaGraphNodeType.cudaGraphNodeTypeKernel for v in nodes)


def fp64_peak_tflops(lib, torch, stream):
    out = torch.zeros(1, dtype=torch.float64, device="cuda")
    blocks, threads, iters = 148 * 16, 256, 4096
    lib.vb_fp64_probe(out.data_ptr(), blocks, threads, 64, stream)
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    best = 0.0
    for _ in range(3):
        e0.record()
        lib.vb_fp64_probe(out.data_ptr(), blocks, threads, iters, stream)
        e1.record()
        e1.synchronize()
        ms = e0.elapsed_time(e1)
        best = max(best, 2.0 * 8 * iters * blocks * threads / (ms * 1e-3) / 1e12)
    return best


def run_config2(args, torch):
    """The uneven batch: 256 atmospheres, nz ~ U[60, 200], ni in {30, 69, 89}
    (three networks), per-atmosphere T offset, Kzz scale and dt, stepped as
    one CUDA-graph replay of the multi-network batch, next to the same
    atmospheres stepped one at a time."""
    syn, chem, jstep = pkg("synthetic"), pkg("chem"), pkg("jax_step")
    nets, cases = syn.config2_batch(seed=2, batch=args.batch or 256)
    dev = {id(n): chem.to_device(n.tables) for n in nets.values()}
    items = [(dev[id(c.net)], jstep.atm_from_dict(c.atm), c.y, c.k, c.dt) for c in cases]
    # launch shapes per network group chosen by the autotuner on this GPU (the
    # automatic shapes and timed candidates: factor kernel, factor CTAs per SM,
    # sweep ring depth, layers per assembly CTA)
    batch = jstep.MultiNetworkBatch(items, tuning="tune")
    batch.capture()
    for _ in range(args.warmup):
        batch.step()
    torch.cuda.synchronize()
    clocks = ClockSampler(0)
    clocks.start()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(args.steps):
        batch.step()
    e1.record()
    torch.cuda.synchronize()
    clk = clocks.stop()
    ms = e0.elapsed_time(e1) / args.steps
    # the same atmospheres, one single-instance step after another
    singles = [(jstep.Ros2Step(it[0], it[1]), torch.as_tensor(it[2], device="cuda"),
                torch.as_tensor(it[3], device="cuda"), torch.full((1,), it[4], dtype=torch.float64, device="cuda"))
               for it in items]
    outs = [(torch.empty_like(y), torch.empty_like(y)) for _, y, _, _ in singles]
    for (st, y, k, dt), o in zip(singles, outs):
        st(y, k, dt, out=o)
    torch.cuda.synchronize()
    e0.record()
    for (st, y, k, dt), o in zip(singles, outs):
        st(y, k, dt, out=o)
    e1.record()
    torch.cuda.synchronize()
    seq_ms = e0.elapsed_time(e1)
    n = len(cases)
    layers = sum(c.y.shape[0] for c in cases)
    return {"metric": METRIC, "value": n / (ms * 1e-3), "unit": UNIT, "n_gpus": 1, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ms, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f64", "data": "synthetic (seeded uneven batch; stiff k)",
            "config": {"workload": f"uneven batch of {n} atmospheres, nz in [60, 200] ({layers} layers), "
                                   f"ni in {{30, 69, 89}} (370/1400/2000 reactions), one CUDA-graph replay",
                       "groups": len(batch.groups), "l2": "inputs larger than L2, no flush"},
            "sequential_single_instance": {"value": n / (seq_ms * 1e-3), "unit": UNIT, "ms_per_pass": seq_ms},
            "speedup_vs_sequential": seq_ms / ms, "gpu_launches": args.steps * sum(
                kernel_launches(torch, lambda g=g: g["step"](g["y"], g["k"], g["dt"], out=(g["sol"], g["delta"])))
                for g in batch.groups),
            "tuning": {k: {"tuning": v["tuning"], "ms": v["ms"], "candidates_ms": v["candidates"]}
                       for k, v in batch.tuned.items()},
            "clocks": clk}


def run_config3(args, torch):
    """The mixed-precision block solve at the SNCHO shape (ni=89, 2000
    reactions, nz=150, B=128): FP32 factor + FP64 refinement (<= 3 passes)
    with FP64 fallback, against the FP64 factor + solve, on the specified
    stiff rate constants (k in [1e-45, 1e-6]) and on order-scaled
    (well-conditioned) ones of the same shapes."""
    syn, chem, jstep, solver = pkg("synthetic"), pkg("chem"), pkg("jax_step"), pkg("solver")
    B = args.batch or 128
    net = syn.config3_case().net
    dn = chem.to_device(net.tables)
    out = {}
    for label, mild in (("stiff", False), ("well_conditioned", True)):
        cases = [syn.make_case(seed=(3000 + b,), ni=89, n_fwd=1000, nz=150, elements=("C", "H", "O", "N", "S"),
                               k_range=(-45.0, -6.0) if not mild else (-45.0, 4.0), mild=mild, net=net)
                 for b in range(B)]
        Y = torch.as_tensor(np.stack([c.y for c in cases]), device="cuda")
        K = torch.as_tensor(np.stack([c.k for c in cases]), device="cuda")
        A = {kk: (v if isinstance(v, bool) else np.stack([c.atm[kk] for c in cases])) for kk, v in cases[0].atm.items()}
        M = torch.as_tensor(A["M"], device="cuda")
        # the stage-1 system of the Ros2 step: c0 I - J - diag(diag_d), negated off-diagonals
        J = chem.chem_jac_analytical(Y, M, K, dn)
        diff, diag_d, sup_d, sub_d = jstep.diffusion(Y, jstep.atm_from_dict(A))
        dt = torch.as_tensor(np.array([c.dt for c in cases]), device="cuda")
        c0 = 1.0 / ((1.0 + 1.0 / np.sqrt(2.0)) * dt)
        eye = torch.eye(89, dtype=torch.float64, device="cuda")
        diag = c0[:, None, None, None] * eye - J - torch.diag_embed(diag_d)
        rhs = chem.chem_rhs(Y, M, K, dn) + diff
        sup_n, sub_n = -sup_d, -sub_d

        def timed(fn, reps=3):
            fn()
            torch.cuda.synchronize()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            for _ in range(reps):
                res = fn()
            e1.record()
            torch.cuda.synchronize()
            return e0.elapsed_time(e1) / reps, res

        t64, x64 = timed(lambda: solver.block_thomas_diag_offdiag(diag, sup_n, sub_n, rhs))
        tf64, _ = timed(lambda: solver.factor_block_thomas_diag_offdiag(diag, sup_n, sub_n))
        tf32, _ = timed(lambda: solver.factor_block_thomas_mixed(diag, sup_n, sub_n))

        def mixed():
            f = solver.factor_block_thomas_mixed(diag, sup_n, sub_n)
            x, passes = solver.solve_block_thomas_mixed(f, rhs, max_refine=3, tol=1e-13)
            return x, passes, f.status

        tmx, (xm, passes, status) = timed(mixed)
        rel = ((xm - x64).abs() / x64.abs().clamp_min(1e-30)).amax(dim=(0, 1)).cpu().numpy()
        st = status.cpu().numpy()
        out[label] = {"fp64_ms": t64, "mixed_ms": tmx, "speedup": t64 / tmx,
                      "fp64_factor_ms": tf64, "fp32_factor_ms": tf32,
                      "fallback_fraction": float(((st & 4) != 0).mean()),
                      "passes_max": int(passes.max().item()),
                      "max_rel_err_vs_fp64": float(rel.max()),
                      "per_species_max_rel_err_vs_fp64": [float(v) for v in rel]}
    return {"metric": "mixed-precision block solve vs FP64 (SNCHO shape)", "unit": "ms per batch solve",
            "higher_is_better": False, "config": {"workload": f"block solve of {B} SNCHO-shaped stage-1 systems "
                                                              f"(ni=89, nz=150)", "batch": B},
            "results": out}


def run_config1(args, torch):
    """The adaptive loop with photochemistry at the config-1 shapes (ni=69,
    700+700 reactions plus 40 photolysis branches, nz=120, 2500 bins over
    2-800 nm): every attempt is one Ros2 step, the loop body, the
    convergence update and, on the reference cadence, the photo branch of
    the atmospheres that are due, all on the device. Timed for one
    atmosphere (the latency of an adaptive step) and for a batch of
    atmospheres with their own initial states, each taking its own accept /
    reject / photo path; the atmosphere refresh runs every 100 accepted
    steps, as the reference's default `update_frq`. Rate constants: forward
    order-scaled (pseudo-first-order 1e-12 .. 1e4 /s; with the stiff config-0
    constants the reference contract force-accepts at dt_min with the state
    unchanged), reverse in detailed balance with a seeded equilibrium
    composition (synthetic.make_balanced_rates), so the chemistry relaxes;
    the batch then runs to the loop's own stop (the reference's default
    stopping rule) and the attempts and device time to that stop are
    reported."""
    syn, chem, jstep, loop, photo = pkg("synthetic"), pkg("chem"), pkg("jax_step"), pkg("outer_loop"), pkg("photo")
    ar = pkg("atm_refresh")
    net = syn.make_network(0, 69, 700, n_photo=40)
    dn = chem.to_device(net.tables)
    bins, din12 = syn.make_bins()
    nz = 120

    def setup(B):
        atms, extras = zip(*[syn.make_atmosphere((b,), net, nz=nz) for b in range(B)])
        A = {kk: (v if isinstance(v, bool) else np.stack([a[kk] for a in atms])) for kk, v in atms[0].items()}
        ph = syn.make_photo(0, net, atms[0]["Tco"], bins, din12)       # Tco is the same profile for every seed
        KY = [syn.make_balanced_rates((b,), net, nz, e["n"], -12.0, 4.0, M=a["M"]) for b, (a, e) in
              enumerate(zip(atms, extras))]
        K = np.stack([kk for kk, _ in KY])
        # start near each network's equilibrium composition (each mixing ratio
        # scaled by up to 2x), as a run restarted from a nearby state
        rng = np.random.default_rng(17)
        ymix0 = [ym * 10.0 ** rng.uniform(-0.3, 0.3, ym.shape) for _, ym in KY]
        ymix0 = [ym / ym.sum() for ym in ymix0]
        y0 = np.stack([ym[None, :] * e["n"][:, None] for ym, e in zip(ymix0, extras)])
        atom_ini = np.einsum("bzi,ia->ba", y0, net.compo)
        sm = np.concatenate([loop.slope_min_of(a["Kzz"], e["Hp"]) for a, e in zip(atms, extras)])
        refresh = ar.AtmRefreshStatic(pico=np.stack([e["pico"] for e in extras]), mol_mass=net.ms,
                                      diff_esc_idx=[0], pref_indx=0, zco_pref=0.0, gs=syn.GS, Rp=syn.RP)
        runner = loop.AdaptiveRunner(dn, jstep.atm_from_dict(A), loop.LoopStatics(dt_max=1e17), net.compo, atom_ini,
                                     batch=B, conv=loop.ConvStatics(use_photo=True), slope_min=sm,
                                     photo=photo.PhotoDevice(ph, nz), dz=np.stack([e["dz"] for e in extras]),
                                     flux_atol=1.0, refresh=refresh, update_frq=100)
        state = loop.LoopState(y0, y0 / y0.sum(axis=2, keepdims=True), 1e-10, np.zeros_like(atom_ini), rtol=0.2)
        runner.start(state)
        return runner, state, torch.as_tensor(K, device="cuda").contiguous()

    def timed(B, attempts):
        runner, state, k = setup(B)
        for _ in range(args.warmup):
            runner.attempt(state, k)
        torch.cuda.synchronize()
        n_photo = torch.zeros((), dtype=torch.int64, device="cuda")
        acc0 = state.scalars_host()["accept_count"].sum()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(attempts):
            n_photo += state.photo_due.sum()
            runner.attempt(state, k)
        e1.record()
        torch.cuda.synchronize()
        ms = e0.elapsed_time(e1)
        # the photo branch alone with every atmosphere due (on a copy of k made
        # before the timed region)
        due = torch.ones(B, dtype=torch.int32, device="cuda")
        k_copy = k.clone()
        torch.cuda.synchronize()
        e0.record()
        for _ in range(5):
            photo.photo_branch(runner.photo_carry, state.y, state.ymix, runner.dz, k_copy, runner.photo, due=due,
                               flux_atol=1.0)
        e1.record()
        torch.cuda.synchronize()
        sc = state.scalars_host()
        return {"batch": B, "attempts": attempts, "ms_per_attempt": ms / attempts,
                "value": B * attempts / (ms * 1e-3), "accepted": int(sc["accept_count"].sum() - acc0),
                "photo_updates": int(n_photo.item()), "photo_branch_ms_all_due": e0.elapsed_time(e1) / 5,
                "max_abs_atom_loss": float(np.abs(state.atom_loss.cpu().numpy()).max())}

    def to_stop(B, cap=4000):
        runner, state, k = setup(B)
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        n = runner.run_to_convergence(state, k, max_attempts=cap, check_every=100)
        e1.record()
        torch.cuda.synchronize()
        sc, cv = state.scalars_host(), state.conv_host()
        conv = (cv["longdy"] < runner.conv.yconv_min) & (cv["done"] == 1)
        return {"batch": B, "attempts": n, "ms": e0.elapsed_time(e1), "all_done": bool((cv["done"] == 1).all()),
                "stopped_converged": int(conv.sum()),
                "accepted_at_stop_median": float(np.median(sc["accept_count"])),
                "accepted_at_stop_max": int(sc["accept_count"].max()), "t_at_stop_median": float(np.median(sc["t"])),
                "max_abs_atom_loss": float(np.abs(state.atom_loss.cpu().numpy()).max())}

    B = args.batch or torch.cuda.get_device_properties(0).multi_processor_count
    single = timed(1, max(args.steps, 50))
    clocks = ClockSampler(0)
    clocks.start()
    batched = timed(B, args.steps)
    clk = clocks.stop()
    steady = to_stop(B)
    return {"metric": "adaptive-loop attempts/s (Ros2 step + body + convergence + photo on cadence)",
            "value": batched["value"], "unit": "atmosphere-attempts/s", "n_gpus": 1, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": batched["ms_per_attempt"], "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f64",
            "data": "synthetic (seeded config-1 shapes; order-scaled forward k, detailed-balance reverse k)",
            "config": {"workload": f"adaptive loop with photochemistry, {B} atmospheres of ni=69, nz=120, "
                                   f"2500 bins, 40 branches", "l2": "state larger than L2 at this batch, no flush"},
            "batched": batched, "single_atmosphere": single, "to_steady_state": steady,
            "gpu_launches_per_attempt": "8 or 9 (step) + 1 (body) + 1 (refresh) + 1 (convergence) + 3 (photo)",
            "clocks": clk}


def run_photo(args, torch):
    """The photo update alone at the config-1 shapes (nz=120, 2500 bins, 19
    absorbers of which 4 temperature dependent, 2 scatterers, 40 branches of
    which 10 temperature dependent) for B atmospheres: tau, flux and J timed
    separately with CUDA events, each against the HBM roofline of its
    algorithmic bytes (per-atmosphere arrays read / written once, the shared
    cross-section tables once per launch)."""
    import ctypes as C
    syn, photo, _lib = pkg("synthetic"), pkg("photo"), pkg("_lib")
    net = syn.make_network(0, 69, 700, n_photo=40)
    atm, extra = syn.make_atmosphere(0, net, nz=120)
    bins, din12 = syn.make_bins()
    dev = photo.PhotoDevice(syn.make_photo(0, net, atm["Tco"], bins, din12), 120)
    s = dev.struct
    B = args.batch or torch.cuda.get_device_properties(0).multi_processor_count
    nz, ni, nbin, nr = 120, 69, s.nbin, net.tables.nr
    y = torch.as_tensor(np.stack([extra["y"]] * B), device="cuda").contiguous()
    x = torch.as_tensor(np.stack([extra["ymix"]] * B), device="cuda").contiguous()
    dz = torch.as_tensor(np.stack([extra["dz"]] * B), device="cuda").contiguous()
    tau = torch.empty((B, nz + 1, nbin), dtype=torch.float64, device="cuda")
    af = torch.empty((B, nz, nbin), dtype=torch.float64, device="cuda")
    sf, dd, du = torch.empty_like(tau), torch.empty_like(tau), torch.zeros_like(tau)
    k = torch.zeros((B, nr + 1, nz), dtype=torch.float64, device="cuda")
    L = _lib.lib()
    sh = _lib.stream_handle()
    launches = {
        "tau": lambda: L.vb_photo_tau(B, nz, ni, C.addressof(s), y.data_ptr(), dz.data_ptr(), tau.data_ptr(), sh),
        "flux": lambda: L.vb_photo_flux(B, nz, ni, C.addressof(s), tau.data_ptr(), x.data_ptr(), du.data_ptr(),
                                        af.data_ptr(), sf.data_ptr(), dd.data_ptr(), du.data_ptr(), sh),
        "J": lambda: L.vb_photo_j(B, nz, nr, C.addressof(s), af.data_ptr(), None, None, k.data_ptr(), sh)}
    per_atm = {"tau": 8 * (nz * ni + nz + (nz + 1) * nbin),
               "flux": 8 * ((nz + 1) * nbin * 2 + nz * ni + nz * nbin + 3 * (nz + 1) * nbin),
               "J": 8 * (nz * nbin + (s.n_br + s.n_br_T) * nz)}
    shared = {"tau": 8 * nbin * (s.n_abs + s.n_scat + s.n_abs_T * nz),
              "flux": 8 * nbin * (s.n_abs + s.n_scat + s.n_abs_T * nz + 2),
              "J": 8 * nbin * (s.n_br + s.n_br_T * nz)}
    peak = json.load(open(os.path.join(ROOT, "MEASURED_PEAKS.json"))).get("hbm_gbs", 6650.0) \
        if os.path.exists(os.path.join(ROOT, "MEASURED_PEAKS.json")) else 6650.0
    for _ in range(args.warmup):
        for f in launches.values():
            f()
    torch.cuda.synchronize()
    clocks = ClockSampler(0)
    clocks.start()
    out = {}
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    for name, f in launches.items():
        e0.record()
        for _ in range(args.steps):
            f()
        e1.record()
        torch.cuda.synchronize()
        ms = e0.elapsed_time(e1) / args.steps
        bytes_ = B * per_atm[name] + shared[name]
        out[name] = {"ms_per_launch": ms, "algorithmic_bytes": bytes_, "achieved_gbs": bytes_ / (ms * 1e-3) / 1e9,
                     "hbm_frac": bytes_ / (ms * 1e-3) / 1e9 / peak}
    clk = clocks.stop()
    total = sum(v["ms_per_launch"] for v in out.values())
    return {"metric": "photo updates/s (tau + two-stream flux + J-rates into k)", "value": B / (total * 1e-3),
            "unit": "atmosphere-photo-updates/s", "n_gpus": 1, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": total, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
            "data": "synthetic (seeded config-1 photochemistry)",
            "config": {"workload": f"photo update of {B} atmospheres, nz=120, 2500 bins, 40 branches",
                       "l2": "flux arrays larger than L2 at B >= 8, no flush"},
            "kernels": out, "hbm_peak_gbs": peak, "clocks": clk}


def run_config4(args, torch):
    """The implicit steady-state adjoint, batched: for B atmospheres of the
    config-1 shape (ni=69, 700+700 Arrhenius / Lindemann reactions with NASA-9
    reverse rates plus 40 photolysis rows, nz=120, molecular diffusion and
    boundary fluxes on), the loss sum of seeded weights times log ymix at 10
    layers, and its gradient with respect to log k, T (through the rate
    constants, Tco and Ti), log Kzz and the boundary fluxes: one rate build
    with dk/dT, the block factor + transposed solve + VJP kernels, the
    transport-leaf VJP and the composition, per batch."""
    from types import SimpleNamespace
    syn, chem, jstep, ssg, rates, network = (pkg("synthetic"), pkg("chem"), pkg("jax_step"),
                                             pkg("steady_state_grad"), pkg("rates"), pkg("network"))
    net = network.parse_network_text(syn.make_rate_network(0, ni=69, n_fwd=700, n_kinf=60, n_nokinf=20, n_photo=40,
                                                           special=False))
    coeffs = syn.make_nasa9(0, net.ni)
    dn = chem.to_device(net)
    rt = rates.RateTables(net, coeffs)
    ms = np.random.default_rng(0).uniform(2.0, 60.0, net.ni)
    layers = np.random.default_rng(1).choice(120, 10, replace=False)

    def setup(B):
        atms, extras = zip(*[syn.make_atmosphere((b,), SimpleNamespace(tables=net, ms=ms), nz=120, moldiff=True,
                                                 fluxes=True) for b in range(B)])
        A = {kk: (v if isinstance(v, bool) else np.stack([a[kk] for a in atms])) for kk, v in atms[0].items()}
        y = torch.as_tensor(np.stack([e["y"] for e in extras]), device="cuda")
        w = torch.as_tensor(np.random.default_rng(2).normal(0.0, 1.0, (B, 10, net.ni)), device="cuda")
        return jstep.atm_from_dict(A), A, y, w

    def gradient(atm, A, y, w):
        T = torch.as_tensor(A["Tco"], device="cuda")
        M = torch.as_tensor(A["M"], device="cuda")
        k, dkdT = rt(T, M, with_dkdT=True)
        yv = y.clone().requires_grad_(True)
        ymix = yv[:, layers] / yv[:, layers].sum(dim=2, keepdim=True)
        (v,) = torch.autograd.grad((w * torch.log(ymix)).sum(), [yv])
        cot = ssg.implicit_cotangents(y, k, atm, dn, v)
        return dict(log_k=cot["k_arr"] * k, T=ssg.temperature_cotangent(cot, dkdT),
                    log_Kzz=cot["Kzz"] * torch.as_tensor(A["Kzz"], device="cuda"),
                    top_flux=cot["top_flux"], bot_flux=cot["bot_flux"], bot_vdep=cot["bot_vdep"],
                    status=cot["status"])

    def timed(B, reps):
        atm, A, y, w = setup(B)
        for _ in range(args.warmup):
            g = gradient(atm, A, y, w)
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(reps):
            g = gradient(atm, A, y, w)
        e1.record()
        torch.cuda.synchronize()
        ms_ = e0.elapsed_time(e1) / reps
        finite = all(bool(torch.isfinite(v).all()) for kk, v in g.items() if kk != "status")
        return {"batch": B, "ms_per_batch_gradient": ms_, "value": B / (ms_ * 1e-3), "finite": finite,
                "nonzero_status": int((g["status"] != 0).sum())}

    B = args.batch or 64
    reps = max(3, min(args.steps, 20))
    single = timed(1, reps)
    clocks = ClockSampler(0)
    clocks.start()
    batched = timed(B, reps)
    clk = clocks.stop()
    return {"metric": "implicit steady-state gradients/s (log k, T, log Kzz, boundary fluxes)",
            "value": batched["value"], "unit": "atmosphere-gradients/s", "n_gpus": 1, "steps": reps,
            "warmup": args.warmup, "ms_per_step": batched["ms_per_batch_gradient"], "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f64",
            "data": "synthetic (seeded config-1 shapes, rates from NASA-9; states not converged)",
            "config": {"workload": f"adjoint of {B} atmospheres, ni={net.ni}, nr={net.nr}, nz=120, loss over 10 "
                                   f"layers", "l2": "per-batch inputs larger than L2 at B=64, no flush"},
            "batched": batched, "single_atmosphere": single, "clocks": clk}


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=50)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--batch", type=int, default=0,
                    help="atmospheres per GPU (default: two per SM, 296 on a B200)")
    ap.add_argument("--impl", default="b200", choices=["b200", "reference"])
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--minimal", choices=["fp64", "mixed"], default=None,
                    help="profiling runs: only the warm-up and the timed steps of the config-0 batch with the "
                         "default launch shapes (plain FP64 or mixed step), one short JSON line")
    ap.add_argument("--workload", default="config0", choices=["config0", "config1", "config2", "config3",
                                                             "config4", "photo"],
                    help="config0: the headline batch (default); config1: the adaptive loop with "
                         "photochemistry; config2: the uneven multi-network batch; "
                         "config3: the mixed-precision block solve against FP64; config4: the batched "
                         "implicit adjoint; photo: the photo kernels against HBM")
    args = ap.parse_args()
    args.warmup = max(args.warmup, 3)
    if args.impl == "reference":
        run_reference(args)
        return

    import torch
    import torch.distributed as dist

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    if world > 1:
        from datetime import timedelta
        dist.init_process_group("nccl", timeout=timedelta(seconds=300))

    if args.workload in ("config1", "config2", "config3", "config4", "photo"):
        if rank == 0:
            run = {"config1": run_config1, "config2": run_config2, "config3": run_config3,
                   "config4": run_config4, "photo": run_photo}[args.workload]
            print(json.dumps(run(args, torch)), flush=True)
        return
    _lib = pkg("_lib")
    chem = pkg("chem")
    jstep = pkg("jax_step")
    L = _lib.lib()
    stream = torch.cuda.current_stream()
    sh = _lib.stream_handle(stream)

    B = args.batch or 2 * torch.cuda.get_device_properties(local).multi_processor_count
    net, cases, Y, K, DT, A = make_batch(B, rank)
    dn = chem.to_device(net.tables)
    atm = jstep.atm_from_dict(A)
    step = jstep.Ros2Step(dn, atm)
    y = torch.as_tensor(Y, device="cuda")
    k = torch.as_tensor(K, device="cuda")
    dt = torch.as_tensor(DT, device="cuda")
    sol = torch.empty_like(y)
    delta = torch.empty_like(y)

    def one():
        step(y, k, dt, out=(sol, delta))

    if args.minimal:
        if args.minimal == "mixed":
            step = jstep.Ros2Step(dn, atm, mixed=True)
        for _ in range(args.warmup):
            one()
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(args.steps):
            one()
        e1.record()
        torch.cuda.synchronize()
        ms = e0.elapsed_time(e1) / args.steps
        if rank == 0:
            print(json.dumps({"metric": METRIC, "value": B / (ms * 1e-3), "unit": UNIT, "ms_per_step": ms,
                              "minimal": args.minimal, "batch": B, "status_ok": bool((step.status == 0).all())}))
        return

    # launch shapes chosen by the project's autotuner on this GPU (factor kernel,
    # factor CTAs per SM, sweep ring depth, one or two streams), timed before
    # the measured region
    at = pkg("autotune")
    tuned, tune_ms = at.tune_group(dict(step=step, y=y, k=k, dt=dt, sol=sol, delta=delta), reps=3, split=True)
    launches = kernel_launches(torch, one)
    for _ in range(args.warmup):
        one()
    torch.cuda.synchronize()
    if world > 1:
        dist.barrier()
    clocks = ClockSampler(local)
    clocks.start()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    torch.cuda.synchronize()
    e0.record()
    for _ in range(args.steps):
        one()
    e1.record()
    torch.cuda.synchronize()
    clk = clocks.stop()
    ms = max_over_ranks(e0.elapsed_time(e1) / args.steps, dist, world, "cuda")
    if world > 1:
        dist.barrier()
    value = job_value(world, B, ms)

    # per-kernel device times over a separate profiled pass (events on the launch
    # stream; kernels serialised on one stream so each launch is attributed)
    at.set_tuning(dn, dict(tuned, streams=1))
    L.vb_profile(1)
    for _ in range(args.steps):
        one()
    torch.cuda.synchronize()
    site_ms = (np.zeros(8), np.zeros(8, dtype=np.int64))
    L.vb_profile_read(site_ms[0].ctypes.data, site_ms[1].ctypes.data, 8)
    L.vb_profile(0)
    check = oracle_check(net, cases, sol, delta, step.status, *step.stages(), samples=(0, B - 1)) \
        if rank == 0 else None

    # the FP64 factor kernels on the same batch (per-launch event split)
    variants = {}
    for vid, vname in ((2, "panel_gauss_jordan"), (3, "pipelined_gauss_jordan"), (4, "paired_gauss_jordan"),
                       (1, "blocked_dmma")):
        at.set_tuning(dn, dict(tuned, streams=1, factor_kernel=vid))
        for _ in range(args.warmup):
            one()
        torch.cuda.synchronize()
        L.vb_profile(1)
        for _ in range(args.steps):
            one()
        torch.cuda.synchronize()
        vms, vcnt = np.zeros(8), np.zeros(8, dtype=np.int64)
        L.vb_profile_read(vms.ctypes.data, vcnt.ctypes.data, 8)
        L.vb_profile(0)
        variants[vname] = {"factor_ms": float(vms[1] / max(vcnt[1], 1)),
                           "step_ms_sum_of_kernels": float(sum(vms[i] / max(vcnt[i], 1) for i in range(6)))}
    at.set_tuning(dn, tuned)
    names = _lib.PROFILE_SITES
    per_kernel = {n: {"ms_per_launch": float(site_ms[0][i] / max(site_ms[1][i], 1)),
                      "launches": int(site_ms[1][i])} for i, n in enumerate(names)}
    tot = sum(v["ms_per_launch"] for v in per_kernel.values())
    for v in per_kernel.values():
        v["share"] = v["ms_per_launch"] / tot if tot else 0.0

    # end to end through the public API with pinned host buffers: every step
    # copies its inputs in and its results out; the copies run on two copy
    # streams against double-buffered device arrays, so step i's inputs go
    # up and step i-1's results come down while the steps compute (one
    # compute stream: the steps share their workspace)
    y_h = torch.as_tensor(Y).pin_memory()
    dt_h = torch.as_tensor(DT).pin_memory()
    sol_h = [torch.empty_like(y_h).pin_memory() for _ in range(2)]
    delta_h = [torch.empty_like(y_h).pin_memory() for _ in range(2)]
    y_d = [torch.empty_like(y) for _ in range(2)]
    dt_d = [torch.empty_like(dt) for _ in range(2)]
    sol_d = [torch.empty_like(y) for _ in range(2)]
    delta_d = [torch.empty_like(y) for _ in range(2)]
    cs = torch.cuda.current_stream()
    up, down = torch.cuda.Stream(), torch.cuda.Stream()
    ev_in = [torch.cuda.Event() for _ in range(2)]
    ev_done = [torch.cuda.Event() for _ in range(2)]
    ev_out = [torch.cuda.Event() for _ in range(2)]

    def e2e_run(n):
        up.wait_stream(cs)
        for i in range(n):
            b2 = i % 2
            up.wait_event(ev_done[b2])                    # step i-2 has read this input slot
            with torch.cuda.stream(up):
                y_d[b2].copy_(y_h, non_blocking=True)
                dt_d[b2].copy_(dt_h, non_blocking=True)
                ev_in[b2].record(up)
            cs.wait_event(ev_in[b2])
            cs.wait_event(ev_out[b2])                     # step i-2's results are on the host
            step(y_d[b2], k, dt_d[b2], out=(sol_d[b2], delta_d[b2]), stream=cs)
            ev_done[b2].record(cs)
            down.wait_event(ev_done[b2])
            with torch.cuda.stream(down):
                sol_h[b2].copy_(sol_d[b2], non_blocking=True)
                delta_h[b2].copy_(delta_d[b2], non_blocking=True)
                ev_out[b2].record(down)
        for b2 in range(2):
            cs.wait_event(ev_out[b2])

    e2e_run(args.warmup)
    torch.cuda.synchronize()
    e0.record(cs)
    e2e_run(args.steps)
    e1.record(cs)
    torch.cuda.synchronize()
    e2e_ms = max_over_ranks(e0.elapsed_time(e1) / args.steps, dist, world, "cuda")
    h2d = y_h.numel() * 8 + dt_h.numel() * 8
    d2h = 2 * y_h.numel() * 8

    # plain single-instance FP64 step (one atmosphere; automatic launch shapes for
    # a batch of one, not the batch's tuning)
    at.set_tuning(dn, {})
    step1 = jstep.Ros2Step(dn, jstep.atm_from_dict(cases[0].atm))
    y1, k1, dt1 = y[:1].contiguous(), k[:1].contiguous(), dt[:1].contiguous()
    s1, d1 = torch.empty_like(y1), torch.empty_like(y1)
    for _ in range(3):
        step1(y1, k1, dt1, out=(s1, d1))
    torch.cuda.synchronize()
    n1 = max(3, args.steps)
    e0.record()
    for _ in range(n1):
        step1(y1, k1, dt1, out=(s1, d1))
    e1.record()
    torch.cuda.synchronize()
    single_ms = e0.elapsed_time(e1) / n1
    at.set_tuning(dn, tuned)

    # the same batch size on the well-conditioned draw (order-scaled rate
    # constants), where the step agrees with the oracle elementwise
    _, wcases, Yw, Kw, DTw, Aw = make_batch(B, rank, mild=True)
    stepw = jstep.Ros2Step(dn, jstep.atm_from_dict(Aw))
    yw, kw, dtw = (torch.as_tensor(v, device="cuda") for v in (Yw, Kw, DTw))
    solw, deltaw = torch.empty_like(yw), torch.empty_like(yw)
    for _ in range(args.warmup):
        stepw(yw, kw, dtw, out=(solw, deltaw))
    torch.cuda.synchronize()
    e0.record()
    for _ in range(args.steps):
        stepw(yw, kw, dtw, out=(solw, deltaw))
    e1.record()
    torch.cuda.synchronize()
    wc_ms = max_over_ranks(e0.elapsed_time(e1) / args.steps, dist, world, "cuda")
    wcheck = oracle_check(net, wcases, solw, deltaw, stepw.status, *stepw.stages(), samples=(0, B - 1)) \
        if rank == 0 else None

    # the mixed-precision step (FP32 row-equilibrated factor on the TF32
    # tensor cores, FP64 refinement, FP64 fallback) on both draws, same batch
    def mixed_run(stepm, yy, kk, dd, cs):
        sm_, dm_ = torch.empty_like(yy), torch.empty_like(yy)
        for _ in range(args.warmup):
            stepm(yy, kk, dd, out=(sm_, dm_))
        torch.cuda.synchronize()
        e0.record()
        for _ in range(args.steps):
            stepm(yy, kk, dd, out=(sm_, dm_))
        e1.record()
        torch.cuda.synchronize()
        mms = max_over_ranks(e0.elapsed_time(e1) / args.steps, dist, world, "cuda")
        st_m = stepm.status.cpu().numpy()
        out = {"value": job_value(world, B, mms), "unit": UNIT, "ms_per_step": mms,
               "fallback_fraction": float(((st_m & 4) != 0).mean()),
               "passes_max": int(stepm.passes.max().item()), "passes_mean": float(stepm.passes.float().mean())}
        if rank == 0:
            chk = oracle_check(net, cs, sm_, dm_, stepm.status, *stepm.stages(), samples=(0, B - 1))
            out.update(status_ok_or_fallback=bool(((st_m & ~4) == 0).all()) and chk["finite"],
                       max_rel_err_vs_oracle=chk["max_rel_err_vs_oracle"],
                       stage_backward_error_max=chk["stage_backward_error_max"],
                       per_species_max_rel_err_vs_oracle=chk["per_species_max_rel_err_vs_oracle"])
        return out

    at.set_tuning(dn, {})
    stepm = jstep.Ros2Step(dn, atm, mixed=True)
    mixed_stiff = mixed_run(stepm, y, k, dt, cases)
    stepmw = jstep.Ros2Step(dn, jstep.atm_from_dict(Aw), mixed=True)
    mixed_wc = mixed_run(stepmw, yw, kw, dtw, wcases)
    del stepm, stepmw
    at.set_tuning(dn, tuned)

    peak64 = fp64_peak_tflops(L, torch, sh)
    ni, nz = net.tables.ni, Y.shape[1]
    # Gauss-Jordan inverse of every layer block: ni^3 FMAs = 2*ni^3 flops counted
    fac_flops = B * nz * 2.0 * ni ** 3
    fac_ms = per_kernel["factor"]["ms_per_launch"]
    achieved = fac_flops / (fac_ms * 1e-3) / 1e12 if fac_ms > 0 else 0.0
    # algorithmic bytes of the factor: read each D_j, write each inverse (ni^2 doubles each)
    fac_bytes = B * nz * 2.0 * ni * ni * 8
    # DRAM read + write bytes of one factor launch measured by ncu, per atmosphere,
    # scaled to the batch: the panel factor, 160 atmospheres, 773.7 MB read +
    # 694.7 MB written
    fac_traffic = (773.72e6 + 694.66e6) / 160 * B
    peaks = {}
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            peaks = json.load(f)
    except (OSError, ValueError):
        pass
    hbm_peak = float(peaks.get("hbm_gbs", 6650.0))
    hbm_src = "MEASURED_PEAKS.json hbm_gbs" if "hbm_gbs" in peaks else "fallback 6650 GB/s"
    hbm_achieved = fac_bytes / (fac_ms * 1e-3) / 1e9 if fac_ms > 0 else 0.0

    if rank == 0:
        line = {
            "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ms, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f64",
            "data": "synthetic (seeded config-0-shaped atmospheres; stiff k log-uniform 1e-40..1e-8)",
            "config": {"workload": f"batched Ros2 step, {B} config-0-shaped atmospheres per GPU "
                                   f"(ni={ni}, nr={net.tables.nr}, nz={nz}, dt=1e-6)",
                       "batch_per_gpu": B, "ni": ni, "nr": int(net.tables.nr), "nz": int(nz),
                       "precision": "fp64", "parallelism": f"replicas x{world}",
                       "tuning": tuned, "tuning_candidates_ms": tune_ms,
                       "l2": f"inputs larger than L2 (rates {K.nbytes / 1e6:.0f} MB + solver workspace "
                             f"{step.ws_bytes / 1e6:.0f} MB per GPU), no flush"},
            "e2e": {"value": job_value(world, B, e2e_ms), "unit": UNIT, "h2d_bytes_per_step": int(h2d),
                    "d2h_bytes_per_step": int(d2h),
                    "note": "y and dt copied in from pinned host memory, sol and delta read back, every step, "
                            "on two copy streams with double-buffered device arrays (step i's inputs go up and "
                            "step i-1's results come down while the steps compute); rates and atmosphere stay "
                            "resident (as in the reference runner's device carry)"},
            # per step: diffusion rows, stage 1, factor, back sweep, diffusion rows,
            # stage 2 (one kernel by tiles of eight layers; rates and sums in batches
            # too small for tiles), forward sweep, back sweep (twice with two streams)
            "gpu_launches": launches * args.steps,
            "roofline": {"bound": "fp64", "kernel": "factor (Gauss-Jordan inverse with threshold partial pivoting of "
                                                    "each layer block, serial in z, one CTA per atmosphere)",
                         "achieved": achieved, "peak": peak64, "unit": "TFLOP/s",
                         "frac": achieved / peak64 if peak64 else None, "traffic": fac_traffic,
                         "traffic_source": "ncu dram__bytes_read.sum + dram__bytes_write.sum of one launch of "
                                           "the panel factor, per atmosphere, scaled to the batch",
                         "peak_source": "measured live: FP64 FMA probe kernel (vb_fp64_probe); "
                                        "MEASURED_PEAKS.json has no FP64 figure",
                         "algorithmic": f"2*ni^3 flops per layer block x {nz} layers x {B} atmospheres",
                         "hbm_view": {"achieved": hbm_achieved, "peak": hbm_peak, "unit": "GB/s",
                                      "frac": hbm_achieved / hbm_peak, "peak_source": hbm_src,
                                      "algorithmic": f"read D_j + write inverse, 2*ni^2*8 B per layer x "
                                                     f"{nz} x {B}"}},
            "kernels": per_kernel,
            "factor_variants": dict(variants, note="blocked_dmma: one warp per 8-column panel, "
                                                   "pivot steps inside the warp, rank-8 trailing updates on "
                                                   "the FP64 tensor cores (mma.sync m8n8k4); "
                                                   "panel_gauss_jordan (default): by panels of eight "
                                                   "columns, one block barrier per panel, the same "
                                                   "multiply-adds as a scalar elimination, on the "
                                                   "FP64 tensor cores"),
            "single_instance_fp64": {"value": 1.0 / (single_ms * 1e-3), "unit": UNIT, "ms_per_step": single_ms},
            "status_ok": check["status_ok"],
            "max_rel_err_vs_oracle": check["max_rel_err_vs_oracle"],
            "correctness": dict(check, note="the specified stiff draw makes a single step ill-conditioned "
                                            "(Schur block condition numbers far beyond 1/eps), so sol is checked "
                                            "by the backward errors of its two block solves; elementwise errors "
                                            "are reported, not bounded"),
            "mixed_precision": {"well_conditioned": mixed_wc, "stiff": mixed_stiff,
                                "vs_single_instance_fp64_well_conditioned":
                                    mixed_wc["value"] * single_ms * 1e-3,
                                "note": "vb_ros2_step_mixed: FP64 assembly, row-equilibrated FP32 "
                                        "Gauss-Jordan factor (the tuned factor kernel's FP32 instance: "
                                        f"factor_kernel {tuned.get('factor_kernel')}), FP64-residual "
                                        "refinement of both stages (<= 3 passes, tol 1e-12), FP64 refactor "
                                        "fallback; errors against the oracle on atmospheres 0 and B-1"},
            "well_conditioned": {"value": job_value(world, B, wc_ms), "unit": UNIT, "ms_per_step": wc_ms,
                                 "data": "same shapes, order-scaled rate constants (pseudo-first-order rates "
                                         "log-uniform in [1e-40, 1e4] s^-1)",
                                 "status_ok": wcheck["status_ok"],
                                 "max_rel_err_vs_oracle": wcheck["max_rel_err_vs_oracle"],
                                 "stage_backward_error_max": wcheck["stage_backward_error_max"],
                                 "per_species_max_rel_err_vs_oracle":
                                     wcheck["per_species_max_rel_err_vs_oracle"]},
            "clocks": clk,
        }
        if world == 1 and not args.no_cpu_baseline:
            line["cpu_baseline"] = cpu_baseline_port()
        print(json.dumps(line), flush=True)
    if world > 1:
        dist.barrier()
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
