#!/usr/bin/env python
"""Benchmark of the linear PMCHWT solve on B200: solves/s (assemble + LU + solve).

Workload (N=1): the mixed-precision solve at scale -- an icosphere of radius
50 nm subdivided 4 times (5120 triangles, 7680 RWG edges, 15360 PMCHWT
unknowns, complex128), interior eps = -9 + 1.3i, vacuum outside, vacuum
wavelength 600 nm, x-polarised plane wave along +z.  One step = one solve:
system-matrix assembly + right-hand side + LU factorisation + solve with FP64
iterative refinement to a relative residual <= 1e-12.  The FP64 path is timed
beside it ("fp64"), and sigma_ext of both is compared with the CPU oracle's FP64
solve of the same workload (tests/golden/oracle_sphere_s4.npz).  The timed
steps run with the kernel timers off; per-kernel times and rooflines come from
a separate profiled pass right after.

Data are synthetic (a seeded icosphere; no dataset exists for this path).  The
3.8 GB FP64 matrix exceeds the 126 MB L2, so no L2 flush is needed between steps.

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl reference]

For N > 1 (torchrun) every rank solves its own wavelength, a shard of a
wavelength sweep (the path has no data exchange at one wavelength); the step
time is the max over ranks.
"""
from __future__ import annotations

import argparse
import csv
import io
import json
import os
import statistics
import subprocess
import sys
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(ROOT, "for90-mom2_b200")
sys.path.insert(0, PKG)

METRIC = "solves/s (assemble+LU+solve), mixed vs FP64 on 1 B200 at sigma_ext rel err <=1e-6"
WL = 600e-9
SHARD_DWL = 5e-9  # with N ranks, rank r solves the wavelength WL + SHARD_DWL r (a wavelength-sweep shard)
EPS_IN = complex(-9.0, 1.3)
SUBDIV = 4
RADIUS_NM = 50.0
TOL = 1e-12
MAXIT = 60


def workload_name(subdiv):
    F = 20 * 4 ** subdiv
    return "icosphere r=50nm s=%d (%d triangles, %d unknowns), eps=-9+1.3i, 600 nm, x-pol pw +z" % (
        subdiv, F, 3 * F)


def dist_env():
    return int(os.environ.get("RANK", 0)), int(os.environ.get("LOCAL_RANK", 0)), int(os.environ.get("WORLD_SIZE", 1))


def load_peaks():
    path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(path):
        with open(path) as fh:
            d = json.load(fh)
        return d.get("hbm_gbs", 6650.0), d.get("bf16_tflops", 1590.0), "measured"
    return 6650.0, 1590.0, "fallback"


class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled during the timed region."""

    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,clocks_event_reasons.hw_slowdown,"
         "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
         "clocks_event_reasons.sw_power_cap")

    def __init__(self, dev):
        self.dev = dev
        self.p = None

    def start(self):
        try:
            self.p = subprocess.Popen(["nvidia-smi", "-i", str(self.dev), "--query-gpu=" + self.Q,
                                       "--format=csv,noheader,nounits", "-lms", "200"],
                                      stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
        except OSError:
            self.p = None

    def stop(self):
        if self.p is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.p.terminate()
        out, _ = self.p.communicate(timeout=10)
        rows = [r for r in csv.reader(io.StringIO(out)) if len(r) >= 9]
        sm, mx, reasons = [], None, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for r in rows:
            try:
                sm.append(float(r[1]))
                mx = float(r[2])
            except ValueError:
                continue
            for nm, v in zip(names, r[5:9]):
                if v.strip().lower() == "active":
                    reasons.add(nm)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": mx, "reasons": sorted(reasons),
                "samples": len(sm)}


def make_problem(M, subdiv):
    import numpy as np
    from mom_b200 import meshgen
    nodes, faces = meshgen.icosphere(subdiv, RADIUS_NM)
    ids = np.ones(len(faces), dtype=np.int32)
    return nodes, faces, ids, [[1], [-1]]


_LU_CACHE = {}


def _oracle():
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle as O
    return O


def cpu_lu_full(n, threads):
    """ZGETRF + ZGETRS (scipy's OpenBLAS, the LAPACK step of solve_multi_linsys) timed
    once at the full order n on a dense complex Gaussian matrix, which pivots like the
    PMCHWT matrix does (no diagonal dominance).  Cached per process."""
    if n in _LU_CACHE:
        return _LU_CACHE[n]
    import numpy as np
    from scipy.linalg import lapack
    os.environ.setdefault("OMP_NUM_THREADS", str(threads))
    rng = np.random.default_rng(0)
    A = np.empty((n, n), dtype=np.complex128, order="F")
    for j in range(0, n, 1024):  # column blocks: bounded temporaries
        w = min(1024, n - j)
        A[:, j:j + w] = rng.standard_normal((n, w)) + 1j * rng.standard_normal((n, w))
    t0 = time.perf_counter()
    lu, piv, info = lapack.zgetrf(A, overwrite_a=True)
    t_lu = time.perf_counter() - t0
    swaps = int(np.count_nonzero(piv != np.arange(n)))
    b = rng.standard_normal(n) + 0j
    t0 = time.perf_counter()
    lapack.zgetrs(lu, piv, b)
    t_rs = time.perf_counter() - t0
    del lu, A
    _LU_CACHE[n] = (t_lu, t_rs, swaps)
    return _LU_CACHE[n]


def cpu_calibration(subdiv, threads, m_s):
    """Checks the row-sample extrapolation of the CPU assembly on the next smaller
    sphere (subdiv - 1): one full, unsampled oracle sysmat against the same
    m_s-row sample scaled by F / m_s.  Also times ZGETRF on that assembled PMCHWT
    matrix against a Gaussian matrix of the same order."""
    import numpy as np
    from scipy.linalg import lapack
    from mom_b200 import meshgen
    O = _oracle()
    nodes, faces = meshgen.icosphere(subdiv, RADIUS_NM)
    P = O.OracleProblem(nodes, faces, np.ones(len(faces), int), 1e-9, [[1], [-1]])
    F = len(faces)
    om = O.omega_of(WL)
    ri = [1.0, np.sqrt(EPS_IN)]
    t0 = time.perf_counter()
    A = P.sysmat(om, ri, nthreads=threads)
    t_full = time.perf_counter() - t0
    t0 = time.perf_counter()
    P.sysmat_sample(om, ri, 0, m_s, threads)
    t_smp = (time.perf_counter() - t0) * F / m_s
    n = A.shape[0]
    t0 = time.perf_counter()
    lu, piv, info = lapack.zgetrf(A, overwrite_a=True)
    t_lu_real = time.perf_counter() - t0
    t_lu_rand = cpu_lu_full(n, threads)[0]
    return {"workload": workload_name(subdiv), "assembly_full_s": t_full, "assembly_sample_extrapolated_s": t_smp,
            "extrapolation_over_full": t_smp / t_full, "zgetrf_pmchwt_s": t_lu_real, "zgetrf_gaussian_s": t_lu_rand,
            "zgetrf_pmchwt_row_swaps": int(np.count_nonzero(piv != np.arange(n)))}


class CpuBaseline:
    """The CPU oracle (C + OpenMP restatement of the reference's loops, OpenBLAS
    ZGETRF/ZGETRS) on one solve of the workload.  Measured per call: the sysmat
    work of m_s test-face rows of every domain, srcvec and cs_prtsrf in full.
    Measured once per process: ZGETRF/ZGETRS at the full order.  Modelled: the
    assembly as the row sample times F / m_s (every test-face row does the same
    work: F source faces, near pairs uniform on the sphere), checked against a
    full assembly on the next smaller sphere (cpu_calibration)."""

    def __init__(self, subdiv, threads, m_s=64):
        import numpy as np
        from mom_b200 import meshgen
        O = _oracle()
        os.environ.setdefault("OMP_NUM_THREADS", str(threads))
        nodes, faces = meshgen.icosphere(subdiv, RADIUS_NM)
        self.O, self.threads = O, threads
        self.P = O.OracleProblem(nodes, faces, np.ones(len(faces), int), 1e-9, [[1], [-1]])
        self.F = len(faces)
        self.n = 2 * self.P.N
        self.m_s = max(2, min(self.F, m_s))
        self.om = O.omega_of(WL)
        self.ri = [1.0, np.sqrt(EPS_IN)]
        self.src = dict(type="pw", theta=0.0, phi=90 * O.DEGTORAD, psi=0.0)
        self.x = np.zeros(self.n, dtype=np.complex128)
        self.t_lu, self.t_rs, self.swaps = cpu_lu_full(self.n, threads)

    def step(self):
        """One step: the measured pieces of a solve; returns the modelled seconds per solve."""
        t0 = time.perf_counter()
        self.P.sysmat_sample(self.om, self.ri, 0, self.m_s, self.threads)
        t_asm = (time.perf_counter() - t0) * self.F / self.m_s
        t0 = time.perf_counter()
        self.P.srcvec(self.om, self.ri[0], self.src)
        t_rhs = time.perf_counter() - t0
        t0 = time.perf_counter()
        self.P.cs(self.om, self.ri[0], self.x, self.src)
        t_cs = time.perf_counter() - t0
        self.phases = dict(assembly=t_asm, rhs=t_rhs, lu=self.t_lu, getrs=self.t_rs, cs=t_cs)
        return sum(self.phases.values())

    def describe(self):
        return {"modelled": True,
                "model": "assembly = time of %d of %d test-face rows per domain x %d (measured each step); "
                         "ZGETRF + ZGETRS measured once at the full order n = %d on a Gaussian matrix "
                         "(%d row interchanges); srcvec and cs_prtsrf measured in full"
                         % (self.m_s, self.F, self.F // self.m_s, self.n, self.swaps),
                "sample": "sysmat rows %d/%d per domain, full-order zgetrf/zgetrs, full srcvec + cs; "
                          "OpenMP + OpenBLAS" % (self.m_s, self.F),
                "phases_s": self.phases}


def cpu_sample(subdiv, threads, calibrate=True):
    """cpu_baseline leg of the GPU arm: one CpuBaseline step plus the calibration."""
    cb = CpuBaseline(subdiv, threads)
    total = cb.step()
    out = dict(total_s=total, **cb.describe())
    if calibrate and subdiv > 1:
        out["extrapolation_check"] = cpu_calibration(subdiv - 1, threads, cb.m_s)
    return out


def reduce_max(x, world, device):
    """Max of a per-rank scalar over the process group (step times are taken as the max over ranks)."""
    if world == 1:
        return x
    import torch
    import torch.distributed as dist
    t = torch.tensor([x], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def replica_value(ms_per_step_max, world):
    """Whole-job solves/s of N independent replicas: every rank completes one solve per step."""
    return world * 1000.0 / ms_per_step_max


def host_cores():
    try:
        return len(os.sched_getaffinity(0))
    except AttributeError:
        return os.cpu_count() or 1


def bench_config(subdiv, world):
    """The workload description shared by both arms (identical dicts)."""
    return {"workload": workload_name(subdiv), "refine_tol": TOL,
            "l2": "matrix %.2f GB > 126 MB L2, no flush" % (16.0 * (3 * 20 * 4 ** subdiv) ** 2 / 1e9),
            "parallelism": ("wavelength shards x%d (rank r at 600 + %g r nm, one solve per rank per step)"
                            % (world, SHARD_DWL * 1e9) if world > 1 else "replicas x1")}


def run_reference(args, rank, world):
    """Reference arm: the CPU restatement of the reference's path (the Fortran
    reference cannot be compiled here: no Fortran compiler), all host threads.
    Each timed step measures the row sample of the assembly plus srcvec and
    cs_prtsrf; ZGETRF/ZGETRS are measured once at the full order during the
    warm-up.  The reported solves/s is the modelled full solve (CpuBaseline)."""
    if rank != 0:
        return 0
    cores = host_cores()
    cb = CpuBaseline(args.subdiv, cores)
    for _ in range(args.warmup):
        cb.step()
    t0 = time.perf_counter()
    totals = [cb.step() for _ in range(args.steps)]
    wall = time.perf_counter() - t0
    v = 1.0 / statistics.median(totals)
    desc = cb.describe()
    line = {"impl": "reference", "metric": METRIC, "value": v, "unit": "solves/s", "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1e3 / v, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "complex128", "data": "synthetic",
            "precision": "FP64 (CPU)", "config": bench_config(args.subdiv, world),
            "modelled": True, "timed_region_s": wall,
            "cpu_baseline": dict({"value": v, "unit": "solves/s", "cores": cores, "kind": "port"}, **desc),
            "e2e": {"value": v, "unit": "solves/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)
    return 0


def run_ours(args, rank, local_rank, world):
    import numpy as np
    import torch
    import mom_b200 as M
    torch.cuda.set_device(local_rank)
    if world > 1:
        import torch.distributed as dist
        from datetime import timedelta
        dist.init_process_group("nccl", timeout=timedelta(seconds=600))
    nodes, faces, ids, doms = make_problem(M, args.subdiv)
    S = M.Solver(local_rank)
    S.set_problem(M.Problem.from_arrays(nodes, faces, ids, 1e-9, doms))
    # each rank solves its own wavelength of a sweep of N wavelengths
    # WL + SHARD_DWL i (unit i on rank i); rank 0's is the 600 nm of the sigma fixture
    om = M.omega_of(WL + SHARD_DWL * rank)
    ri = [1.0, np.sqrt(EPS_IN)]
    src = [M.src_pw(0, 90, 0)]
    stream = torch.cuda.ExternalStream(S.stream)

    def step(prec):
        S.sysmat(om, ri, prec)
        S.srcvec(om, ri[0], src)
        S.solve(prec, tol=TOL, maxit=MAXIT, want_host=False)

    def barrier():
        torch.cuda.synchronize()
        if world > 1:
            torch.distributed.barrier()
        torch.cuda.synchronize()

    def max_over_ranks(x):
        return reduce_max(x, world, "cuda")

    def timed(prec, steps, warm):
        """Device time of `steps` solves with the kernel timers off (no events between launches)."""
        S.profile(False)
        for _ in range(warm):
            step(prec)
        barrier()
        l0, b0 = S.launch_count, S.library_calls
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        iters = []
        for _ in range(steps):
            step(prec)
            iters.append(S.iters)
        e1.record(stream)
        e1.synchronize()
        barrier()
        ms = e0.elapsed_time(e1) / steps
        return max_over_ranks(ms), S.launch_count - l0, S.library_calls - b0, iters

    def profiled(prec, steps):
        """Per-kernel device times from a separate pass of `steps` solves with the
        kernel timers on (CUDA events on the library stream around every launch
        category; inside the LU graph they are event nodes).  One untimed solve
        first captures the LU graph with its timing nodes."""
        S.profile(True)
        step(prec)
        S.profile(True)  # reset the counters
        f0 = S.tensor_flops
        for _ in range(steps):
            step(prec)
        prof = S.profile_read()
        S.profile(False)
        barrier()
        return prof, S.tensor_flops - f0

    # ---- mixed precision (the headline) ----
    sampler = ClockSampler(local_rank)
    sampler.start()
    ms_mixed, launches, libcalls, iters = timed(M.MIXED, args.steps, args.warmup)
    clocks = sampler.stop()
    csca, cabs = S.cross_sections(om, ri[0], src)
    ext_mixed = float(csca[0] + cabs[0])
    psteps = max(1, min(args.steps, 5))
    prof, tc_flops = profiled(M.MIXED, psteps)
    # ---- FP64 path, same workload ----
    ms_fp64, prof64, ext_fp64 = None, {}, None
    if args.fp64_steps > 0:
        ms_fp64, _, _, _ = timed(M.FP64, args.fp64_steps, 1)
        csca64, cabs64 = S.cross_sections(om, ri[0], src)
        ext_fp64 = float(csca64[0] + cabs64[0])
        prof64, _ = profiled(M.FP64, 1)

    # ---- end to end through the C ABI with pinned host buffers ----
    e2e_ms = None
    if not args.no_e2e:
        pin_x = torch.empty((1, 2 * S.N * 2), dtype=torch.float64, pin_memory=True).numpy()
        xh = pin_x.view(np.complex128).reshape(2 * S.N, 1, order="F")
        S.solve_wavelength(om, ri, src, M.MIXED, TOL, MAXIT, want_host=True)
        barrier()
        t0 = time.perf_counter()
        for _ in range(args.steps):
            x = S.solve_wavelength(om, ri, src, M.MIXED, TOL, MAXIT, want_host=True)
            xh[:, 0] = x[:, 0]
            S.cross_sections(om, ri[0], src)
        torch.cuda.synchronize()
        e2e_ms = max_over_ranks((time.perf_counter() - t0) * 1e3 / args.steps)
    h2d = 48 * len(src) + 16 * len(ri)  # mom_src structs + refractive indices
    d2h = 16 * 2 * S.N * len(src) + 16 * len(src)  # solution + (csca, cabs)

    # ---- rooflines of the timed kernels (device times of the profiled pass) ----
    hbm_gbs, bf16_tf, peak_src = load_peaks()
    F = len(faces)
    n = 2 * S.N
    nb = 64
    sm_mhz = clocks.get("sm_mhz") or 1965.0
    roofs = {}
    ms, cnt = prof["tc_gemm"]
    if cnt:
        ach = tc_flops / (ms * 1e-3) / 1e12
        roofs["tc_gemm"] = {"kernel": "tc_gemm_kernel (tcgen05 kind::f16, 3 passes on two-part FP16 operands, LU trailing update)",
                            "bound": "tensor", "achieved": ach, "unit": "TFLOP/s", "peak": bf16_tf,
                            "frac": ach / bf16_tf, "traffic": None,
                            "peak_note": "%s bf16 burst peak (FP16 has the same rate); FLOP = 3 passes executed" % peak_src}
    ms, cnt = prof["panel"]
    if cnt:
        bytes_ = sum(2.0 * 8 * (n - k * nb) * nb for k in range(n // nb)) * psteps  # FP32 panel read + write
        ach = bytes_ / (ms * 1e-3) / 1e9
        # DRAM bytes of one panel (four subpanels of 0.539 MB, ncu capture at 3,648
        # rows), scaled by rows to the average panel height of this order
        traffic = 4 * 0.539e6 * (n / 2.0) / 3648.0
        roofs["panel"] = {"kernel": "panel_reg_kernel<float2> (pivoted panel in the registers of one cluster, one exchange per column)",
                          "bound": "hbm", "achieved": ach, "unit": "GB/s", "peak": hbm_gbs, "frac": ach / hbm_gbs,
                          "traffic": traffic, "traffic_note": "bytes per launch, ncu at 3648 rows scaled by rows",
                          "peak_note": "%s; latency-bound: one pivot exchange per column over the cluster" % peak_src}
    ms, cnt = prof["pair"]
    if cnt:
        # 169 point pairs x 88 FLOP per unordered face pair (each evaluated once and
        # used for both blocks) + a 3,042-FLOP contraction per block, F^2 blocks per
        # launch (one domain); 17,914 FLOP per face pair when every ordered pair is
        # evaluated (MOM_PAIR_SYM=0)
        if os.environ.get("MOM_PAIR_SYM", "1") != "0":
            flop = (14872.0 * F * (F + 1) / 2.0 + 3042.0 * F * F) * cnt
        else:
            flop = 17914.0 * F * F * cnt
        ach = flop / (ms * 1e-3) / 1e12
        peak = 148 * 128 * 2 * sm_mhz * 1e6 / 1e12
        roofs["pair"] = {"kernel": "pair_kernel<float,13> (far-pair assembly, FP32 pipe)", "bound": "fp32",
                         "achieved": ach, "unit": "TFLOP/s", "peak": peak, "frac": ach / peak,
                         "traffic": 430.4e6 * (F / 1280.0) ** 2,
                         "traffic_note": "bytes per launch, ncu at 1280 faces scaled by face pairs",
                         "peak_note": "nominal FP32 SIMT at the sampled SM clock %.0f MHz" % sm_mhz}
    ms, cnt = prof["trsv"]
    if cnt:
        bytes_ = 8.0 * n * n * cnt  # FP32 L and U factors read once per solve
        ach = bytes_ / (ms * 1e-3) / 1e9
        roofs["trsv"] = {"kernel": "trsv_flow_kernel<float2> (forward+backward substitution, published solved blocks)",
                         "bound": "hbm", "achieved": ach, "unit": "GB/s", "peak": hbm_gbs, "frac": ach / hbm_gbs,
                         "traffic": 125.4e6 * (n / 3840.0) ** 2,
                         "traffic_note": "bytes per launch, ncu at 3840 unknowns scaled by n^2",
                         "peak_note": peak_src}
    ms, cnt = prof["residual"]
    if cnt:
        bytes_ = 16.0 * n * n * cnt  # FP64 matrix read once per residual
        ach = bytes_ / (ms * 1e-3) / 1e9
        roofs["residual"] = {"kernel": "gemv_partial_kernel (FP64 refinement residual)", "bound": "hbm",
                             "achieved": ach, "unit": "GB/s", "peak": hbm_gbs, "frac": ach / hbm_gbs,
                             "traffic": None, "peak_note": peak_src}
    top = max(roofs, key=lambda k: prof[k][0])  # the kernel with the most device time per step
    roof = dict(roofs[top])
    roof["timing"] = "separate profiled pass of %d solves after the timed region" % psteps

    phases = {k: {"ms_per_step": v[0] / psteps, "launches_per_step": v[1] / psteps} for k, v in prof.items()}
    # the LU's kernels on both streams against its wall time: the look-ahead
    # runs the panels of the next outer block beside the trailing update
    lu_kernels = sum(prof[k][0] for k in ("panel", "gemm", "pivot_aux", "diag_inv")) / psteps
    lu_overlap = {"lu_wall_ms": prof["lu"][0] / psteps, "lu_kernels_sum_ms": lu_kernels,
                  "panel_ms": prof["panel"][0] / psteps,
                  "hidden_ms": lu_kernels - prof["lu"][0] / psteps}
    phases64 = {k: {"ms_per_step": v[0]} for k, v in prof64.items()}

    # sigma_ext against the oracle's FP64 solve of this workload (committed fixture)
    ref_ext = None
    fx = os.path.join(ROOT, "tests", "golden", "oracle_sphere_s%d.npz" % args.subdiv)
    if os.path.exists(fx):
        ref_ext = float(np.load(fx)["sigma"][2])

    def rel(a, b):
        return abs(a - b) / abs(b) if (a is not None and b) else None

    value = replica_value(ms_mixed, world)
    line = {"metric": METRIC, "value": value, "unit": "solves/s", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ms_mixed, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "fp32 far pairs + LU (fp32-accurate fp16x2 tensor-core updates), fp64 near pairs + refinement (complex)",
            "data": "synthetic", "precision": "mixed", "config": bench_config(args.subdiv, world),
            "gpu_launches": int(launches), "library_gemm_calls": libcalls,
            "roofline": roof, "clocks": clocks,
            "e2e": ({"value": world * 1000.0 / e2e_ms, "unit": "solves/s", "h2d_bytes_per_step": h2d,
                     "d2h_bytes_per_step": d2h} if e2e_ms else None)}
    if not args.no_extras and world == 1:
        for key, fn in (("sweep", lambda: bench_sweep(M, args.sweep_workers, local_rank)),
                        ("adjoint", lambda: bench_adjoint(M, local_rank)),
                        ("core_shell", lambda: bench_core_shell(M, local_rank)),
                        ("near_field", lambda: bench_nearfield(M, local_rank, with_cpu=not args.no_cpu)),
                        ("shg", lambda: bench_shg(M, local_rank, with_cpu=not args.no_cpu))):
            try:
                line[key] = fn()
            except Exception as exc:  # a side measurement must not cost the bench line
                line[key] = {"error": repr(exc)[:300]}
    if rank == 0 and world == 1 and not args.no_cpu:
        cores = host_cores()
        info = cpu_sample(args.subdiv, cores)
        line["cpu_baseline"] = dict({"value": 1.0 / info.pop("total_s"), "unit": "solves/s", "cores": cores,
                                     "kind": "port"}, **info)
    line["autotune_panel"] = {"mixed": tune_or_none(M, S, M.MIXED),
                              "fp64": tune_or_none(M, S, M.FP64) if ms_fp64 else None}
    line["rooflines"] = roofs
    line["phases"] = phases
    line["lu_overlap"] = lu_overlap
    line["phases_fp64"] = phases64
    line["refine_iters"] = iters
    # the FP64 comparison last, where a truncated record still keeps it
    line["sigma_ext"] = {"mixed": ext_mixed, "fp64": ext_fp64, "oracle_fp64": ref_ext,
                         "mixed_vs_oracle": rel(ext_mixed, ref_ext), "fp64_vs_oracle": rel(ext_fp64, ref_ext),
                         "mixed_vs_fp64": rel(ext_mixed, ext_fp64)}
    line["fp64"] = ({"value": world * 1000.0 / ms_fp64, "unit": "solves/s", "ms_per_step": ms_fp64}
                    if ms_fp64 else None)
    line["mixed_over_fp64"] = (ms_fp64 / ms_mixed) if ms_fp64 else None
    if rank == 0:
        print(json.dumps(line), flush=True)
    S.close()
    if world > 1:
        torch.distributed.destroy_process_group()
    return 0


def bench_nearfield(M, dev, n=101, with_cpu=True):
    """Near fields (scat_fields + incident, the nfpl plane) of the cfg1 sphere
    (s=3, FP64 solution at 600 nm): an n x n grid 200 nm wide in the xz plane
    through the particle, exterior domain.  GPU time per plane through the C ABI
    (host points in, host fields out); with with_cpu, the CPU baseline of this
    row: the oracle on a sample of points on one host core, and the largest
    relative difference on that sample."""
    import numpy as np
    from mom_b200 import workloads as W
    nodes, faces, ids, doms = W.sphere(3)
    S = M.Solver(dev)
    S.set_problem(M.Problem.from_arrays(nodes, faces, ids, 1e-9, doms))
    om = M.omega_of(WL)
    src = [M.src_pw(0, 90, 0)]
    x = S.solve_wavelength(om, [1.0, np.sqrt(EPS_IN)], src, M.FP64, 1e-12, 30)
    a, b = np.meshgrid(np.linspace(-100e-9, 100e-9, n), np.linspace(-100e-9, 100e-9, n), indexing="ij")
    pts = np.stack([a.ravel(), np.zeros(n * n), b.ravel()], axis=1)
    S.scat_fields(om, 1.0, pts, x=x, srcs=src, dom=0)  # warm-up
    reps = 3
    t0 = time.perf_counter()
    for _ in range(reps):
        e, h = S.scat_fields(om, 1.0, pts, x=x, srcs=src, dom=0)
    gpu_s = (time.perf_counter() - t0) / reps
    S.close()
    F = len(faces)
    flop = 1300.0 * n * n * F  # ~13 x 70 FLOP of quadrature + ~400 of contraction per point-face pair
    out = {"workload": "nfpl plane %d x %d points (200 nm, xz) on the s=3 sphere, exterior domain, + incident" % (n, n),
           "gpu_ms_per_plane": gpu_s * 1e3, "points_per_s": n * n / gpu_s,
           "point_face_pairs_per_s": n * n * F / gpu_s,
           "fp64_tflops_est": flop / gpu_s / 1e12,
           "fp64_peak_note": "nominal FP64 SIMT 148 SM x 64 FMA x 2 x 1.965 GHz = 37 TFLOP/s; FLOP per pair estimated"}
    if with_cpu:
        sys.path.insert(0, os.path.join(ROOT, "oracle"))
        import oracle as O
        P = O.OracleProblem(nodes, faces, ids, 1e-9, doms)
        idx = np.linspace(0, n * n - 1, 16).astype(int)
        t0 = time.perf_counter()
        eo, ho = P.scat_fields(om, 1.0, x, pts[idx], srcs=src, d=0)
        cpu_s = time.perf_counter() - t0
        err = max(float(np.abs(e[0, idx] - eo[0]).max() / np.abs(eo[0]).max()),
                  float(np.abs(h[0, idx] - ho[0]).max() / np.abs(ho[0]).max()))
        out["cpu_baseline"] = {"value": len(idx) / cpu_s, "unit": "points/s", "cores": 1, "kind": "port",
                               "sample": "16 of the plane's points"}
        out["max_rel_diff_vs_oracle"] = err
    return out


def bench_shg(M, dev, with_cpu=True):
    """Second-harmonic generation (solver.f90:143-217) from a surface
    nonlinearity of the particle (chi_nnn, chi_ntt, chi_ttn = 1, 0.5, 0.2 x
    1e-18 m^2/V) on the s=4 sphere (15,360 unknowns) at 1000 nm, SH index
    sqrt(-2 + 3.5i): time of the SH solve (source expansion + assembly at
    2 omega + LU + solve) after the fundamental solve, FP64 and mixed, and the
    SH sigma_sca.  With with_cpu, the oracle's restatement on the s=2 sphere
    (1,920 unknowns, one host thread for the expansion, OpenMP assembly) against
    the GPU on the same s=2 problem: time and the largest relative difference
    of the SH solution."""
    import numpy as np
    from mom_b200 import workloads as W
    wl = 1000e-9
    om = M.omega_of(wl)
    ri = [1.0, np.sqrt(EPS_IN)]
    shri = [1.0, np.sqrt(complex(-2.0, 3.5))]
    chi = (1.0e-18, 0.5e-18, 0.2e-18)
    src = [M.src_pw(0, 90, 0)]
    out = {"workload": "icosphere s=4 (15360 unknowns), nlsurf chi (1, 0.5, 0.2)e-18 in the particle, 1000 nm, "
                       "SH index sqrt(-2+3.5i), x-pol pw +z"}
    S = M.Solver(dev)
    nodes, faces, ids, doms = W.sphere(4)
    S.set_problem(M.Problem.from_arrays(nodes, faces, ids, 1e-9, doms))
    for name, prec in (("fp64", M.FP64), ("mixed", M.MIXED)):
        times = []
        for rep in range(3):
            S.solve_wavelength(om, ri, src, prec, 1e-12, 30, want_host=False)
            S.synchronize()
            t0 = time.perf_counter()
            S.shg_solve(om, ri, shri, [None, chi], prec, 1e-12, 30, want_host=False)
            S.synchronize()
            times.append(time.perf_counter() - t0)
        csca, _ = S.cross_sections(2 * om, 1.0, [M.src_none()])
        out[name] = {"shg_solve_ms": min(times[1:]) * 1e3, "sigma_sca_sh": float(csca[0]),
                     "refine_iters": S.iters}
    out["mixed_vs_fp64_sigma_sh"] = abs(out["mixed"]["sigma_sca_sh"] / out["fp64"]["sigma_sca_sh"] - 1)
    if with_cpu:
        sys.path.insert(0, os.path.join(ROOT, "oracle"))
        import oracle as O
        nodes, faces, ids, doms = W.sphere(2)
        S.set_problem(M.Problem.from_arrays(nodes, faces, ids, 1e-9, doms))
        S.solve_wavelength(om, ri, src, M.FP64, want_host=False)
        S.synchronize()
        t0 = time.perf_counter()
        nlx = S.shg_solve(om, ri, shri, [None, chi], M.FP64)
        gpu_s = time.perf_counter() - t0
        P = O.OracleProblem(nodes, faces, ids, 1e-9, doms)
        osrc = dict(type="pw", theta=0.0, phi=90 * O.DEGTORAD, psi=0.0)
        x = O.solve(P.sysmat(om, ri), P.srcvec(om, 1.0, osrc)[:, None])
        t0 = time.perf_counter()
        nlo = O.shg_solve(P, om, ri, shri, [None, chi], x)
        cpu_s = time.perf_counter() - t0
        out["s2"] = {"gpu_shg_solve_ms": gpu_s * 1e3,
                     "max_rel_diff_vs_oracle": float(np.linalg.norm(nlx[:, 0] - nlo[:, 0]) / np.linalg.norm(nlo[:, 0]))}
        out["cpu_baseline"] = {"value": 1.0 / cpu_s, "unit": "SH solves/s", "kind": "port",
                               "cores": host_cores(), "sample": "the s=2 sphere (1920 unknowns), whole SH solve"}
    S.close()
    return out


def bench_sweep(M, workers, dev):
    """Uneven wavelength sweep: the s=3 sphere and three seeded ellipsoids, 64 wavelengths
    on 400-900 nm with a Drude permittivity, mixed precision refined to 1e-12; every mesh's
    wavelengths split over `workers` contexts that run concurrently (mom_gpu_sweep_many)."""
    import numpy as np
    from mom_b200 import workloads as W
    meshes = W.sweep_meshes()
    wls = W.sweep_wavelengths(64)
    oms = np.array([M.omega_of(w) for w in wls])
    ri = np.stack([np.ones(len(wls)), np.sqrt(W.drude_eps(wls))], axis=1)
    src = [M.src_pw(0, 90, 0)]
    solvers, parts = [], []
    for _, (nodes, faces, ids, doms) in meshes:
        prob = M.Problem.from_arrays(nodes, faces, ids, 1e-9, doms)
        for w in range(workers):
            s = M.Solver(dev)
            s.set_problem(prob)
            solvers.append(s)
            parts.append(np.arange(w, len(wls), workers))
    out = {"workload": "sweep: sphere s=3 + 3 ellipsoids (%s unknowns), 64 wavelengths 400-900 nm, Drude eps"
                       % "/".join(str(2 * solvers[i * workers].N) for i in range(len(meshes))),
           "contexts": len(solvers)}
    for prec, name in ((M.MIXED, "mixed"), (M.FP64, "fp64")):
        # warm-up: autotuning and graph capture of every context
        M.sweep_many(solvers, [oms[p[:1]] for p in parts], [ri[p[:1]] for p in parts], src, prec)
        t0 = time.perf_counter()
        res = M.sweep_many(solvers, [oms[p] for p in parts], [ri[p] for p in parts], src, prec)
        dt = time.perf_counter() - t0
        out[name] = {"solves_per_s": len(meshes) * len(wls) / dt, "seconds": dt,
                     "panel_ctas_by_height": [
                         (lambda t: dict(zip(t["heights"], t["ctas"])) if t else None)(
                             tune_or_none(M, solvers[i * workers], prec)) for i in range(len(meshes))]}
        out[name + "_sigma_ext_first"] = float(res[0][0][0, 0] + res[0][1][0, 0])
    for s in solvers:
        s.close()
    return out


def tune_or_none(M, S, prec):
    """The LU autotuner's table, or None when tuning is off (MOM_AUTOTUNE=0 / MOM_PANEL_CTAS)."""
    try:
        return S.autotune_result(prec)
    except M.MomError:
        return None


def bench_core_shell(M, dev, nsrc=512):
    """Core-shell (30,720 unknowns, 3 domains) with 512 incidences: one factorisation reused
    for all right-hand sides (GEMM-based blocked solves, FP64 ZGEMM residuals), cross
    sections, and d(mean sigma_ext, sigma_abs)/d(shell eps) by the adjoint; mixed and FP64."""
    import numpy as np
    from mom_b200 import workloads as W
    nodes, faces, ids, doms = W.core_shell(4)
    srcs = W.incidences(nsrc)
    S = M.Solver(dev)
    S.set_problem(M.Problem.from_arrays(nodes, faces, ids, 1e-9, doms))
    om = M.omega_of(WL)
    ri = [1.0, np.sqrt(W.EPS_AU), np.sqrt(W.EPS_SILICA)]
    out = {"workload": "core-shell s=4 (r 40/60 nm, %d unknowns), %d pw_elliptic incidences" % (2 * S.N, nsrc)}
    ext = {}
    for prec, name in ((M.MIXED, "mixed"), (M.FP64, "fp64")):
        # untimed: autotune + graph capture, and the workspaces of 512 right-hand
        # sides and of the adjoint (allocated on first use)
        S.solve_wavelength(om, ri, srcs, prec, TOL, MAXIT, want_host=False)
        S.adjoint_mean_eps(om, ri, srcs, prec, eps_dom=1, tol=TOL, maxit=MAXIT)
        S.synchronize()
        t0 = time.perf_counter()
        S.solve_wavelength(om, ri, srcs, prec, TOL, MAXIT, want_host=False)
        a, b = S.cross_sections(om, ri[0], srcs)
        t1 = time.perf_counter()
        g = S.adjoint_mean_eps(om, ri, srcs, prec, eps_dom=1, tol=TOL, maxit=MAXIT)
        t2 = time.perf_counter()
        ext[name] = a + b
        out[name] = {"solve_s": t1 - t0, "rhs_per_s": nsrc / (t1 - t0), "adjoint_mean_eps_s": t2 - t1,
                     "refine_iters": S.iters, "dmean_ext_deps": [g[0, 0], g[0, 1]]}
    out["sigma_ext_max_rel_mixed_vs_fp64"] = float(np.max(np.abs(ext["mixed"] - ext["fp64"]) / np.abs(ext["fp64"])))
    S.close()
    return out


def bench_adjoint(M, dev):
    """Adjoint gradients on the perturbed s=3 sphere (3840 unknowns, 642 vertices):
    time of d sigma / d eps and of d sigma / d(all vertex coordinates), and the eps
    gradient against central differences (step 1e-6) of the FP64 cross sections."""
    import numpy as np
    from mom_b200 import workloads as W
    nodes, faces, ids, doms = W.perturbed(3)
    S = M.Solver(dev)
    S.set_problem(M.Problem.from_arrays(nodes, faces, ids, 1e-9, doms))
    om = M.omega_of(WL)
    src = [M.src_pw(0, 90, 0)]

    def sig(eps, prec=M.FP64):
        ri = [1.0, np.sqrt(eps)]
        S.solve_wavelength(om, ri, src, prec, 1e-12, 30)
        a, b = S.cross_sections(om, ri[0], src)
        return np.array([a[0] + b[0], b[0]])

    out = {"workload": "perturbed sphere s=3 (3840 unknowns, %d vertices)" % len(nodes)}
    fd = []
    for dz in (1e-6, 1e-6j):
        fd.append((sig(EPS_IN + dz) - sig(EPS_IN - dz)) / 2e-6)
    fd = np.array(fd)
    for prec, name in ((M.FP64, "fp64"), (M.MIXED, "mixed")):
        ri = [1.0, np.sqrt(EPS_IN)]
        sig(EPS_IN, prec)
        S.adjoint(om, ri, src, prec, eps_dom=1)  # untimed: first-call set-up
        t0 = time.perf_counter()
        g = S.adjoint(om, ri, src, prec, eps_dom=1)["deps"][0]
        t1 = time.perf_counter()
        sig(EPS_IN, prec)
        t2 = time.perf_counter()
        S.adjoint(om, ri, src, prec, nodes=True)
        t3 = time.perf_counter()
        out[name] = {"eps_grad_ms": (t1 - t0) * 1e3, "vertex_grad_ms": (t3 - t2) * 1e3,
                     "eps_grad_vs_fd_max_rel": float(np.max(np.abs(g.T - fd) / np.abs(fd)))}
    # vertex gradients against central differences (1e-4 nm) of the FP64 cross
    # sections on 24 seeded (vertex, axis) pairs; entries with |FD| > 1e-3 max
    prob = M.Problem.from_arrays(nodes, faces, ids, 1e-9, doms)
    ri = [1.0, np.sqrt(EPS_IN)]
    grads = {}
    for prec, name in ((M.FP64, "fp64"), (M.MIXED, "mixed")):
        sig(EPS_IN, prec)
        dn = S.adjoint(om, ri, src, prec, nodes=True)["dnodes"]
        gv = np.zeros((2, len(nodes), 3))
        for d, gd in enumerate(dn):
            np.add.at(gv, (slice(None), prob.node_parent(d)), gd[0] * 1e-9)
        grads[name] = gv
    rng = np.random.default_rng(11)
    picks = list(zip(rng.choice(len(nodes), 24, replace=False), rng.integers(0, 3, 24)))
    h = 1e-4
    fdv = []
    for v, k in picks:
        sv = []
        for sgn in (1.0, -1.0):
            nd = nodes.copy()
            nd[v, k] += sgn * h
            S.set_problem(M.Problem.from_arrays(nd, faces, ids, 1e-9, doms))
            sv.append(sig(EPS_IN))
        fdv.append((sv[0] - sv[1]) / (2 * h))
    for name, gv in grads.items():
        gmax = np.abs(gv).max(axis=(1, 2))
        sel = [(o, v, k, f[o]) for (v, k), f in zip(picks, fdv) for o in range(2) if abs(f[o]) > 1e-3 * gmax[o]]
        errs = [abs(gv[o, v, k] - fo) / abs(fo) for o, v, k, fo in sel]
        errm = [abs(gv[o, v, k] - fo) / gmax[o] for o, v, k, fo in sel]
        out[name]["vertex_grad_vs_fd_max_rel"] = float(max(errs)) if errs else None
        out[name]["vertex_grad_vs_fd_max_over_largest_entry"] = float(max(errm)) if errm else None
        out[name]["vertex_grad_vs_fd_entries"] = len(errs)
    S.close()
    return out


def run_kernel_cases(subdiv):
    """One pass over the kernels outside the LU on the icosphere of `subdiv`
    (default 3: 1280 faces, 3840 unknowns; the matrix and the face-pair
    buffer exceed L2), for per-kernel profiling captures: FP64 assembly
    (pair_kernel<double>, near_kernel, gather_kernel), srcvec, cs_prtsrf,
    the 91 x 180 far field, a 41 x 41 near-field plane, the FP64 eps adjoint
    (adj_pair_kernel), then the mixed solve (pair_kernel<float>, the FP64
    refinement residual gemv_partial_kernel) and an FP64 second-harmonic solve
    with a surface nonlinearity of the particle (nls_face_kernel,
    gram_cg_kernel, nls_cm_kernel)."""
    import numpy as np
    import mom_b200 as M
    nodes, faces, ids, doms = make_problem(M, subdiv)
    S = M.Solver(0)
    S.set_problem(M.Problem.from_arrays(nodes, faces, ids, 1e-9, doms))
    om = M.omega_of(WL)
    ri = [1.0, np.sqrt(EPS_IN)]
    src = [M.src_pw(0, 90, 0)]
    S.solve_wavelength(om, ri, src, M.FP64, want_host=False)
    a, b = S.cross_sections(om, ri[0], src)
    S.rcs(om, ri[0], 91, 180)
    g = np.linspace(-100e-9, 100e-9, 41)
    pts = np.stack(np.meshgrid(g, [0.0], g, indexing="ij"), axis=-1).reshape(-1, 3)
    S.scat_fields(om, 1.0, pts, srcs=src, dom=0)
    S.adjoint(om, ri, src, M.FP64, eps_dom=1)
    S.solve_wavelength(om, ri, src, M.MIXED, TOL, MAXIT, want_host=False)
    S.solve_wavelength(om, ri, src, M.FP64, want_host=False)
    S.shg_solve(om, ri, [1.0, np.sqrt(complex(-2.0, 3.5))], [None, (1.0e-18, 0.5e-18, 0.2e-18)], M.FP64,
                want_host=False)
    S.synchronize()
    S.close()
    print(json.dumps({"kernel_cases": workload_name(subdiv), "sigma_ext_fp64": float(a[0] + b[0])}), flush=True)
    return 0


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--fp64-steps", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--subdiv", type=int, default=SUBDIV)
    ap.add_argument("--no-cpu", action="store_true", help="skip the CPU baseline sample")
    ap.add_argument("--no-e2e", action="store_true", help="skip the end-to-end (host buffer) measurement")
    ap.add_argument("--no-extras", action="store_true", help="skip the sweep and adjoint side measurements")
    ap.add_argument("--sweep-workers", type=int, default=6, help="concurrent contexts per sweep mesh")
    ap.add_argument("--kernels", action="store_true",
                    help="run the non-LU kernels once on the --subdiv sphere (for profiling captures), no timing")
    args = ap.parse_args()
    rank, local_rank, world = dist_env()
    if args.kernels:
        return run_kernel_cases(args.subdiv)
    if args.impl == "reference":
        return run_reference(args, rank, world)
    return run_ours(args, rank, local_rank, world)


if __name__ == "__main__":
    sys.exit(main())
