"""Benchmark of the Ryser / Gray-code permanent hot path on B200.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
                    [--workload dense32|dense24|complex28|binary36|sparse40|batch20|approx100|serve|...]

A step is one permanent of the workload matrix (the headline: dense real FP64
n=32, entries U[0,1) from SplitMix64 seed 7).  The metric is Gray steps per
second, n*2^(n-1) per permanent (the reference's own unit of work, the NW
Gray walk of Algorithms/CPU/Dense/dpNaivePerman.h:116-133), summed over all
ranks.  Multi-GPU runs are independent replicas (the path has no data
exchange; one process per GPU, max-over-ranks device time).

Printed JSON line (rank 0):
  value      device-resident input, CUDA-event time per step on the launch stream
  e2e        same metric through the C ABI with a pinned host matrix, timed by
             the host clock around each call: H2D copy, kernels, D2H of the
             result and the call's host work inside the timed region
  roofline   dominant kernel (the Gray walk): FP64 pipe instructions per
             launch / walk-kernel time, against the FP64 FMA pipe peak measured
             by a DFMA microbenchmark in the same run
  cpu_baseline  the reference's CPU Ryser (oracle/_ref) on this host's cores
"""
from __future__ import annotations

import argparse
import ctypes
import json
import math
import os
import statistics
import subprocess
import sys
import tempfile
import threading
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

WORKLOADS = {
    # name: (kind, n, seed, description)
    "dense32": ("dense", 32, 7, "dense_f64_u01_n32_seed7"),
    "dense24": ("dense", 24, 3, "dense_f64_u01_n24_seed3"),
    "dense28": ("dense", 28, 28, "dense_f64_u01_n28_seed28"),
    "complex28": ("complex", 28, 6, "complex128_haar256_block_n28_seed6"),
    "binary36": ("binary", 36, 4, "binary_bernoulli0.5_or_identity_n36_seed4"),
    "binary28": ("binary", 28, 4, "binary_bernoulli0.5_or_identity_n28_seed4"),
    "batch20": ("batch", 20, 11, "batch_4096_dense_u01_n20_seed11"),
    "sparse40": ("sparse", 40, 5, "sparse_perm_plus3_u0.5-1.5_n40_seed5"),
    # sampling permanent (the reference's algorithm=approximation) beyond n=63
    "approx100": ("approx", 100, 5, "sampling_pattern_perm_plus3_n100_seed5_4Msamples"),
}

# DRAM bytes (read + write) per walk_real<32> launch, the mean of two launches in
# one ncu capture of this workload (dram__bytes_read.sum + dram__bytes_write.sum).
NCU_TRAFFIC = {"dense32": 435584}


def env_int(name, default):
    try:
        return int(os.environ.get(name, default))
    except ValueError:
        return default


# ----------------------------------------------------------------- clocks --
class ClockSampler:
    """Samples SM clock and throttle reasons through NVML while running."""

    REASONS = {
        0x1: "gpu_idle", 0x2: "applications_clocks_setting", 0x4: "sw_power_cap",
        0x8: "hw_slowdown", 0x10: "sync_boost", 0x20: "sw_thermal_slowdown",
        0x40: "hw_thermal_slowdown", 0x80: "hw_power_brake_slowdown",
        0x100: "display_clock_setting",
    }

    def __init__(self, device: int, period_s: float = 0.005):
        self.device, self.period = device, period_s
        self.samples, self.reasons = [], 0
        self._stop = threading.Event()
        self._thread = None
        self.max_mhz = None
        try:
            import pynvml
            pynvml.nvmlInit()
            self._nv = pynvml
            self._h = pynvml.nvmlDeviceGetHandleByIndex(device)
            self.max_mhz = pynvml.nvmlDeviceGetMaxClockInfo(self._h, pynvml.NVML_CLOCK_SM)
        except Exception:  # no NVML: report no clocks rather than fail
            self._nv = None

    def _run(self):
        nv = self._nv
        while not self._stop.is_set():
            try:
                self.samples.append(nv.nvmlDeviceGetClockInfo(self._h, nv.NVML_CLOCK_SM))
                self.reasons |= nv.nvmlDeviceGetCurrentClocksEventReasons(self._h)
            except Exception:
                pass
            time.sleep(self.period)

    def __enter__(self):
        if self._nv is not None:
            self._thread = threading.Thread(target=self._run, daemon=True)
            self._thread.start()
        return self

    def __exit__(self, *exc):
        self._stop.set()
        if self._thread:
            self._thread.join()

    def summary(self):
        if self._nv is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvml unavailable"]}
        names = [v for k, v in self.REASONS.items() if self.reasons & k and v != "gpu_idle"]
        return {"sm_mhz": statistics.median(self.samples) if self.samples else None,
                "sm_max_mhz": self.max_mhz, "reasons": names, "samples": len(self.samples)}


# ----------------------------------------------------- reference (CPU) arm --
def write_mtx(path, a):
    import numpy as np
    n = a.shape[0]
    lines = []
    cplx = np.iscomplexobj(a)
    for i in range(n):
        for j in range(n):
            v = a[i, j]
            if v == 0:
                continue
            if cplx:
                lines.append(f"{i + 1} {j + 1} {float(v.real)!r} {float(v.imag)!r}")
            else:
                lines.append(f"{i + 1} {j + 1} {float(v)!r}")
    with open(path, "w") as f:
        f.write(f"{n} {n} {len(lines)}\n" + "\n".join(lines) + "\n")


def reference_step(a, threads, complex_=False, timeout=1800):
    """One run of the reference CPU binary; returns its own reported seconds."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle as O
    with tempfile.TemporaryDirectory() as d:
        p = os.path.join(d, "m.mtx")
        write_mtx(p, a)
        extra = ["complex=true"] if complex_ else []
        _, secs = O.run_reference(p, threads=threads, extra=extra, timeout=timeout)
    return secs


def port_step(a, threads, complex_=False):
    """Fallback when the reference binary is absent: the oracle's restatement."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle as O
    t0 = time.perf_counter()
    if complex_:
        O.complex_nw(a, threads=threads)
    else:
        O.dense_nw(a, threads=threads)
    return time.perf_counter() - t0


def cpu_sample(kind, n, seed, cores):
    """Bounded CPU sample of the workload: the same generator at the largest
    n' <= n whose estimated reference time is <= ~20 s on `cores` threads
    (dense: ~1e10 Gray steps/s on 8 cores, scaling with cores)."""
    rate = 1.2e9 * cores * (0.3 if kind == "complex" else 1.0)
    m = n
    while m > 12 and m * 2 ** (m - 1) / rate > 20.0:
        m -= 1
    return m


def make_matrix(kind, n, seed):
    from superman_b200 import workloads as W
    if kind == "dense":
        return W.dense_uniform(n, seed)
    if kind == "complex":
        return W.haar_block(n, seed)
    raise ValueError(kind)


def run_cpu_baseline(kind, n, seed, steps=1):
    ref_bin = os.path.join(ROOT, "oracle", "_ref", "superman_ref")
    cores = os.cpu_count() or 1
    m = cpu_sample(kind, n, seed, cores)
    a = make_matrix(kind, m, seed)
    use_ref = os.path.exists(ref_bin)
    times = []
    for _ in range(steps):
        times.append(reference_step(a, cores, kind == "complex") if use_ref
                     else port_step(a, cores, kind == "complex"))
    t = statistics.mean(times)
    return {"value": m * 2 ** (m - 1) / t, "unit": "gray-steps/s", "cores": cores,
            "kind": "reference" if use_ref else "port",
            "sample": f"one full permanent of the same generator at n={m} "
                      f"({'reference CPU binary oracle/_ref, mode=cpu' if use_ref else 'oracle port'}, "
                      f"thread_count={cores}); mean of {steps} run(s), {t:.3f} s each"}, times


def unavailable_line(why):
    print(json.dumps({"impl": "reference", "unavailable": why}), flush=True)
    return 0


def reference_other(args, kind, n, seed, desc):
    """Reference arm for the sparse-pipeline and 0/1 workloads: the reference's
    CPU program on the same input (0/1: binary=true, its FP64 path), on all host
    cores; the 0/1 size is bounded like the dense CPU sample."""
    import numpy as np
    from superman_b200 import workloads as W
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle as O
    cores = os.cpu_count() or 1
    if not os.path.exists(O.ref_binary_path()):
        return unavailable_line("the reference CPU program (oracle/_ref) is not built")
    with tempfile.TemporaryDirectory() as d:
        p = os.path.join(d, "m.mtx")
        if kind == "sparse":
            a = W.sparse_perm_plus(n, seed)
            write_mtx(p, a)
            extra, m = [], n
        else:
            m = cpu_sample("dense", n, seed, cores)
            a = W.binary_bernoulli(m, seed)
            with open(p, "w") as f:  # binary=true reads "i j" lines
                ij = np.argwhere(a != 0)
                f.write(f"{m} {m} {len(ij)}\n" + "".join(f"{i + 1} {j + 1}\n" for i, j in ij))
            extra = ["binary=true"]
        for _ in range(args.warmup):
            O.run_reference(p, threads=cores, extra=extra, timeout=1800)
        times = [O.run_reference(p, threads=cores, extra=extra, timeout=1800)[1] for _ in range(args.steps)]
    t = statistics.mean(times)
    if kind == "sparse":
        metric, value, unit = "sparse_pipeline_perms_per_s", 1.0 / t, "perms/s"
        sample = f"reference CPU program on the n={n} matrix (its decomposition and sparse Ryser)"
    else:
        metric, value, unit = "ryser_gray_steps_per_s", m * 2 ** (m - 1) / t, "gray-steps/s (NW, n*2^(n-1))"
        sample = f"reference CPU program, binary=true, on the same generator at n={m}"
    cb = {"value": value, "unit": unit, "cores": cores, "kind": "reference",
          "sample": f"{sample}; mean of {args.steps} run(s), {t:.3f} s each"}
    line = {"metric": metric, "value": value, "unit": unit, "n_gpus": args.gpus, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": t * 1e3, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": {"workload": desc, "kind": kind, "n": n, "seed": seed}, "impl": "reference",
            "cpu_baseline": cb, "e2e": {"value": value, "unit": unit, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)
    return 0


def reference_arm(args, wl):
    rank = env_int("RANK", 0)
    if rank != 0:
        return 0
    if wl in SERVE_WORKLOADS:
        return unavailable_line("the reference has no serving loop: it computes one matrix per process run")
    kind, n, seed, desc = WORKLOADS[wl]
    if kind == "batch":
        return unavailable_line("the reference has no batched entry point: one matrix per process run")
    if kind == "approx":
        return unavailable_line("the reference's approximation (aspSingleGPU) exists only in its GPU build; "
                                "this arm times the reference's CPU program, which has no approximation")
    if kind in ("sparse", "binary"):
        return reference_other(args, kind, n, seed, desc)
    for _ in range(args.warmup):
        run_cpu_baseline(kind, n, seed, steps=1)
    cb, times = run_cpu_baseline(kind, n, seed, steps=args.steps)
    t = statistics.mean(times)
    line = {"metric": "ryser_gray_steps_per_s", "value": cb["value"], "unit": "gray-steps/s",
            "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": t * 1e3, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": {"workload": desc, "kind": kind, "n": n, "seed": seed},
            "impl": "reference", "cpu_baseline": cb,
            "e2e": {"value": cb["value"], "unit": "gray-steps/s",
                    "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)
    return 0


def reference_gpu_arm(args, wl):
    """The reference's own GPU program (oracle/_ref/superman_ref_gpu, built from
    its sources by `make -C oracle ref_gpu`) on the same matrix, mode=single_gpu:
    its dpSingleGPU driver with xRegisterMSharedKahan (dense real) or
    gpuComputeComplex with xRegisterMSharedComplex (complex), timed by its own
    "Computed in" clock.  A second reference column beside the CPU arm; rank 0
    only."""
    rank = env_int("RANK", 0)
    if rank != 0:
        return 0
    binp = os.path.join(ROOT, "oracle", "_ref", "superman_ref_gpu")
    if not os.path.exists(binp):
        print(json.dumps({"impl": "reference_gpu", "unavailable": "oracle/_ref/superman_ref_gpu is not built "
                                                                   "(make -C oracle ref_gpu)"}), flush=True)
        return 0
    if wl not in WORKLOADS or WORKLOADS[wl][0] not in ("dense", "complex"):
        print(json.dumps({"impl": "reference_gpu", "unavailable": f"workload {wl}: timed for the dense and complex "
                                                                   "workloads only"}), flush=True)
        return 0
    import re
    kind, n, seed, desc = WORKLOADS[wl]
    a = make_matrix(kind, n, seed)

    def run_once():
        with tempfile.TemporaryDirectory() as d:
            p = os.path.join(d, "m.mtx")
            write_mtx(p, a)
            os.makedirs(os.path.join(d, "build"), exist_ok=True)
            argv = [binp, "pid=2", f"repo_dir={d}/", f"filename={p}", "mode=single_gpu", "device_id=0"]
            if kind == "complex":
                argv.append("complex=true")
            out = subprocess.run(argv, check=True, capture_output=True, text=True, timeout=1800).stdout
        m = re.search(r"Permanent: \(?([^ ,)]+),?([^ )]*)\)? - Computed in: (\S+) seconds", out)
        if m is None:
            raise RuntimeError("unexpected reference output: " + out[-400:])
        v = complex(float(m.group(1)), float(m.group(2))) if m.group(2) else float(m.group(1))
        return v, float(m.group(3))

    for _ in range(args.warmup):
        run_once()
    runs = [run_once() for _ in range(args.steps)]
    t = statistics.median(x[1] for x in runs)
    value = n * 2 ** (n - 1) / t
    line = {"metric": "ryser_gray_steps_per_s", "value": value, "unit": "gray-steps/s", "n_gpus": 1,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": t * 1e3, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": {"workload": desc, "kind": kind, "n": n, "seed": seed,
                       "permanent": repr(runs[0][0]),
                       "timing": "the reference program's own 'Computed in' clock (host wall time of its "
                                 "driver: allocations, copies, chunked kernel launches, host reduction)"},
            "impl": "reference_gpu",
            "kernel": "xRegisterMSharedComplex" if kind == "complex" else "xRegisterMSharedKahan"}
    print(json.dumps(line), flush=True)
    return 0


# ------------------------------------------------------------- our GPU arm --
def max_over_ranks(values, dist, device):
    """Element-wise maximum of per-rank timings over the process group (the
    replicas' job takes as long as its slowest rank); identity on one rank."""
    if dist is None:
        return list(values)
    import torch
    t = torch.tensor(list(values), device=device, dtype=torch.float64)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return [float(x) for x in t.tolist()]


def ours_arm(args, wl):
    import numpy as np
    import torch
    import superman_b200 as S
    from superman_b200 import _lib

    kind, n, seed, desc = WORKLOADS[wl]
    world = env_int("WORLD_SIZE", 1)
    rank = env_int("RANK", 0)
    local = env_int("LOCAL_RANK", 0)
    dist = None
    if world > 1:
        import datetime
        import torch.distributed as dist
        torch.cuda.set_device(local)
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=300),
                                device_id=torch.device("cuda", local))
    device = local
    torch.cuda.set_device(device)
    L = _lib.lib()

    a = make_matrix(kind, n, seed)
    comps = 2 if kind == "complex" else 1
    host = torch.from_numpy(np.ascontiguousarray(a).view(np.float64).copy()).pin_memory()
    dev_a = host.to(f"cuda:{device}")
    flush = torch.empty(256 * 1024 * 1024, dtype=torch.uint8, device=f"cuda:{device}")
    # The library runs on its own stream and times each call with CUDA events
    # recorded on that stream (spb_result.device_s / kernel_s).
    opt = _lib.default_options(device=device, precision=_lib.SPB_PREC_DD if args.precision == "dd"
                               else _lib.SPB_PREC_FP64)
    res = _lib.spb_result()
    fn_dev = L.spb_perm_dense_c128_dev if comps == 2 else L.spb_perm_dense_f64_dev
    fn_host = L.spb_perm_dense_c128 if comps == 2 else L.spb_perm_dense_f64
    host_ptr = ctypes.cast(ctypes.c_void_p(host.data_ptr()), ctypes.POINTER(ctypes.c_double))

    peak = ctypes.c_double()
    _lib.check(L.spb_measure_pipe_peak(device, 0, ctypes.byref(peak)))

    def step_dev():
        _lib.check(fn_dev(ctypes.c_void_p(dev_a.data_ptr()), n, ctypes.byref(opt), ctypes.byref(res)))
        return res.device_s, res.kernel_s, res.launches

    # The e2e arm times the call itself on the host, so it asks the library
    # not to time its device work as well (spb_options.skip_timing).
    opt_e2e = _lib.default_options(device=device, precision=opt.precision, skip_timing=1)

    def step_host():
        # host wall clock around the public C-ABI call on the pinned host
        # matrix: H2D copy, kernels, D2H of the result and the call's own
        # host work (the call returns after its stream synchronize)
        t0 = time.perf_counter()
        _lib.check(fn_host(host_ptr, n, ctypes.byref(opt_e2e), ctypes.byref(res)))
        return time.perf_counter() - t0, res.kernel_s, res.launches

    def timed(step):
        for _ in range(args.warmup):
            flush.zero_()
            torch.cuda.synchronize()
            step()
        if dist:
            dist.barrier()
        torch.cuda.synchronize()
        total_ms, walk_s, launches = 0.0, 0.0, 0
        for _ in range(args.steps):
            flush.zero_()  # evict L2 between steps (outside the step's events)
            torch.cuda.synchronize()
            ds, ks, nl = step()  # returns after its own stream synchronize
            total_ms += ds * 1e3
            walk_s += ks
            launches += nl
        torch.cuda.synchronize()
        if dist:
            dist.barrier()
        total_ms, walk_s = max_over_ranks([total_ms, walk_s], dist, f"cuda:{device}")
        return total_ms / args.steps, walk_s / args.steps, launches

    with ClockSampler(device) as clk:
        ms_dev, walk_dev, launches = timed(step_dev)
    value_dev = float(res.value) + 1j * float(res.imag) if comps == 2 else float(res.value)
    ms_e2e, _, _ = timed(step_host)

    steps_per_perm = n * 2 ** (n - 1)
    value = world * steps_per_perm / (ms_dev * 1e-3)
    e2e = world * steps_per_perm / (ms_e2e * 1e-3)
    alg = walk_work(n, comps == 2)  # FP64 pipe instructions per walk launch
    achieved = alg / walk_dev
    roofline = {"bound": "fp64", "achieved": achieved / 1e12, "peak": peak.value / 1e12,
                "unit": "T FP64-pipe inst/s", "frac": achieved / peak.value,
                "traffic": NCU_TRAFFIC.get(wl),
                "peak_source": "DFMA microbenchmark in this run (spb_measure_pipe_peak); "
                               "MEASURED_PEAKS.json has no FP64 figure",
                "algorithmic_per_launch": alg}

    golden_name = {"dense32": "dense_u01_n32_s7", "dense24": "dense_u01_n24_s3",
                   "complex28": "complex_haar_n28_s6"}.get(wl)
    golden = os.path.join(ROOT, "tests", "golden", f"{golden_name}.json")

    def err_vs_exact(v):
        """Relative error of v against the committed exact value (None when
        this workload has no fixture)."""
        if not (golden_name and os.path.exists(golden)):
            return None
        from fractions import Fraction
        g = json.load(open(golden))
        if comps == 1 and [float(x).hex() for x in a.ravel()] == g["hex"]:
            ex = Fraction(g["exact"])
            return float(abs(Fraction(v) - ex) / abs(ex))
        if comps == 2 and [float(x.real).hex() for x in a.ravel()] == g["re_hex"]:
            er, ei = Fraction(g["exact_re"]), Fraction(g["exact_im"])
            d2 = (Fraction(v.real) - er) ** 2 + (Fraction(v.imag) - ei) ** 2
            return math.sqrt(float(d2 / (er * er + ei * ei)))
        return None

    err = err_vs_exact(value_dev) if rank == 0 else None

    # The FP32-product variant beside the line, with its measured error and the
    # call's own estimate.  It is offered only within a caller's bound: at the
    # library's 1e-12 the call refuses it (SPB_ERR_ACCURACY), so it is timed
    # with a bound it can meet (FP32_BOUND) and the refusal is recorded.
    f32 = None
    FP32_BOUND = 1e-4
    if rank == 0 and n <= 40:
        o32 = _lib.default_options(device=device, precision=_lib.SPB_PREC_FP32, rel_tol=FP32_BOUND)
        r32 = _lib.spb_result()
        st32 = 0
        for _ in range(2):
            st32 = fn_dev(ctypes.c_void_p(dev_a.data_ptr()), n, ctypes.byref(o32), ctypes.byref(r32))
        ks = []
        for _ in range(5):
            flush.zero_()
            torch.cuda.synchronize()
            st32 = fn_dev(ctypes.c_void_p(dev_a.data_ptr()), n, ctypes.byref(o32), ctypes.byref(r32))
            ks.append(r32.kernel_s)
        t32 = statistics.median(ks)
        o_def = _lib.default_options(device=device, precision=_lib.SPB_PREC_FP32)
        r_def = _lib.spb_result()
        st_def = fn_dev(ctypes.c_void_p(dev_a.data_ptr()), n, ctypes.byref(o_def), ctypes.byref(r_def))
        v32 = complex(r32.value, r32.imag) if comps == 2 else r32.value
        f32 = {"ms_per_step": t32 * 1e3, "gray_steps_per_s": n * 2 ** (n - 1) / t32,
               "speedup_vs_value": (ms_dev * 1e-3) / t32,
               "rel_err_vs_exact": err_vs_exact(v32), "err_est": r32.err_est,
               "status_at_bound": {"bound": FP32_BOUND, "status": _lib.lib().spb_status_string(st32).decode()},
               "status_at_default_bound_1e-12": _lib.lib().spb_status_string(st_def).decode(),
               "timing": "walk kernel events, median of 5 (FP32 products, double-double unit bases and sum)"}

    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        cpu, _ = run_cpu_baseline(kind, n, seed, steps=1)

    line = {"metric": "ryser_gray_steps_per_s", "value": value, "unit": "gray-steps/s",
            "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": ms_dev, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": {"workload": desc, "kind": kind, "n": n, "seed": seed,
                       "precision": args.precision, "l2": "flushed between steps (256 MiB write)",
                       "permanent": repr(value_dev), "rel_err_vs_exact": err},
            "e2e": {"value": e2e, "unit": "gray-steps/s", "h2d_bytes_per_step": n * n * 8 * comps,
                    "d2h_bytes_per_step": 16 * comps + 4,
                    "timing": "host wall clock (perf_counter) around each spb_perm_dense_* call on the "
                              "pinned host matrix, spb_options.skip_timing = 1 (no device timing queries)"},
            "roofline": roofline, "cpu_baseline": cpu, "clocks": clk.summary(),
            "gpu_launches": launches}
    if f32 is not None:
        line["fp32_products"] = f32
    if rank == 0:
        print(json.dumps(line), flush=True)
    if dist:
        dist.barrier()
        dist.destroy_process_group()
    return 0


# --------------------------------------------------------- serving (C5) --
SERVE_WORKLOADS = {
    # name: (n_lo, n_hi, requests, description)
    "serve": (8, 32, 20000, "serve_mixed_n8-32_real+complex_20k"),
    "serve_small": (8, 20, 20000, "serve_mixed_n8-20_real+complex_20k"),
}

# Requests served by the batched kernel at FP64 (n <= 24, about 1e-13 relative
# on these inputs); larger ones run the whole-GPU walk in double-double mode.
SERVE_BATCH_MAX_N = 24


# Smallest n of the derivative walk: kMinDerivReal and kMinDerivComplex
# (dense_impl.cuh), has_deriv (batch.cu).
MIN_DERIV = {"real": 24, "complex": 22, "batch": 11}


def walk_work(n, cplx, batched=False, pivot=True):
    """FP64 pipe instructions of one permanent.  The plain walk takes 2^(n-1)
    subsets at 2 per row (real: DADD + DMUL) or 6 (complex: 2 DADD, 2 DMUL, 2
    DFMA); the derivative walk, from MIN_DERIV on for a matrix with a pivot column
    (one without zeros, as every workload here has), 2^(n-2) subsets at 3 (DADD,
    DMUL, DFMA) or 10 (2 DADD, 2 DMUL, 6 DFMA)."""
    if pivot and n >= MIN_DERIV["batch" if batched else "complex" if cplx else "real"]:
        return (10 if cplx else 3) * n * 2 ** (n - 2)
    return (6 if cplx else 2) * n * 2 ** (n - 1)


def serve_work(n, cplx):
    """walk_work on the path the serving loop gives the size (batches to n = 20)."""
    return walk_work(n, cplx, batched=n <= 20)


def serve_sample(stream):
    """Requests of the stream with committed exact permanents
    (tests/golden/serve_sample.json, made by tests/golden/make_serve_golden.py):
    {index: (kind, exact)}, only those whose rebuilt matrix has the recorded
    digest."""
    from fractions import Fraction
    from superman_b200 import workloads as W
    path = os.path.join(ROOT, "tests", "golden", "serve_sample.json")
    if not os.path.exists(path):
        return {}
    g = json.load(open(path))
    if g["stream"]["count"] > len(stream) or g["stream"]["seed"] != stream.seed:
        return {}
    out = {}
    for e in g["entries"]:
        if W.matrix_sha256(stream.matrix(e["index"])) != e["sha256"]:
            continue
        if e["kind"] == "complex":
            out[e["index"]] = (Fraction(e["exact_re"]), Fraction(e["exact_im"]))
        else:
            out[e["index"]] = Fraction(e["exact"])
    return out


def rel_err_exact(v, exact):
    from fractions import Fraction
    if isinstance(exact, tuple):
        er, ei = exact
        d2 = (Fraction(v.real) - er) ** 2 + (Fraction(v.imag) - ei) ** 2
        return math.sqrt(float(d2 / (er * er + ei * ei)))
    return float(abs(Fraction(v) - exact) / abs(exact))


def serve_arm(args, wl):
    import numpy as np
    import superman_b200 as S
    from superman_b200 import _lib
    from superman_b200 import workloads as W
    from superman_b200.serving import Server, now

    n_lo, n_hi, count, desc = SERVE_WORKLOADS[wl]
    count = args.requests or count
    stream = W.ServeStream(n_lo, n_hi, count)
    mats = stream.matrices()
    cplx = [np.iscomplexobj(a) for a in mats]
    # the client keeps its requests packed: one float64 buffer, sizes, flags
    ns_all = np.array([a.shape[0] for a in mats], dtype=np.int32)
    cx_all = np.array(cplx, dtype=np.int32)
    flat = np.concatenate([(a.view(np.float64) if c else a).ravel() for a, c in zip(mats, cplx)])
    offs = np.zeros(count + 1, dtype=np.int64)
    offs[1:] = np.cumsum(ns_all.astype(np.int64) ** 2 * (1 + cx_all))
    sample = serve_sample(stream) if wl == "serve" else {}
    peak = ctypes.c_double()
    _lib.check(_lib.lib().spb_measure_pipe_peak(0, 0, ctypes.byref(peak)))
    work = sum(serve_work(a.shape[0], c) for a, c in zip(mats, cplx))
    bound_s = work / peak.value  # the stream's FP64 work at the measured pipe rate

    def one_at_a_time(sample_mats):
        t0 = time.perf_counter()
        for a in sample_mats:
            prec = "fp64" if a.shape[0] <= SERVE_BATCH_MAX_N else "dd"
            if np.iscomplexobj(a):
                S.perm_complex(a, precision=prec)
            else:
                S.perm_dense(a, precision=prec)
        return time.perf_counter() - t0

    def run_stream(srv, gaps):
        """Submits the stream (saturating when gaps is None, else at the given
        inter-arrival gaps), waits for every result; returns (results, span).
        Each result's latency counts from the request's arrival: the first
        submit for saturating arrivals, its scheduled Poisson time otherwise
        (requests that fell due while the client was busy are submitted
        together, so the client's pace does not hide queueing)."""
        tickets = []
        t_first = now()
        arrive = np.full(count, t_first)
        def submit_range(a, b):
            """Requests a..b-1 (contiguous in the packed buffer), resubmitting
            refused ones until admitted."""
            while a < b:
                got = srv.submit_flat(flat[offs[a]:offs[b]], ns_all[a:b], cx_all[a:b])
                k = 0
                while k < len(got) and got[k]:
                    tickets.append((a + k, got[k]))
                    k += 1
                for j in range(k, len(got)):  # after the first refusal, one at a time
                    if got[j]:
                        tickets.append((a + j, got[j]))
                    else:
                        while True:
                            t2 = srv.submit_flat(flat[offs[a + j]:offs[a + j + 1]], ns_all[a + j:a + j + 1],
                                                 cx_all[a + j:a + j + 1])[0]
                            if t2:
                                tickets.append((a + j, t2))
                                break
                            time.sleep(50e-6)
                a = b

        if gaps is None:
            for a in range(0, count, 1024):
                submit_range(a, min(count, a + 1024))
        else:
            arrive = t_first + np.cumsum(gaps)
            nxt = 0
            while nxt < count:
                t = now()
                if arrive[nxt] > t:
                    continue
                end = int(np.searchsorted(arrive, t, side="right"))
                submit_range(nxt, end)
                nxt = end
        res = {i: srv.wait(t, timeout_s=900) for i, t in tickets}
        for i, r in res.items():
            r["latency_s"] = r["done_s"] - arrive[i]
        span = max(r["done_s"] for r in res.values()) - t_first
        return res, span

    def latency(res, sel=lambda n: True):
        lat = np.array([r["latency_s"] for r in res.values() if sel(r["n"])])
        if lat.size == 0:
            return None
        return {"p50": float(np.percentile(lat, 50) * 1e3), "p99": float(np.percentile(lat, 99) * 1e3),
                "max": float(lat.max() * 1e3), "requests": int(lat.size)}

    one_at_a_time(mats[:50])  # warm-up (contexts, kernel attributes)
    with Server(max_batch=2048, slots=4, max_wait_s=args.max_wait) as srv:
        # warm-up (untimed): singles, then a burst of the stream, so the batch
        # shapes and padded batch sizes of the timed runs are already captured
        for a in mats[:200]:
            srv.wait(srv.submit(a))
        warm = list(mats[:4096])
        while warm:
            got = srv.submit_many(warm[:1024])
            for t in got:
                if t:
                    srv.wait(t, timeout_s=900)
            warm = [a for a, t in zip(warm[:1024], got) if not t] + warm[1024:]
        stats0 = srv.stats()
        with ClockSampler(0) as clk:
            res_sat, span_sat = run_stream(srv, None)
        capacity = count / span_sat
        rate = args.rate if args.rate > 0 else 0.8 * capacity
        gaps = np.random.default_rng(7).exponential(1.0 / rate, size=count)
        res_poi, span_poi = run_stream(srv, gaps)
        stats = srv.stats()
    for k in stats:
        if k not in ("queued_bytes", "pool_bytes"):
            stats[k] -= stats0.get(k, 0)
    bad = [r for r in list(res_sat.values()) + list(res_poi.values()) if r["status"] != 0]
    assert not bad, f"{len(bad)} requests failed"
    # accuracy: the sampled requests against their exact permanents, in both runs
    errs = []
    for i, ex in sample.items():
        for res in (res_sat, res_poi):
            errs.append(rel_err_exact(res[i]["permanent"], ex))
    # one request at a time through the plain entry points, same stream
    t_base = one_at_a_time(mats)
    base = count / t_base
    # the same matrix served in the mix and computed alone (first 64 requests)
    for i in range(64):
        a = mats[i]
        prec = "fp64" if a.shape[0] <= SERVE_BATCH_MAX_N else "dd"
        want = (S.perm_complex(a, precision=prec) if cplx[i] else S.perm_dense(a, precision=prec)).permanent
        assert abs(res_sat[i]["permanent"] - want) <= 1e-12 * abs(want), "served result differs from alone"
    in_bytes = sum(a.nbytes for a in mats)
    out_bytes = count * 32
    line = {"metric": "served_perms_per_s", "value": capacity, "unit": "perms/s", "n_gpus": 1,
            "steps": 1, "warmup": 1, "ms_per_step": span_sat * 1e3, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": {"workload": desc, "requests": count, "n_range": [n_lo, n_hi],
                       "kinds": "half real U[0,1), half blocks of 4 Haar 256x256 unitaries (seed 2026)",
                       "precision": f"batched n<={SERVE_BATCH_MAX_N}: fp64 products, dd sums; larger: dd",
                       "max_wait_s": args.max_wait,
                       "value": "saturating arrivals (whole stream submitted at once): served perms/s"},
            "latency_ms": latency(res_poi),
            "poisson": {"rate_per_s": rate, "rate_rule": "given" if args.rate > 0 else "0.8 x saturating capacity",
                        "seed": 7, "served_perms_per_s": count / span_poi,
                        "latency_ms": latency(res_poi),
                        "latency_ms_small_n_le_20": latency(res_poi, lambda n: n <= 20),
                        "latency_ms_mid_21_24": latency(res_poi, lambda n: 20 < n <= 24),
                        "latency_ms_large_n_gt_24": latency(res_poi, lambda n: n > 24)},
            "saturating": {"served_perms_per_s": capacity, "latency_ms": latency(res_sat)},
            "one_at_a_time": {"value": base, "unit": "perms/s", "seconds": t_base,
                              "how": "spb_perm_dense_f64 / spb_perm_dense_c128 per request, fp64 for n<=24, dd above"},
            "speedup_vs_one_at_a_time": capacity / base,
            "compute_bound": {"fp64_instructions": work, "peak_per_s": peak.value, "bound_s": bound_s,
                              "max_perms_per_s": count / bound_s, "served_s": span_sat,
                              "efficiency": bound_s / span_sat,
                              "one_at_a_time_efficiency": bound_s / t_base},
            "rel_err_vs_exact": {"max": max(errs) if errs else None, "sampled_requests": len(sample),
                                 "sizes": sorted({mats[i].shape[0] for i in sample}),
                                 "source": "tests/golden/serve_sample.json"},
            "e2e": {"value": capacity, "unit": "perms/s", "h2d_bytes_per_step": in_bytes,
                    "d2h_bytes_per_step": out_bytes,
                    "timing": "host clock from the first submit to the last completion"},
            "server_stats": stats, "clocks": clk.summary(), "gpu_launches": stats["batches"] * 2 + stats["large_launches"] * 5}
    print(json.dumps(line), flush=True)
    return 0


def other_arm(args, wl):
    """0/1 exact and sparse-pipeline workloads (one GPU, device-event timing)."""
    import numpy as np
    import superman_b200 as S
    from superman_b200 import _lib, workloads as W
    kind, n, seed, desc = WORKLOADS[wl]
    L = _lib.lib()
    peak = ctypes.c_double()
    if kind == "batch":
        import torch
        count = 4096
        mats = np.stack([W.dense_uniform(n, seed * 100000 + k) for k in range(count)])
        d_in = torch.from_numpy(mats).cuda()
        d_out = torch.empty(count * 2, dtype=torch.float64, device="cuda")
        _lib.check(L.spb_measure_pipe_peak(0, 0, ctypes.byref(peak)))

        def step():
            _lib.check(L.spb_perm_batch_dev(ctypes.c_void_p(d_in.data_ptr()), n, 0, count,
                                            ctypes.c_void_p(d_out.data_ptr()), None))
        for _ in range(args.warmup):
            step()
        torch.cuda.synchronize()
        with ClockSampler(0) as clk:
            t0 = time.perf_counter()
            for _ in range(args.steps):
                step()
            torch.cuda.synchronize()  # device-wide: the launches run on the library's default stream
            t = (time.perf_counter() - t0) / args.steps
        alg = count * walk_work(n, False, batched=True)
        got = d_out.cpu().numpy()[0::2]
        want0 = S.perm_dense(mats[0]).permanent
        assert abs(got[0] - want0) <= 1e-13 * abs(want0)
        # end to end: the matrices from page-locked host memory to the device,
        # the batched call, the results back, every step (host clock)
        h_in = torch.from_numpy(mats).pin_memory()
        h_out = torch.empty(count * 2, dtype=torch.float64).pin_memory()

        def step_e2e():
            d_in.copy_(h_in, non_blocking=True)
            step()
            h_out.copy_(d_out, non_blocking=True)
            torch.cuda.synchronize()
        step_e2e()
        t0 = time.perf_counter()
        for _ in range(args.steps):
            step_e2e()
        t_e2e = (time.perf_counter() - t0) / args.steps
        line = {"metric": "batched_perms_per_s", "value": count / t, "unit": "perms/s",
                "n_gpus": 1, "steps": args.steps, "warmup": args.warmup, "ms_per_step": t * 1e3,
                "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
                "data": "synthetic",
                "config": {"workload": desc, "n": n, "count": count,
                           "gray_steps_per_s": count * n * 2 ** (n - 1) / t,
                           "timing": "host clock around the launches, device-wide synchronize after"},
                "roofline": {"bound": "fp64", "achieved": alg / t / 1e12, "peak": peak.value / 1e12,
                             "unit": "T FP64-pipe inst/s", "frac": alg / t / peak.value, "traffic": None},
                "e2e": {"value": count / t_e2e, "unit": "perms/s", "h2d_bytes_per_step": int(mats.nbytes),
                        "d2h_bytes_per_step": int(h_out.numel() * 8),
                        "timing": "host clock per step: pinned host matrices copied in, spb_perm_batch_dev, "
                                  "results copied back, synchronize"},
                "clocks": clk.summary(), "gpu_launches": args.steps}
        print(json.dumps(line), flush=True)
        return 0
    if kind == "approx":
        a = (W.sparse_perm_plus(n, seed) != 0).astype(np.uint8)
        samples = 1 << 22
        for _ in range(args.warmup):
            S.perm_approx(a, samples=1 << 16, seed=1)
        rs, walls = [], []
        with ClockSampler(0) as clk:
            for k in range(args.steps):
                t0 = time.perf_counter()
                rs.append(S.perm_approx(a, samples=samples, seed=1 + k))
                walls.append(time.perf_counter() - t0)
        t = statistics.mean(x.kernel_s for x in rs)
        dt = statistics.mean(x.time for x in rs)
        nnz = int(np.count_nonzero(a))
        # the call copies the pattern (row and column pointers and indices)
        # and the two float scaling vectors in, the two-double total out
        h2d = 4 * 2 * (n + 1) + 4 * 2 * nnz + 4 * 2 * n
        line = {"metric": "samples_per_s", "value": samples / t, "unit": "samples/s",
                "n_gpus": 1, "steps": args.steps, "warmup": args.warmup, "ms_per_step": dt * 1e3,
                "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32/f64",
                "data": "synthetic",
                "config": {"workload": desc, "n": n, "samples": samples, "estimate": rs[0].permanent,
                           "rel_std_error": rs[0].err_est,
                           "timing": "kernel events of spb_perm_approx; samples per step = 2^22"},
                "roofline": None,
                "e2e": {"value": samples / statistics.mean(walls), "unit": "samples/s", "h2d_bytes_per_step": h2d,
                        "d2h_bytes_per_step": 16,
                        "timing": "host clock around each perm_approx call on the host 0/1 matrix"},
                "clocks": clk.summary(), "gpu_launches": args.steps}
        print(json.dumps(line), flush=True)
        return 0
    if kind == "binary":
        a = W.binary_bernoulli(n, seed)
        _lib.check(L.spb_measure_pipe_peak(0, 1, ctypes.byref(peak)))
        for _ in range(args.warmup):
            r = S.perm_binary(a)
        rs, walls = [], []
        with ClockSampler(0) as clk:
            for _ in range(args.steps):
                t0 = time.perf_counter()
                rs.append(S.perm_binary(a))
                walls.append(time.perf_counter() - t0)
        assert all(x.permanent == rs[0].permanent for x in rs)
        t = statistics.mean(x.kernel_s for x in rs)
        dt = statistics.mean(x.time for x in rs)
        # what the call copies: the start vector, the doubled low-column
        # table and the high columns in (its width rule), the limbs out
        wb = 8
        while wb > 2 and ((1 << wb) * n * 4 > 32 * 1024 or n - 2 - wb < 16):
            wb -= 1
        h2d = 4 * n + 4 * (1 << wb) * n + (n - 2 - wb) * n
        # limbs read back: the Bregman-Minc bound rule of the call
        nz = a != 0
        def side(m):
            rs_ = m.sum(axis=1)
            return sum(math.lgamma(r + 1) / math.log(2) / r for r in rs_) if rs_.min() > 0 else 0.0
        bits = min(side(nz), side(nz.T)) + (n - 2) + 2
        limbs = 4 if bits <= 128 else 5 if bits <= 160 else 6 if bits <= 192 else 10 if bits <= 320 else 12
        steps = n * 2 ** (n - 1)  # the integer NW walk: 2^(n-1) subsets of n rows
        # the expanded walk: 2^(n-2) subsets, one integer add + one multiply per
        # row, one multiply-add more per row of the line with the fewest ones
        m = min(int(nz.sum(axis=0).min()), int(nz.sum(axis=1).min()))
        alg = (2 * n + m) * 2 ** (n - 2)
        line = {"metric": "ryser_gray_steps_per_s", "value": steps / t, "unit": "gray-steps/s (NW, n*2^(n-1))",
                "n_gpus": 1, "steps": args.steps, "warmup": args.warmup, "ms_per_step": dt * 1e3,
                "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "int32/multi-limb",
                "data": "synthetic",
                "config": {"workload": desc, "n": n, "seed": seed, "permanent": str(rs[0].permanent),
                           "plain_ryser_equivalent_steps_per_s": n * 2 ** n / t},
                "roofline": {"bound": "int", "achieved": alg / t / 1e12, "peak": peak.value / 1e12,
                             "unit": "T int32 ops/s (row adds, products, derivative) vs IMAD pipe",
                             "frac": alg / t / peak.value, "traffic": None},
                "e2e": {"value": steps / statistics.mean(walls), "unit": "gray-steps/s (NW, n*2^(n-1))",
                        "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": 4 * limbs,
                        "timing": "host clock around each perm_binary call on the host 0/1 matrix"},
                "clocks": clk.summary(), "gpu_launches": args.steps}
    else:
        a = W.sparse_perm_plus(n, seed)
        arr = (ctypes.c_char_p * 1)(b"calculation_precision=" + args.precision.replace("fp64", "kahan").encode())
        out = _lib.spb_pipeline_result()
        def step():
            t0 = time.perf_counter()
            _lib.check(L.spb_perm_pipeline(a.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), n, arr, 1,
                                           ctypes.byref(out)))
            return time.perf_counter() - t0
        for _ in range(args.warmup):
            step()
        with ClockSampler(0) as clk:
            ts = [step() for _ in range(args.steps)]
        t = statistics.mean(ts)
        # the pieces are expanded row by row (a chain of dependent steps): no
        # pipe or memory rate bounds them, so the line has no roofline
        _, pieces = S.plan_pieces(a)
        rs = [S.perm_dense(pc, precision=args.precision) for _, pc in pieces]
        launched = sum(r.launches for r in rs)
        # the same matrix as one request of the serving loop: decomposed there,
        # its pieces run as independent requests on two whole-GPU workers
        from superman_b200.serving import Server
        with Server() as srv:
            for _ in range(2):
                srv.wait(srv.submit(a), timeout_s=600)
            lat = [srv.wait(srv.submit(a), timeout_s=600)["latency_s"] for _ in range(args.steps)]
            served_val = srv.wait(srv.submit(a), timeout_s=600)["permanent"]
            burst = 8
            t0 = time.perf_counter()
            ts_b = [srv.submit(a) for _ in range(burst)]
            for tk in ts_b:
                srv.wait(tk, timeout_s=600)
            t_burst = time.perf_counter() - t0
        err = None
        gpath = os.path.join(ROOT, "tests", "golden", "sparse_n40_s5.json")
        if os.path.exists(gpath) and n == 40 and seed == 5:
            from fractions import Fraction
            ex = Fraction(json.load(open(gpath))["exact"])
            err = float(abs(Fraction(out.permanent) - ex) / ex)
        line = {"metric": "sparse_pipeline_perms_per_s", "value": 1.0 / t, "unit": "perms/s",
                "n_gpus": 1, "steps": args.steps, "warmup": args.warmup, "ms_per_step": t * 1e3,
                "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
                "data": "synthetic",
                "config": {"workload": desc, "n": n, "seed": seed, "pieces": out.pieces, "avg_piece_n": out.avg_n,
                           "components": out.components, "algorithm": out.algorithm,
                           "permanent": repr(out.permanent),
                           "rel_err_vs_exact": err, "precision": args.precision,
                           "timing": "host wall clock around spb_perm_pipeline (pruning, decomposition, GPU pieces)"},
                "roofline": None,
                "kernels": {"kernel_us": [r.kernel_s * 1e6 for r in rs],
                            "open_columns_or_active_rows": [r.active_rows for r in rs]},
                "served": {"latency_ms_mean": statistics.mean(lat) * 1e3, "requests": len(lat),
                           "burst_of_8_perms_per_s": burst / t_burst,
                           "permanent": repr(served_val),
                           "how": "the same matrix submitted to the serving loop, which prunes and decomposes it "
                                  "and runs the pieces as independent requests"},
                "e2e": {"value": 1.0 / t, "unit": "perms/s", "h2d_bytes_per_step": n * n * 8,
                        "d2h_bytes_per_step": 16 * max(1, len(pieces)),
                        "timing": "host wall clock around the public call"},
                "clocks": clk.summary(), "gpu_launches": launched * args.steps}
    if not args.no_cpu_baseline:
        cores = os.cpu_count() or 1
        import tempfile
        with tempfile.TemporaryDirectory() as d:
            p = os.path.join(d, "m.mtx")
            write_mtx(p, a.astype(np.float64))
            sys.path.insert(0, os.path.join(ROOT, "oracle"))
            import oracle as O
            if os.path.exists(O.ref_binary_path()):
                v, secs = O.run_reference(p, threads=cores, timeout=1800)
                line["cpu_baseline"] = {"value": (1.0 / secs) if kind == "sparse" else (n * 2 ** (n - 1) / secs),
                                        "unit": line["unit"] if kind == "sparse" else "gray-steps/s (NW)",
                                        "cores": cores, "kind": "reference",
                                        "sample": f"reference CPU binary on the same matrix, {secs:.3f} s",
                                        "permanent": v}
    print(json.dumps(line), flush=True)
    return 0


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", choices=["ours", "reference", "reference_gpu"], default="ours")
    ap.add_argument("--workload", choices=sorted(WORKLOADS) + sorted(SERVE_WORKLOADS), default="dense32")
    ap.add_argument("--requests", type=int, default=0, help="serving: stream length (0 = workload default)")
    ap.add_argument("--rate", type=float, default=0.0,
                    help="serving: Poisson arrivals per s (0 = 0.8 x the measured saturating capacity)")
    ap.add_argument("--max-wait", type=float, default=200e-6, help="serving: batch fill window (s)")
    # dd: the accuracy bar of the headline (<= 1e-12 relative at n=32) needs the
    # double-double re-evaluation of the dominant units; fp64 is ~3e-12 there.
    ap.add_argument("--precision", choices=["fp64", "dd"], default="dd")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    args = ap.parse_args()
    if args.warmup < 3:
        args.warmup = 3
    if args.impl == "reference":
        return reference_arm(args, args.workload)
    if args.impl == "reference_gpu":
        return reference_gpu_arm(args, args.workload)
    if args.workload in SERVE_WORKLOADS:
        return serve_arm(args, args.workload)
    if WORKLOADS[args.workload][0] in ("binary", "sparse", "batch", "approx"):
        return other_arm(args, args.workload)
    return ours_arm(args, args.workload)


if __name__ == "__main__":
    sys.exit(main())
