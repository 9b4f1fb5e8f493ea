#!/usr/bin/env python
"""LDL^T solve benchmark on B200.

Default workload (the metric's largest single-GPU configuration): plain FP64
blocked Bunch-Kaufman LDL^T factorization plus the solve of 4 right-hand
sides for a random symmetric indefinite matrix, n = 40000 (12.8 GB FP64 in
HBM), entries uniform[-1, 1] plus N(0, 0.01) on the diagonal, block size
256.  Seeded synthetic inputs.

metric: GFLOP/s = (n^3 / 3) / (time of factorization + solve), whole job.
The same line carries the metric's other two parts:
  mixed     FP64 vs low-precision trailing updates (FP32, BF16x3, BF16) +
            FP64 FGMRES refinement, time to backward error <= 1e-12, on the
            n = 40000 matrix above and on the ill-conditioned spectral matrix
            (n = 20000, condition ~1e8, 16 right-hand sides);
  batched   4096 KKT matrices, n ~ U[16, 512], factored and solved in one
            persistent launch (CUDA graph), FP64 and FP32 + FP64 refinement,
            matrices/s against looping the single-matrix path.

Arms:
  (default)          this library on the GPU(s); one process per GPU under
                     torchrun, replicas only (every rank factors its own copy).
  --impl reference   the reference's own CPU implementation (compiled from its
                     sources into oracle/_ref) on the host cores, a bounded
                     sample of the workload per step.
"""
from __future__ import annotations

import argparse
import csv
import datetime
import io
import json
import math
import os
import statistics
import subprocess
import sys
import tempfile
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "LDL^T solve GFLOP/s: FP64 vs FP32/BF16+IR at <=1e-12 bwd err; batched mats/s"
UNIT = "GFLOP/s"
MEASURED_PEAKS = os.path.join(ROOT, "MEASURED_PEAKS.json")
FALLBACK_HBM_GBS = 6650.0
FALLBACK_BF16_TFLOPS = 1400.0
DIGIT_PRODUCTS = 34  # INT8 products per FP64 product of the digit update (csrc/update_i8.cu)


def parse_args():
    ap = argparse.ArgumentParser(description=__doc__, formatter_class=argparse.RawDescriptionHelpFormatter)
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="b200", choices=["b200", "reference"])
    ap.add_argument("--workload", default="all", choices=["all", "fp64", "mixed", "batched"],
                    help="all: the FP64 line with the mixed and batched parts attached (default); "
                         "fp64: the FP64 line alone; mixed / batched: one part alone, on its own line")
    ap.add_argument("--matrix", default="random", choices=["random", "kkt", "spectral"],
                    help="the FP64 line's matrix: random indefinite (n=40000, block 256, 4 RHS; default), "
                         "KKT saddle point (n=10000, block 128, 1 RHS); mixed alone: random or spectral")
    ap.add_argument("--n", type=int, default=None)
    ap.add_argument("--h", type=int, default=None, help="KKT: H block order (default 0.8 n)")
    ap.add_argument("--block", type=int, default=None)
    ap.add_argument("--nrhs", type=int, default=None)
    ap.add_argument("--mode", default="fp64", choices=["fp64", "fp64_ordered", "fp32", "bf16x3", "bf16"],
                    help="the FP64 line's trailing-update arithmetic (the low-precision modes are for "
                         "profiling their update kernels: the line's solve is then unrefined)")
    ap.add_argument("--seed", type=int, default=20240)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--e2e-steps", type=int, default=3)
    ap.add_argument("--cpu-seconds", type=float, default=12.0, help="target CPU baseline sample time")
    ap.add_argument("--count", type=int, default=4096, help="batched: matrices per GPU")
    ap.add_argument("--loop-sample", type=int, default=256,
                    help="batched: matrices timed through the looped single-matrix path")
    args = ap.parse_args()
    defaults = {"random": (40000, 256, 4), "kkt": (10000, 128, 1), "spectral": (20000, 128, 16)}
    dn, db, dr = defaults[args.matrix]
    args.n = args.n if args.n is not None else dn
    args.block = args.block if args.block is not None else db
    args.nrhs = args.nrhs if args.nrhs is not None else dr
    return args


def flops_ldlt(n: int) -> float:
    return n ** 3 / 3.0


def matrix_description(kind: str, n: int, h=None) -> str:
    if kind == "kkt":
        h = h if h is not None else int(round(0.8 * n))
        return f"KKT saddle point n={n} (H {h} SPD = G G^T/{h} + 1e-2 I, B Gaussian, zero (2,2) block)"
    if kind == "spectral":
        return f"A = Q diag(lam) Q^T, n={n}, |lam| log-uniform [1e-4, 1e4], half negative (condition ~1e8)"
    return f"random symmetric indefinite n={n} (uniform[-1,1] entries plus N(0, 0.01) on the diagonal)"


def workload_config(args, n_used=None) -> dict:
    n = args.n if n_used is None else n_used
    return {
        "workload": f"plain FP64 blocked Bunch-Kaufman LDL^T factor + solve, "
                    f"{matrix_description(args.matrix, n, args.h if n_used is None else None)}, "
                    f"block {args.block}, {args.nrhs} RHS",
        "n": n, "block_size": args.block, "nrhs": args.nrhs, "update": args.mode,
    }


# ---------------------------------------------------------------------------
# multi-process helpers (one process per GPU; NCCL on GPUs, gloo in the CPU tests)
# ---------------------------------------------------------------------------
def reduce_max_over_ranks(value: float, world: int, device) -> float:
    """The maximum of `value` over all ranks of the default process group
    (every rank calls it the same number of times, in the same order)."""
    if world <= 1:
        return float(value)
    import torch
    import torch.distributed as dist
    t = torch.tensor([float(value)], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def job_throughput(units_per_rank: float, world: int, max_ms: float) -> float:
    """Whole-job rate: every rank's units over the slowest rank's time."""
    return world * units_per_rank / (max_ms / 1e3)


def batch_seed(seed: int, rank: int) -> int:
    """Each rank of the batched workload owns its own seeded batch."""
    return seed + 1000 * rank


# ---------------------------------------------------------------------------
# clocks sampling (nvidia-smi during the timed region)
# ---------------------------------------------------------------------------
class ClockSampler:
    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index: int):
        self.gpu = gpu_index
        self.proc = None
        self.path = None

    def start(self):
        try:
            fd, self.path = tempfile.mkstemp(prefix="bbk_clocks_", suffix=".csv")
            os.close(fd)
            self.out = open(self.path, "w")
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--id={self.gpu}", f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits",
                 "-lms", "100"], stdout=self.out, stderr=subprocess.DEVNULL)
        except (OSError, FileNotFoundError):
            self.proc = None

    def stop(self) -> dict:
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        self.out.close()
        rows = []
        with open(self.path) as fh:
            for r in csv.reader(fh):
                if len(r) >= 9:
                    rows.append([x.strip() for x in r])
        os.unlink(self.path)
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["no samples"]}
        sm = [float(r[1]) for r in rows if r[1].replace(".", "").isdigit()]
        mx = [float(r[2]) for r in rows if r[2].replace(".", "").isdigit()]
        loaded = [s for s in sm if s > 0.5 * max(sm)] if sm else []
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[i] for r in rows for i in range(4) if r[5 + i].lower() == "active"})
        return {"sm_mhz": statistics.median(loaded) if loaded else None,
                "sm_max_mhz": max(mx) if mx else None, "reasons": reasons, "samples": len(rows)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def kkt_device(n: int, h: int, seed: int, device):
    import torch
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    gm = torch.randn(h, h, generator=g, dtype=torch.float64, device=device)
    a = torch.zeros(n, n, dtype=torch.float64, device=device)
    a[:h, :h] = gm @ gm.T / h
    a[:h, :h] += 1e-2 * torch.eye(h, dtype=torch.float64, device=device)
    del gm
    bm = torch.randn(n - h, h, generator=g, dtype=torch.float64, device=device)
    a[h:, :h] = bm
    a[:h, h:] = bm.T
    rhs = torch.randn(n, generator=g, dtype=torch.float64, device=device)
    return a, rhs


def kkt_host(n: int, h: int, seed: int):
    import numpy as np
    rng = np.random.default_rng(seed)
    g = rng.standard_normal((h, h))
    a = np.zeros((n, n))
    a[:h, :h] = g @ g.T / h + 1e-2 * np.eye(h)
    bm = rng.standard_normal((n - h, h))
    a[h:, :h] = bm
    a[:h, h:] = bm.T
    return a


def random_indefinite_host(n: int, seed: int):
    """The random indefinite structure on the host (numpy PCG64): entries
    uniform[-1, 1], upper triangle mirrored, plus N(0, 0.01) on the diagonal."""
    import numpy as np
    rng = np.random.default_rng(seed)
    u = rng.uniform(-1.0, 1.0, size=(n, n))
    a = np.triu(u)
    a = a + np.triu(a, 1).T
    a[np.diag_indices(n)] += 0.1 * rng.standard_normal(n)
    return a


def host_matrix(kind: str, n: int, seed: int):
    """A host matrix of the FP64 line's structure for the CPU reference."""
    if kind == "kkt":
        return kkt_host(n, int(round(0.8 * n)), seed)
    if kind == "spectral":
        import numpy as np
        rng = np.random.default_rng(seed)
        q, _ = np.linalg.qr(rng.standard_normal((n, n)))
        lam = np.exp(rng.uniform(np.log(1e-4), np.log(1e4), n)) * np.where(rng.permutation(n) < n // 2, -1.0, 1.0)
        a = (q * lam) @ q.T
        return (a + a.T) / 2
    return random_indefinite_host(n, seed)


def measure_dgemm_tflops(device) -> float:
    import torch
    n = 8192
    x = torch.randn(n, n, dtype=torch.float64, device=device)
    y = torch.randn(n, n, dtype=torch.float64, device=device)
    for _ in range(2):
        z = x @ y
    torch.cuda.synchronize()
    best = float("inf")
    for _ in range(3):
        s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        s.record()
        z = x @ y
        e.record()
        torch.cuda.synchronize()
        best = min(best, s.elapsed_time(e) / 1e3)
    del x, y, z
    return 2 * n ** 3 / best / 1e12


def measured_hbm_gbs():
    try:
        with open(MEASURED_PEAKS) as fh:
            return float(json.load(fh)["hbm_gbs"]), "MEASURED_PEAKS.json hbm_gbs (measured)"
    except (OSError, KeyError, ValueError):
        return FALLBACK_HBM_GBS, "fallback 6.65 TB/s"


# ---------------------------------------------------------------------------
# algorithmic work per kernel class
# ---------------------------------------------------------------------------
def update_flops(n: int, panel_end) -> float:
    f, k0 = 0.0, 0
    for e in panel_end:
        kb, m = e - k0, n - e
        if m > 0:
            f += 2.0 * kb * m * (m + 1) / 2.0
        k0 = e
    return f


def digit_update_flops(n: int, blk: int, panel_end) -> float:
    """The part of update_flops that the integer tensor cores do: the panels
    whose trailing order and block size reach the line drawn in
    csrc/update_i8.cu (launch_update_i8)."""
    f, k0 = 0.0, 0
    for e in panel_end:
        kb, m = e - k0, n - e
        if m >= 1024 and m * blk >= 512 * 1024 and blk >= 64:
            f += 2.0 * kb * m * (m + 1) / 2.0
        k0 = e
    return f


def measured_int8_tops():
    """INT8 tensor peak: twice the measured sustained cuBLAS bf16 rate (the
    tensor cores' INT8 rate is twice their bf16 rate, under the same power
    limit)."""
    try:
        with open(MEASURED_PEAKS) as fh:
            return 2.0 * float(json.load(fh)["bf16_tflops_sustained"]), \
                "2 x MEASURED_PEAKS.json bf16_tflops_sustained (measured)"
    except (OSError, KeyError, ValueError):
        return 2.0 * FALLBACK_BF16_TFLOPS, "2 x fallback 1.4 PFLOP/s sustained bf16"


def panel_bytes(n: int, panel_end) -> float:
    """Compulsory DRAM bytes of the panel launches: each panel of width w
    starting at row k0 reads its w x (n - k0) strip of the matrix and writes
    the workspace rows W and the compact factor rows of the same shape
    (3 x 8 bytes per strip entry)."""
    b, k0 = 0.0, 0
    for e in panel_end:
        b += 24.0 * (e - k0) * (n - k0)
        k0 = e
    return b


# ---------------------------------------------------------------------------
# this library
# ---------------------------------------------------------------------------
def make_matrix(kind: str, n: int, nrhs: int, seed: int, device, h=None):
    """The FP64 line's input on the device: (matrix n x n, right-hand sides
    nrhs x n)."""
    if kind == "kkt":
        a, b0 = kkt_device(n, h if h is not None else int(round(0.8 * n)), seed, device)
        rhs = b0.reshape(1, n).repeat(nrhs, 1).contiguous()
        return a, rhs
    if kind == "spectral":
        a, rhs = spectral_device(n, seed, device)
        return a, rhs[:nrhs].contiguous()
    return random_indefinite_device(n, seed, device, nrhs)


def traffic_per_unit(key: str, kernel: str):
    """DRAM bytes per algorithmic unit of `kernel` measured by ncu on the
    workload `key` (profiles/traffic.json), or None."""
    path = os.path.join(ROOT, "profiles", "traffic.json")
    try:
        with open(path) as fh:
            return float(json.load(fh)["workloads"][key][kernel]["bytes_per_unit"])
    except (OSError, ValueError, KeyError, TypeError):
        return None


def run_main(args):
    """The FP64 factor + solve line (every rank a replica), then, on rank 0
    after the ranks have finished together, the mixed-precision and batched
    parts of the metric (workload "all")."""
    import ctypes

    import numpy as np
    import torch
    import torch.distributed as dist

    import blockedbunchkaufmanldlt_b200 as bbk

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    if world > 1:
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=300), device_id=dev)

    def barrier():
        if world > 1:
            dist.barrier()

    def max_over_ranks(x: float) -> float:
        return reduce_max_over_ranks(x, world, dev)

    n, blk, nrhs = args.n, args.block, args.nrhs
    a0, rhs0 = make_matrix(args.matrix, n, nrhs, args.seed, dev, args.h)
    dgemm = measure_dgemm_tflops(dev)
    hbm, hbm_src = measured_hbm_gbs()

    work = torch.empty_like(a0)
    x = torch.empty_like(rhs0)
    ws_f = torch.empty(bbk.factor_workspace_size(n, blk), dtype=torch.uint8, device=dev)
    ws_s = torch.empty(bbk.solve_workspace_size(n, nrhs), dtype=torch.uint8, device=dev)
    stream = torch.cuda.current_stream()
    L = bbk.lib()
    nb = (n + blk - 1) // blk
    perm = torch.empty(n, dtype=torch.int32, device=dev)
    pt = torch.empty(n, dtype=torch.int32, device=dev)
    pe = torch.empty(nb, dtype=torch.int32, device=dev)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    vp = ctypes.c_void_p
    sp = vp(stream.cuda_stream)
    mode = bbk.UPDATE_MODES[args.mode]

    def step():
        work.copy_(a0)
        bbk.check(L.bbk_factor_device_async(n, blk, vp(work.data_ptr()), n, vp(perm.data_ptr()),
                                            vp(pt.data_ptr()), vp(pe.data_ptr()), mode, vp(ws_f.data_ptr()),
                                            ws_f.numel(), vp(status.data_ptr()), sp))
        x.copy_(rhs0)
        bbk.check(L.bbk_solve_device(n, vp(work.data_ptr()), n, vp(perm.data_ptr()), vp(pt.data_ptr()),
                                     nrhs, vp(x.data_ptr()), n, vp(ws_s.data_ptr()), ws_s.numel(), sp))

    for _ in range(max(args.warmup, 0)):
        step()
    torch.cuda.synchronize()
    if int(status.item()) != 0:
        raise RuntimeError(f"device status {int(status.item())}")

    sampler = ClockSampler(local)
    sampler.start()
    barrier()
    torch.cuda.synchronize()
    launches0 = bbk.kernel_launch_count()
    bbk.profile_begin()
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    ev0.record()
    for _ in range(args.steps):
        step()
    ev1.record()
    torch.cuda.synchronize()
    barrier()
    prof = bbk.profile_end()
    launches = bbk.kernel_launch_count() - launches0
    clocks = sampler.stop()
    ms = max_over_ranks(ev0.elapsed_time(ev1))
    ms_step = ms / args.steps
    value = world * flops_ldlt(n) / (ms_step / 1e3) / 1e9

    # accuracy of the last step: backward error of every solve (FP64, on device)
    r = rhs0.T - a0 @ x.T
    anorm = a0.abs().sum(1).amax()
    berr = float((r.abs().amax(0) / (anorm * x.T.abs().amax(0) + rhs0.T.abs().amax(0))).max().item())
    del r
    pe_h = pe.cpu().numpy().tolist()
    pt_h = pt.cpu().numpy()
    n1, n2 = int((pt_h == 1).sum()), int((pt_h == 2).sum())
    shifts = sum(1 for P, e in enumerate(pe_h) if e < min((P + 1) * blk, n))

    # per-kernel roofline from the live profile
    upd_flops = update_flops(n, pe_h) * args.steps
    pan_bytes = panel_bytes(n, pe_h) * args.steps
    kernels = {}
    if prof["update"]["ms"] > 0:
        kernels["trailing_update"] = {
            "bound": "tensor", "achieved": upd_flops / (prof["update"]["ms"] / 1e3) / 1e12, "unit": "TFLOP/s",
            "peak": dgemm, "peak_source": "cuBLAS DGEMM 8192^3 measured in this run (FP64 tensor peak)",
            "ms": prof["update"]["ms"], "launches": prof["update"]["launches"]}
        # In the FP64 mode large panels run as INT8 digit products on the
        # integer tensor cores, whose peak is then the one that bounds them;
        # the FP64 rate stays beside it.
        digit_flops = digit_update_flops(n, blk, pe_h) * args.steps if args.mode == "fp64" else 0.0
        upd = kernels["trailing_update"]
        upd["fp64_tflops"] = upd["achieved"]
        upd["fp64_of_dgemm"] = upd["achieved"] / dgemm
        if digit_flops > 0.5 * upd_flops:
            upd["achieved"] = DIGIT_PRODUCTS * digit_flops / (prof["update"]["ms"] / 1e3) / 1e12
            upd["unit"] = "TOP/s (INT8)"
            upd["peak"], upd["peak_source"] = measured_int8_tops()
        upd["frac"] = upd["achieved"] / upd["peak"]
    if prof["panel"]["ms"] > 0:
        kernels["panel"] = {
            "bound": "hbm", "achieved": pan_bytes / (prof["panel"]["ms"] / 1e3) / 1e9, "unit": "GB/s",
            "peak": hbm, "peak_source": hbm_src, "ms": prof["panel"]["ms"], "launches": prof["panel"]["launches"],
            "us_per_pivot_step": prof["panel"]["ms"] * 1e3 / (args.steps * n)}
        kernels["panel"]["frac"] = kernels["panel"]["achieved"] / hbm
    for k in ("finalize", "solve", "init"):
        kernels[k] = {"ms": prof[k]["ms"], "launches": prof[k]["launches"]}
    total_prof = sum(prof[k]["ms"] for k in prof)
    for k, v in kernels.items():
        v["share"] = (v["ms"] / total_prof) if total_prof > 0 else None
    dom = max(("trailing_update", "panel"), key=lambda k: kernels.get(k, {}).get("ms", 0.0))
    dk = kernels[dom]
    # DRAM bytes per launch: the bytes per unit an ncu capture of this
    # workload measured (profiles/traffic.json) times the units of an average
    # launch of this run
    traffic = None
    per_unit = traffic_per_unit(f"{args.matrix}_n{n}_b{blk}", dom)
    if per_unit is not None and dk.get("launches"):
        if dom == "panel":
            units, k0 = 0.0, 0
            for e in pe_h:
                units += float(e - k0) * (n - k0)
                k0 = e
            units *= args.steps
        else:
            units = upd_flops
        traffic = per_unit * units / dk["launches"]
    update_units = "2 * width * m(m+1)/2 flops per panel update (m trailing rows), summed over the launches"
    if "INT8" in kernels.get("trailing_update", {}).get("unit", ""):
        update_units += (f"; as {DIGIT_PRODUCTS} INT8 operations per flop on the panels the digit update takes "
                         "(achieved), traffic per FP64 flop")
    roofline = {"kernel": dom, "bound": dk["bound"], "achieved": dk["achieved"], "peak": dk["peak"],
                "unit": dk["unit"], "frac": dk["frac"], "traffic": traffic, "peak_source": dk["peak_source"],
                "algorithmic_units": (update_units if dom == "trailing_update" else
                                      "24 bytes per panel-strip entry (width x trailing order)")}
    if "panel" in kernels:
        # The panel is a chain of pivot steps, each needing one grid-wide
        # exchange (argmax + published scalars) before the next can start:
        # its floor is one bare exchange per step, measured here on the same
        # grid (bbk_probe_exchange_ns: back-to-back exchanges, each with a
        # release fence).
        sms = torch.cuda.get_device_properties(torch.cuda.current_device()).multi_processor_count
        grid = max(min(sms, -(-n // 64)), -(-n // 576))  # the panel launch's grid (64 columns per CTA)
        try:
            x_ns = bbk.probe_exchange_ns(int(grid), 2000)
        except Exception:  # noqa: BLE001 - diagnostics only
            x_ns = None
        per_step_us = kernels["panel"]["ms"] * 1e3 / (args.steps * n)
        if x_ns:
            kernels["panel"]["latency"] = {"unit": "us per pivot step", "achieved": per_step_us,
                                           "floor": x_ns / 1e3, "frac": (x_ns / 1e3) / per_step_us,
                                           "floor_source": "one bare grid exchange per pivot step, "
                                                           "measured live", "grid": int(grid)}
            if dom == "panel":
                roofline["latency"] = kernels["panel"]["latency"]

    # end to end through the host-buffer C ABI (pinned host memory)
    e2e = None
    del work
    if not args.no_e2e:
        ha = a0.cpu().pin_memory()
        hb = rhs0.cpu().pin_memory()
        hwork = torch.empty_like(ha).pin_memory()
        hx = torch.empty_like(hb).pin_memory()
        hperm = torch.empty(n, dtype=torch.int32).pin_memory()
        hpt = torch.empty(n, dtype=torch.int32).pin_memory()
        hpe = torch.empty(nb, dtype=torch.int32).pin_memory()

        def restore():
            hwork.copy_(ha)
            hx.copy_(hb)

        def e2e_call():
            bbk.check(L.bbk_factor_solve_host(n, blk, vp(hwork.data_ptr()), n, vp(hperm.data_ptr()),
                                              vp(hpt.data_ptr()), vp(hpe.data_ptr()), nrhs, vp(hx.data_ptr()),
                                              n, mode))

        restore()
        e2e_call()
        k_e2e = max(1, min(args.steps, args.e2e_steps))
        tot_ms = 0.0
        for _ in range(k_e2e):
            restore()  # the caller's input is restored outside the timed call
            barrier()
            torch.cuda.synchronize()
            s0, s1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            t0 = time.perf_counter()
            s0.record()
            e2e_call()  # synchronous: H2D, factor, solve, D2H
            s1.record()
            torch.cuda.synchronize()
            wall = (time.perf_counter() - t0) * 1e3
            tot_ms += max(s0.elapsed_time(s1), wall)
        ems = max_over_ranks(tot_ms) / k_e2e
        # the host entry points move the upper triangle as 64-row wedges
        upper = sum(8 * (n - k) * min(64, n - k) for k in range(0, n, 64))
        h2d = upper + nrhs * n * 8
        d2h = upper + nrhs * n * 8 + 4 * (2 * n + nb)
        e2e = {"value": world * flops_ldlt(n) / (ems / 1e3) / 1e9, "unit": UNIT, "ms_per_step": ems,
               "steps": k_e2e, "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h,
               "api": "bbk_factor_solve_host (host buffers, pinned): H2D of the matrix's upper triangle "
                      "(64-row wedges) and right-hand sides, factor, solve, D2H of compact factors, pivots "
                      "and solutions, inside each timed step"}
        del ha, hb, hwork, hx

    if world > 1:
        dist.destroy_process_group()
    if rank != 0:
        return

    cpu = None
    if world == 1 and not args.no_cpu_baseline:
        cpu = cpu_baseline_sample(args, target_s=args.cpu_seconds)

    line = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": ms_step, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None,
        "dtype": "f64" if args.mode in ("fp64", "fp64_ordered") else f"f64+{args.mode}-update",
        "data": f"synthetic: seeded {matrix_description(args.matrix, n, args.h)} (torch generators on the device)",
        "config": dict(workload_config(args), parallelism=f"replicas x{world} (one matrix per GPU)",
                       seed=args.seed,
                       l2=f"inputs larger than L2 (the n x n FP64 matrix, {8 * n * n / 1e9:.1f} GB); the input "
                          "is restored by a device copy inside each timed step"),
        "e2e": e2e, "roofline": roofline, "kernels": kernels, "cpu_baseline": cpu,
        "clocks": clocks, "gpu_launches": launches,
        "accuracy": {"backward_error_max_over_rhs": berr, "pivots_1x1": n1, "pivots_2x2": n2,
                     "boundary_shifts": shifts},
        "fp64_dgemm_tflops": dgemm,
    }
    if args.workload == "all":
        # the metric's other parts, on this GPU, after the timed line
        fp64_ref = {"ms": ms_step, "backward_error": berr, "refine_steps": 0,
                    "how": "the FP64 line's factor + solve time per step (input restore included)"}
        modes = ("fp32", "bf16x3", "bf16") if args.matrix == "random" else ("fp32", "bf16x3")
        mixed = {f"{args.matrix}_n{n}": mixed_arms(a0, rhs0, blk, modes, fp64=fp64_ref, x64=x,
                                                   what=f"{matrix_description(args.matrix, n, args.h)}, "
                                                        f"block {blk}, {nrhs} RHS")}
        del a0, rhs0, x
        torch.cuda.empty_cache()
        a3, rhs3 = spectral_device(20000, args.seed, dev)
        mixed["spectral_n20000"] = mixed_arms(a3, rhs3, 128, ("fp32", "bf16x3"),
                                              what=f"{matrix_description('spectral', 20000)}, block 128, 16 RHS")
        del a3, rhs3
        torch.cuda.empty_cache()
        line["mixed"] = mixed
        line["batched"] = batched_results(args, 1, 0, dev)
    print(json.dumps(line), flush=True)


# ---------------------------------------------------------------------------
# CPU: the reference (oracle/_ref) on the host cores
# ---------------------------------------------------------------------------
def _reference_lib():
    os.environ.setdefault("OMP_PROC_BIND", "close")
    from oracle.oracle import Port, Reference
    if Reference.available():
        return Reference(), "reference"
    return Port(), "port"


def _cpu_factor(lib, kind, a, blk):
    if kind == "reference":
        t0 = time.perf_counter()
        f = lib.factor(a, blk)
        return f.seconds if f.seconds else time.perf_counter() - t0
    t0 = time.perf_counter()
    lib.factor(a, blk)
    return time.perf_counter() - t0


def _pick_sample_n(lib, kind, args, target_s: float) -> int:
    n_cal = 1536
    a = host_matrix(args.matrix, n_cal, args.seed)
    t = _cpu_factor(lib, kind, a, args.block)
    rate = flops_ldlt(n_cal) / max(t, 1e-6)
    n_s = int((3.0 * rate * target_s) ** (1.0 / 3.0))
    n_s = max(n_cal, min(args.n, (n_s // args.block) * args.block))
    return n_s


def cpu_baseline_sample(args, target_s: float) -> dict:
    lib, kind = _reference_lib()
    cores = lib.threads() if kind == "reference" else 1
    n_s = _pick_sample_n(lib, kind, args, target_s)
    a = host_matrix(args.matrix, n_s, args.seed)
    t = _cpu_factor(lib, kind, a, args.block)
    return {"value": flops_ldlt(n_s) / t / 1e9, "unit": UNIT, "cores": cores, "kind": kind,
            "sample": f"one factorization of a {matrix_description(args.matrix, n_s)}, block {args.block}, "
                      f"ctor + Factorize() timed with {cores} threads (a bounded sample: the reference at "
                      f"n={args.n} would take far longer than a benchmark run); the reference has no solve",
            "seconds": t}


def run_reference(args):
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    lib, kind = _reference_lib()
    cores = lib.threads() if kind == "reference" else 1
    total_steps = max(1, args.steps) + max(0, args.warmup)
    per_step = max(2.0, min(30.0, 150.0 / total_steps))
    n_s = _pick_sample_n(lib, kind, args, per_step)
    a = host_matrix(args.matrix, n_s, args.seed)
    for _ in range(max(0, args.warmup)):
        _cpu_factor(lib, kind, a, args.block)
    times = [_cpu_factor(lib, kind, a, args.block) for _ in range(max(1, args.steps))]
    tot = sum(times)
    value = flops_ldlt(n_s) * len(times) / tot / 1e9
    sample = (f"each step one factorization of a {matrix_description(args.matrix, n_s)}, block "
              f"{args.block}, ctor + Factorize() timed with {cores} OpenMP threads; n is bounded so the run "
              f"ends in minutes (the reference at n={args.n} would take over an hour); the reference has no "
              "solve")
    cfg = workload_config(args, n_used=n_s)
    cfg["l2"] = "host memory (CPU run): every step factors the same host matrix, copied by the reference's constructor"
    line = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": len(times),
        "warmup": args.warmup, "ms_per_step": tot / len(times) * 1e3, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f64", "impl": "reference",
        "data": f"synthetic: seeded {matrix_description(args.matrix, n_s)} (numpy PCG64)",
        "config": cfg,
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": cores, "kind": kind, "sample": sample},
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


def random_indefinite_device(n: int, seed: int, device, nrhs: int):
    """Entries uniform[-1, 1] (upper triangle mirrored) plus N(0, 0.01) on the
    diagonal: a random symmetric indefinite matrix; nrhs right-hand sides
    N(0, 1) as rows."""
    import torch
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    a = torch.empty(n, n, dtype=torch.float64, device=device).uniform_(-1.0, 1.0, generator=g)
    a = torch.triu(a)
    a = a + torch.triu(a, 1).T
    a.diagonal().add_(torch.randn(n, generator=g, dtype=torch.float64, device=device) * 0.1)
    rhs = torch.randn(nrhs, n, generator=g, dtype=torch.float64, device=device)
    return a, rhs


def spectral_device(n: int, seed: int, device, lo=1e-4, hi=1e4):
    """A = Q diag(lam) Q^T, Q from the QR of a Gaussian matrix, |lam|
    log-uniform in [lo, hi], half the signs negative (condition ~ hi/lo)."""
    import torch
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    q, _ = torch.linalg.qr(torch.randn(n, n, generator=g, dtype=torch.float64, device=device))
    mag = torch.exp(torch.empty(n, dtype=torch.float64, device=device).uniform_(
        float(torch.log(torch.tensor(lo))), float(torch.log(torch.tensor(hi))), generator=g))
    sign = torch.ones(n, dtype=torch.float64, device=device)
    sign[torch.randperm(n, generator=g, device=device)[: n // 2]] = -1.0
    a = (q * (sign * mag)) @ q.T
    del q
    a = (a + a.T) * 0.5
    rhs = torch.randn(16, n, generator=g, dtype=torch.float64, device=device)
    return a, rhs


def mixed_arms(a0, rhs, blk: int, modes, fp64=None, x64=None, what: str = "", tol: float = 1e-12) -> dict:
    """Time to a solution with backward error <= tol for every right-hand
    side (rows of `rhs`): the FP64 path (factor + solve; `fp64` / `x64` when
    the caller already timed it) against each low-precision trailing update
    in `modes` followed by FP64 FGMRES refinement (restart 50, at most 3
    outer steps) against the original matrix.  Each arm: one untimed run,
    then one timed run (CUDA events and the host clock, the larger)."""
    import torch

    import blockedbunchkaufmanldlt_b200 as bbk
    n = a0.shape[0]
    anorm = a0.abs().sum(1).amax()

    def berr(x):
        r = rhs.T - a0 @ x.T
        return float((r.abs().amax(0) / (anorm * x.T.abs().amax(0) + rhs.T.abs().amax(0))).max())

    def timed(fn):
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        t0 = time.perf_counter()
        e0.record()
        out = fn()
        e1.record()
        torch.cuda.synchronize()
        return out, max(e0.elapsed_time(e1), (time.perf_counter() - t0) * 1e3)

    results = {}
    if fp64 is None:
        for _ in range(2):
            w = a0.clone()

            def fp64_path():
                perm, pt, _ = bbk.factor_device(w, blk, mode="fp64")
                x = rhs.clone()
                bbk.solve_device(w, perm, pt, x)
                return x
            x64, ms = timed(fp64_path)
            del w
        fp64 = {"ms": ms, "backward_error": berr(x64), "refine_steps": 0}
    results["fp64"] = fp64
    xnorm = x64.abs().amax()
    for mode in modes:
        for _ in range(2):
            w = a0.clone()

            def mixed_path():
                perm, pt, _ = bbk.factor_device(w, blk, mode=mode)
                x, info = bbk.solve_refined_device(a0, w, perm, pt, rhs, tol=tol, max_iter=3,
                                                   method="gmres", restart=50)
                return x, info
            (x, info), ms = timed(mixed_path)
            del w
        fe = float((x - x64).abs().amax() / xnorm)
        results[mode + "+ir"] = {
            "ms": ms, "backward_error": berr(x), "initial_backward_error": info.initial_backward_error,
            "refine_steps": info.iterations, "gmres_steps": info.inner_iterations,
            "converged": bool(info.converged), "forward_error_vs_fp64": fe,
            "speedup_vs_fp64": fp64["ms"] / ms}
        del x
    conv = [k for k, v in results.items() if k != "fp64" and v["converged"]]
    best = min(conv, key=lambda k: results[k]["ms"]) if conv else None
    return {"workload": what, "n": n, "block_size": blk, "nrhs": int(rhs.shape[0]), "tol": tol,
            "arms": results, "fastest_converged_low_precision": best,
            "best_speedup_vs_fp64": results[best]["speedup_vs_fp64"] if best else None,
            "fp64_meets_tol": results["fp64"]["backward_error"] <= tol}


def run_mixed(args):
    """The mixed-precision part alone on its own line: --matrix random (the
    n=40000 random indefinite matrix, block 256, 4 RHS) or spectral (n=20000,
    condition ~1e8, 16 RHS)."""
    import torch
    dev = torch.device("cuda", 0)
    torch.cuda.set_device(0)
    rand = args.matrix != "spectral"
    n = args.n if args.matrix != "kkt" else 40000
    if rand:
        a0, rhs = random_indefinite_device(n, args.seed, dev, args.nrhs)
        modes = ("fp32", "bf16x3", "bf16")
    else:
        a0, rhs = spectral_device(n, args.seed, dev)
        modes = ("fp32", "bf16x3")
    res = mixed_arms(a0, rhs, args.block, modes,
                     what=f"{matrix_description('random' if rand else 'spectral', n)}, block {args.block}, "
                          f"{rhs.shape[0]} RHS")
    line = {"metric": "time to backward error <= 1e-12, FP64 vs low-precision update + FP64 GMRES-IR",
            "unit": "ms", "higher_is_better": False, "n_gpus": 1, "dtype": "f64 (panel, residual) + update",
            "data": "synthetic: seeded, generated on the device", "config": {"workload": res["workload"]},
            "results": res}
    print(json.dumps(line), flush=True)


BATCH_METRIC = "batched factor+solve matrices/s (KKT, n ~ U[16,512], 1 RHS)"


def batched_sizes(count: int, seed: int) -> list:
    return [int(v) for v in np.random.default_rng(seed).integers(16, 513, size=count)]


def run_batched(args):
    """Config 4: `count` KKT matrices (H 75% of n, SPD; B Gaussian; zero (2,2)
    block), n ~ U[16, 512], one right-hand side each; FP64 and FP32 + FP64
    refinement; one persistent launch replayed from a CUDA graph.  Compared
    with looping the single-matrix path over a subset."""
    import torch
    import torch.distributed as dist

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    if world > 1:
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=300), device_id=dev)
    line = batched_results(args, world, rank, dev)
    if rank == 0:
        print(json.dumps(line), flush=True)
    if world > 1:
        dist.destroy_process_group()


def batched_results(args, world: int, rank: int, dev) -> dict:
    """The batched part (every rank its own batch; collectives only for the
    max over ranks when world > 1): the line's fields as a dict."""
    import ctypes

    import torch

    import blockedbunchkaufmanldlt_b200 as bbk
    from blockedbunchkaufmanldlt_b200 import tuning

    def max_over_ranks(v: float) -> float:
        return reduce_max_over_ranks(v, world, dev)

    seed = batch_seed(args.seed, rank)  # weak scaling: every rank owns its own batch
    sizes = batched_sizes(args.count, seed)
    table = tuning.load_table()
    plan = bbk.BatchedPlan(sizes, block_sizes=table)
    a0, x0 = tuning.kkt_batch_device(sizes, seed, dev)
    flops = sum(flops_ldlt(n) for n in sizes)
    dgemm = measure_dgemm_tflops(dev)
    L = bbk.lib()
    vp = ctypes.c_void_p
    a = torch.empty_like(a0)
    x = torch.empty_like(x0)
    perm = torch.empty(plan.vec_elements, dtype=torch.int32, device=dev)
    pt = torch.empty_like(perm)
    info = torch.zeros(plan.count * ctypes.sizeof(bbk.BatchInfo), dtype=torch.uint8, device=dev)

    def launch(mode, refine):
        bbk.check(L.bbk_batched_factor_solve(
            plan.count, vp(a.data_ptr()), vp(a0.data_ptr()) if refine else None, vp(x.data_ptr()),
            vp(perm.data_ptr()), vp(pt.data_ptr()), bbk.UPDATE_MODES[mode], 1e-12, 12 if refine else 0,
            vp(info.data_ptr()), vp(plan.workspace.data_ptr()), plan.bytes,
            vp(torch.cuda.current_stream().cuda_stream)))

    def graph_for(mode, refine, restore=True):
        s = torch.cuda.Stream()
        s.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(s):
            for _ in range(2):  # warm-up outside the graph (sets kernel attributes)
                a.copy_(a0)
                x.copy_(x0)
                launch(mode, refine)
        torch.cuda.current_stream().wait_stream(s)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            if restore:
                a.copy_(a0)
                x.copy_(x0)
            launch(mode, refine)
        return g

    def time_graph(g, steps, warmup):
        for _ in range(max(warmup, 0)):
            g.replay()
        torch.cuda.synchronize()
        if world > 1:
            dist.barrier()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(steps):
            g.replay()
        e1.record()
        torch.cuda.synchronize()
        if world > 1:
            dist.barrier()
        return max_over_ranks(e0.elapsed_time(e1) / steps)

    def accuracy():
        # backward error of every solution against the original matrix (device)
        worst = 0.0
        for k, n in enumerate(sizes):
            o, v = int(plan.a_offsets[k]), int(plan.rhs_offsets[k])
            m = a0[o:o + n * n].view(n, n)
            xs, bs = x[v:v + n], x0[v:v + n]
            r = bs - m @ xs
            den = m.abs().sum(1).max() * xs.abs().max() + bs.abs().max()
            worst = max(worst, float((r.abs().max() / den).item()))
        return worst

    results = {}
    sampler = ClockSampler(dev.index if dev.index is not None else 0)
    for mode, refine in (("fp64", False), ("fp32", True)):
        g_step = graph_for(mode, refine)
        g_kern = graph_for(mode, refine, restore=False)
        if mode == "fp64":
            sampler.start()
        ms_step = time_graph(g_step, args.steps, args.warmup)
        if mode == "fp64":
            clocks = sampler.stop()
        g_step.replay()  # leave fresh results for the accuracy check
        torch.cuda.synchronize()
        berr = accuracy()
        inf = np.frombuffer(info.cpu().numpy().tobytes(), dtype=np.dtype(
            [("iterations", "<i4"), ("converged", "<i4"), ("backward_error", "<f8")]))
        # kernel alone: factors from the last step are refactored in place, so
        # restore once and time a single launch per replay
        a.copy_(a0)
        x.copy_(x0)
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        kern = []
        for _ in range(max(2, min(args.steps, 5))):
            a.copy_(a0)
            x.copy_(x0)
            e0.record()
            g_kern.replay()
            e1.record()
            torch.cuda.synchronize()
            kern.append(e0.elapsed_time(e1))
        ms_kern = max_over_ranks(float(np.median(kern)))
        results[mode + ("+ir" if refine else "")] = {
            "ms_per_step": ms_step, "matrices_per_s": world * len(sizes) / (ms_step / 1e3),
            "kernel_ms": ms_kern, "kernel_matrices_per_s": world * len(sizes) / (ms_kern / 1e3),
            "gflops_kernel": world * flops / (ms_kern / 1e3) / 1e9,
            "max_backward_error": berr,
            "refine_iterations_max": int(inf["iterations"].max()) if refine else 0,
            "all_converged": bool(inf["converged"].all())}
        del g_step, g_kern

    # the baseline: the single-matrix path (factor + solve), looped over a subset
    sub = list(range(min(args.loop_sample, len(sizes))))
    nmax = max(sizes[k] for k in sub)
    bmax = int(max(plan.block_sizes[k] for k in sub))
    ws_f = torch.empty(max(bbk.factor_workspace_size(nmax, int(plan.block_sizes[k])) for k in sub),
                       dtype=torch.uint8, device=dev)
    ws_s = torch.empty(bbk.solve_workspace_size(nmax, 1), dtype=torch.uint8, device=dev)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    pe = torch.empty(nmax, dtype=torch.int32, device=dev)
    sp = vp(torch.cuda.current_stream().cuda_stream)

    def loop_once():
        for k in sub:
            n, o, v = sizes[k], int(plan.a_offsets[k]), int(plan.rhs_offsets[k])
            bk = int(plan.block_sizes[k])
            bbk.check(L.bbk_factor_device_async(n, bk, vp(a.data_ptr() + 8 * o), n, vp(perm.data_ptr() + 4 * v),
                                                vp(pt.data_ptr() + 4 * v), vp(pe.data_ptr()), 0,
                                                vp(ws_f.data_ptr()), ws_f.numel(), vp(status.data_ptr()), sp))
            bbk.check(L.bbk_solve_device(n, vp(a.data_ptr() + 8 * o), n, vp(perm.data_ptr() + 4 * v),
                                         vp(pt.data_ptr() + 4 * v), 1, vp(x.data_ptr() + 8 * v), n,
                                         vp(ws_s.data_ptr()), ws_s.numel(), sp))
    a.copy_(a0)
    x.copy_(x0)
    loop_once()
    torch.cuda.synchronize()
    a.copy_(a0)
    x.copy_(x0)
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    loop_once()
    e1.record()
    torch.cuda.synchronize()
    loop_ms = max(e0.elapsed_time(e1), (time.perf_counter() - t0) * 1e3)
    loop_rate = len(sub) / (loop_ms / 1e3)
    main = results["fp64"]
    line = {
        "metric": BATCH_METRIC, "value": main["matrices_per_s"], "unit": "matrices/s", "n_gpus": world,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": main["ms_per_step"],
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
        "data": "synthetic: seeded KKT matrices on the device (torch Gaussian generators)",
        "config": {"workload": f"batched factor+solve, {len(sizes)} KKT matrices per GPU, n ~ U[16,512] "
                               "(H 75% of n, SPD = G G^T/h + 1e-2 I; B Gaussian; zero (2,2) block), 1 RHS",
                   "count": len(sizes), "sum_n3_over_3": flops, "block_table": table or "library defaults",
                   "graph": "one CUDA graph per step: device copy restoring inputs + one persistent launch",
                   "l2": f"inputs ({8 * plan.a_elements / 1e9:.2f} GB) larger than L2; restored by a device "
                         "copy inside each step", "parallelism": f"replicas x{world} (own batch per GPU)"},
        "modes": results,
        "looped_single_matrix_path": {"matrices": len(sub), "ms": loop_ms, "matrices_per_s": loop_rate,
                                      "how": "bbk_factor_device_async + bbk_solve_device per matrix, same "
                                             "block sizes, one stream, no host sync between matrices"},
        "speedup_vs_looped": main["matrices_per_s"] / (world * loop_rate),
        "roofline": {"kernel": "batched_kernel", "bound": "tensor", "achieved": main["gflops_kernel"] / 1e3 / world,
                     "peak": dgemm, "unit": "TFLOP/s", "frac": main["gflops_kernel"] / 1e3 / world / dgemm,
                     "traffic": None, "peak_source": "cuBLAS DGEMM 8192^3 measured in this run (FP64 peak; "
                                                     "FP64 FMA and DMMA peaks are equal on B200)"},
        "clocks": clocks, "gpu_launches": 1,
    }
    return line


def run_reference_batched(args):
    """The reference's CPU factorization over a sample of the batch (each
    matrix with the block size the batched plan uses for it)."""
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    from blockedbunchkaufmanldlt_b200 import tuning
    lib, kind = _reference_lib()
    cores = lib.threads() if kind == "reference" else 1
    sizes = batched_sizes(args.count, args.seed)
    table = tuning.load_table() or [32, 32, 32, 32, 24, 12]
    buckets = [32, 64, 128, 256, 512, 1024]

    def block_for(n):
        for i, lim in enumerate(buckets):
            if n <= lim:
                return max(1, min(table[i], n))
        return table[-1]
    total_steps = max(1, args.steps) + max(0, args.warmup)
    budget = max(2.0, min(30.0, 150.0 / total_steps))
    rng = np.random.default_rng(args.seed)
    mats = []
    for n in sizes[:512]:
        h = max(1, int(round(0.75 * n)))
        mats.append((kkt_host(n, h, int(rng.integers(1 << 30))), block_for(n)))
    done, secs = 0, 0.0
    per_step = []
    for step in range(total_steps):
        t0 = time.perf_counter()
        cnt = 0
        while time.perf_counter() - t0 < budget:
            m, b = mats[(done + cnt) % len(mats)]
            lib.factor(m, b)
            cnt += 1
        dt = time.perf_counter() - t0
        if step >= args.warmup:
            per_step.append(cnt / dt)
        done += cnt
    value = float(np.mean(per_step))
    line = {"metric": BATCH_METRIC, "value": value, "unit": "matrices/s", "n_gpus": 1, "steps": len(per_step),
            "warmup": args.warmup, "ms_per_step": 1e3 * args.count / value, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f64", "impl": "reference",
            "data": "synthetic: seeded KKT matrices (numpy PCG64), the batch's size distribution",
            "config": {"workload": f"batched: {args.count} KKT matrices, n ~ U[16,512]", "count": args.count},
            "cpu_baseline": {"value": value, "unit": "matrices/s", "cores": cores, "kind": kind,
                             "sample": f"matrices of the batch's size distribution factored one after another "
                                       f"for {budget:.1f} s per step (ctor + Factorize(); the reference has no "
                                       "solve)"},
            "e2e": {"value": value, "unit": "matrices/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


def main():
    args = parse_args()
    if args.impl == "reference" and args.workload == "batched":
        run_reference_batched(args)
    elif args.impl == "reference":
        run_reference(args)
    elif args.workload == "batched":
        run_batched(args)
    elif args.workload == "mixed":
        run_mixed(args)
    else:
        run_main(args)


if __name__ == "__main__":
    main()
