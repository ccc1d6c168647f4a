"""Benchmark: plane-wave H.psi band-applications/s on one GB300 (mixed and FP64).

Workload (default ``si64``): 64-atom Si cube, side 20.52 bohr, Ecut 20 Ha
(37,073 plane waves), 96^3 FFT grid, Gamma point, 160 bands applied in blocks of
32, 256 projectors (s + p on every atom).  One step = H.psi (kinetic + local
potential + nonlocal) on all 160 bands in one public C-ABI call
(qgb_hamiltonian_mixed / qgb_hamiltonian), as the reference's Davidson calls
Electrons.hamiltonian on all its bands: the local potential runs in FFT blocks
of 32 bands (the plane workspace holds 32 bands), the nonlocal term over all
160 at once (one <beta|psi> and one back-projection, as the reference's
beta @ (D_all @ beta_C)).  Inputs are seeded synthetic data of that shape
(qimpy_gb300.workloads), resident in HBM before the timed region.  The
local-potential / nonlocal breakdown is timed per 32-band block in a separate
loop with the two stages launched apart on one stream.

Precision forms:
  mixed - complex64 wavefunctions, FP32 FFTs, projector GEMMs on the tcgen05
          tensor cores as split-BF16x3 with FP32 accumulation (the headline `value`)
  fp64  - complex128 throughout, the plain drop-in form (reported in `fp64`)

Timing: W warm-up steps, then K steps, each bracketed by CUDA events on the
launching stream with a 512 MB L2 flush between steps (outside the events);
N > 1 GPUs (torchrun) run independent replicas ("replicas only": H.psi has no
exchange step), value = bands of all ranks / max-over-ranks time.

`--impl reference` times the CPU oracle (the reference's FP64 algorithm restated
with numpy/scipy, all host threads) on a bounded band sample of the same
workload and prints the same metric.
"""
from __future__ import annotations

import argparse
import ctypes as ct
import json
import os
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "H.psi band-applications/s"
UNIT = "band-applications/s"


def parse_args():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="gb300", choices=["gb300", "reference"])
    ap.add_argument("--workload", default="si64")
    ap.add_argument("--cpu-sample-bands", type=int, default=32, help="bands of the CPU baseline's sample block")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--eig-reps", type=int, default=3)
    ap.add_argument("--forms", default="fp64,mixed", help="precision forms to run (profiling aid)")
    ap.add_argument("--plane-budget-mb", type=int, default=0, help="slab-plane workspace cap (0 = default)")
    ap.add_argument("--batch", type=int, default=256, help="instances of the batched workload (0 = skip)")
    ap.add_argument("--batch-chunk-mb", type=int, default=0,
                    help="slab-plane MB per batched launch chunk (0 = one chunk per grid shape)")
    ap.add_argument("--serve", type=int, default=16,
                    help="requests of the serving stream sample, the same for both forms (0 = skip)")
    ap.add_argument("--serve-wall", type=float, default=150.0, help="wall-clock cap per serving run (s)")
    ap.add_argument("--no-eigensolve", action="store_true")
    ap.add_argument("--profile-davidson", action="store_true",
                    help="print torch.profiler kernel tables of Davidson solves (si2, si64) instead of the bench line")
    ap.add_argument("--autotune", action="store_true",
                    help="autotuned FFT factorisation for si64 (measured equal to the default within noise)")
    return ap.parse_args()


# ---------------------------------------------------------------------------
# Distributed plumbing (replicas only)
# ---------------------------------------------------------------------------


def dist_init():
    import torch

    ws = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if ws > 1:
        import torch.distributed as dist

        backend = os.environ.get("QGB_DIST_BACKEND", "nccl")  # gloo: CPU tests of the replica plumbing
        if backend == "nccl":
            torch.cuda.set_device(local)
        dist.init_process_group(backend)
    return rank, ws, local


def dist_max(x: float, ws: int) -> float:
    """Maximum of a host scalar over ranks (the slowest replica's time)."""
    if ws == 1:
        return x
    import torch
    import torch.distributed as dist

    dev = "cuda" if dist.get_backend() == "nccl" else "cpu"
    t = torch.tensor([x], dtype=torch.float64, device=dev)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def replica_value(units_per_rank: float, max_seconds: float, ws: int) -> float:
    """Whole-job throughput of `ws` independent replicas: the units of all ranks
    over the max-over-ranks time (from dist_max)."""
    return units_per_rank * ws / max_seconds


def dist_barrier(ws: int):
    if ws > 1:
        import torch.distributed as dist

        dist.barrier()


# ---------------------------------------------------------------------------
# Clock sampling during the timed region
# ---------------------------------------------------------------------------


class ClockSampler:
    """SM clock, power and clock-event reasons sampled every millisecond through
    NVML (read-only queries) in a background thread, so that even a timed region
    of a few tens of milliseconds gets samples.  Falls back to `nvidia-smi -lms`
    where NVML cannot be loaded."""

    # nvmlClocksEventReason* bits (nvml.h)
    REASONS = {0x4: "sw_power_cap", 0x8: "hw_slowdown", 0x20: "sw_thermal_slowdown", 0x40: "hw_thermal_slowdown",
               0x80: "hw_power_brake_slowdown"}

    def __init__(self, index: int):
        self.index = index
        self.samples: list = []
        self._stop = threading.Event()
        self._nvml = None
        self._handle = None
        self._smi = None

    def _open_nvml(self):
        import torch

        lib = ct.CDLL("libnvidia-ml.so.1")
        if lib.nvmlInit_v2() != 0:
            raise OSError("nvmlInit failed")
        h = ct.c_void_p()
        props = torch.cuda.get_device_properties(self.index)
        bus = None
        if all(hasattr(props, a) for a in ("pci_domain_id", "pci_bus_id", "pci_device_id")):
            bus = f"{props.pci_domain_id:08x}:{props.pci_bus_id:02x}:{props.pci_device_id:02x}.0"
        if bus is None or lib.nvmlDeviceGetHandleByPciBusId_v2(bus.encode(), ct.byref(h)) != 0:
            if lib.nvmlDeviceGetHandleByIndex_v2(self.index, ct.byref(h)) != 0:
                raise OSError("no NVML handle")
        self._nvml, self._handle = lib, h
        self._reasons_fn = None
        for name in ("nvmlDeviceGetCurrentClocksEventReasons", "nvmlDeviceGetCurrentClocksThrottleReasons"):
            try:
                self._reasons_fn = getattr(lib, name)
                break
            except AttributeError:
                continue

    def _sample_nvml(self):
        lib, h = self._nvml, self._handle
        sm, smax, pw, rs = ct.c_uint(), ct.c_uint(), ct.c_uint(), ct.c_ulonglong()
        while not self._stop.is_set():
            ok = lib.nvmlDeviceGetClockInfo(h, 1, ct.byref(sm)) == 0  # NVML_CLOCK_SM
            lib.nvmlDeviceGetMaxClockInfo(h, 1, ct.byref(smax))
            lib.nvmlDeviceGetPowerUsage(h, ct.byref(pw))
            if self._reasons_fn is not None:
                self._reasons_fn(h, ct.byref(rs))
            if ok:
                self.samples.append((sm.value, smax.value, pw.value / 1000.0, rs.value))
            time.sleep(0.001)

    def start(self):
        try:
            self._open_nvml()
            self._t = threading.Thread(target=self._sample_nvml, daemon=True)
            self._t.start()
        except (OSError, AttributeError):
            self._nvml = None
            try:
                self._smi = subprocess.Popen(
                    ["nvidia-smi", "-i", str(self.index), "--query-gpu=clocks.sm,clocks.max.sm,power.draw",
                     "--format=csv,noheader,nounits", "-lms", "100"], stdout=subprocess.PIPE,
                    stderr=subprocess.DEVNULL, text=True)
                self._t = threading.Thread(target=self._read_smi, daemon=True)
                self._t.start()
            except OSError:
                self._smi = None

    def _read_smi(self):
        for line in self._smi.stdout:
            parts = [x.strip() for x in line.split(",")]
            try:
                self.samples.append((float(parts[0]), float(parts[1]), float(parts[2]), 0))
            except (ValueError, IndexError):
                continue

    def stop(self) -> dict:
        self._stop.set()
        if self._smi is not None:
            self._smi.terminate()
            try:
                self._smi.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self._smi.kill()
        if getattr(self, "_t", None) is not None:
            self._t.join(timeout=5)
        if not self.samples:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["no clock samples"], "samples": 0}
        sm = [x[0] for x in self.samples]
        reasons = sorted({name for x in self.samples for bit, name in self.REASONS.items() if x[3] & bit})
        return {"sm_mhz": float(np.median(sm)), "sm_max_mhz": float(max(x[1] for x in self.samples)),
                "sm_min_mhz": float(min(sm)), "power_w_median": float(np.median([x[2] for x in self.samples])),
                "reasons": reasons, "samples": len(sm), "source": "nvml" if self._nvml is not None else "nvidia-smi"}


# ---------------------------------------------------------------------------
# Workload
# ---------------------------------------------------------------------------


def make_workload(name: str):
    from qimpy_gb300 import workloads as wl

    p = wl.get(name)
    b = wl.make_basis(p.Gbasis, p.k, p.ke_cutoff, p.grid_shape)
    beta = wl.make_projectors(p, b)
    nb = p.n_bands
    C = wl.make_wavefunctions(p, b, nb)
    return p, b, beta, C


def workload_config(args, ws: int) -> dict:
    """The `config` of the JSON line (the same for both arms)."""
    names = {"si64": "64-atom Si, 96^3 grid, n=37073, Gamma, 160 bands in blocks of 32, P=256"}
    return {"workload": f"{args.workload}: {names.get(args.workload, 'see qimpy_gb300.workloads')}",
            "l2": "flushed (512 MB write) between timed steps", "parallelism": f"replicas x{ws}"}


def roofline_counts(p, b, tables, nb_tile: int, real_bytes: int):
    """Algorithmic bytes and flops per band-application: local 2*5 N log2 N + 2N + 2n
    flops and 2 n s_c + (N s_r + 4 n) / B_tile bytes (psi in, H psi out, V and the
    sphere index shared by the B_tile bands of a block); nonlocal 2*8 P n + 8 P p_atom
    flops and 2 n s_c + 2 P n s_c / B_tile bytes (beta read for both GEMMs)."""
    N = int(np.prod(p.grid_shape))
    n = float(b.n.mean())
    P = p.n_projectors
    s_c = 2 * real_bytes
    log2N = np.log2(N)
    flops_loc = 2 * 5 * N * log2N + 2 * N + 2 * n
    flops_nl = 2 * 8 * P * n + 8 * P * p.p_atom
    bytes_loc = 2 * n * s_c + (N * real_bytes + n * 4) / nb_tile
    bytes_nl = 2 * n * s_c + 2 * P * n * s_c / nb_tile
    return dict(flops_loc=flops_loc, flops_nl=flops_nl, bytes_loc=bytes_loc, bytes_nl=bytes_nl)


# DRAM bytes (read + write) per 32-band si64 block, from ncu captures of the
# mixed form (default cache control: caches flushed before every kernel, so planes
# one kernel writes and the next reads count as DRAM traffic although they stay in
# L2 in a timed run).  Recorded constants of those captures
# (profiles/ncu_si64_block.md), not measured by this run: k_ifft_yz, k_xpass and
# k_fft_yz_gather, and the five kernels of the nonlocal chain in its store form.
NCU_DRAM_BYTES_PER_BLOCK = {"local": 296.1e6, "nonlocal": 176.6e6}

#: Reference H.psi time over the torch port's (oracle/hpsi_torch.py), si64 by
#: band count, both on all 8 cores of one x86 host (tests/golden/time_reference_vs_port.py).
#: The reference's source is not installed where the bench runs, so its CPU
#: baseline is the port.  (The numpy port, oracle.hpsi, took 1.7x, 1.9x and
#: 3.3x the reference's time at 2, 8 and 32 bands; the torch port matches it.)
REFERENCE_OVER_PORT = {"2": 0.78, "8": 1.03, "32": 1.09, "host": "8-core x86 container, torch 2.11 CPU"}


def local_roofline(rc, band_apps, t_loc, hbm_peak, peaks) -> dict:
    """Roofline of the local-potential apply (three launches in one C-ABI call,
    one 32-band block): achieved = algorithmic bytes / CUDA-event time against
    the measured HBM copy bandwidth, with the measured DRAM traffic beside it;
    the bound that binds is the FP32 CUDA-core pipe (5 N log2 N flops per FFT at
    ~300 flop per compulsory byte), reported as `pipe`."""
    ach_gbs = rc["bytes_loc"] * band_apps / t_loc / 1e9
    ach_tflops = rc["flops_loc"] * band_apps / t_loc / 1e12
    traffic = NCU_DRAM_BYTES_PER_BLOCK["local"]
    t_lb = max(rc["bytes_loc"] * band_apps / (hbm_peak * 1e9), rc["flops_loc"] * band_apps / (peaks["fp32"] * 1e12))
    return {"kernel": "local potential: k_ifft_yz + k_xpass + k_fft_yz_gather, one 32-band block, FP32",
            "bound": "hbm", "achieved": ach_gbs, "peak": hbm_peak, "unit": "GB/s", "frac": ach_gbs / hbm_peak,
            "peak_source": "measured (MEASURED_PEAKS.json hbm_gbs)", "traffic": traffic,
            "traffic_source": "constant: one cold-cache ncu capture of a 32-band block",
            "dram_gbs_from_traffic": traffic / t_loc / 1e9 if traffic else None,
            "binding": "fp32 CUDA-core pipe",
            "pipe": {"achieved_tflops": ach_tflops, "peak_tflops": peaks["fp32"], "frac": ach_tflops / peaks["fp32"],
                     "peak_source": "measured FMA burn (qgb_fma_burn)"},
            "lower_bound_over_measured": t_lb / t_loc, "seconds_per_launch_group": t_loc}


def nonlocal_roofline(rc, band_apps, t_nl, hbm_peak, bf16_peak) -> dict:
    """Tensor-core nonlocal chain (split, <beta|psi> GEMM, reduce, D, back-projection
    GEMM) for one 32-band block: algorithmic complex flops (2 * 8 P n per band)
    against the bf16 tensor peak, counting the 3 bf16 products of split-BF16x3
    and the 4 real products of a complex MAC as issued MMA work."""
    flops = rc["flops_nl"] * band_apps
    issued = 3.0 * flops  # split-BF16x3: hi*hi + hi*lo + lo*hi
    traffic = NCU_DRAM_BYTES_PER_BLOCK["nonlocal"]
    return {"bound": "hbm" if rc["bytes_nl"] / hbm_peak > rc["flops_nl"] * 3 / (bf16_peak * 1e3) else "tensor",
            "achieved_tflops": flops / t_nl / 1e12, "issued_mma_tflops": issued / t_nl / 1e12,
            "peak_tflops": bf16_peak, "frac_issued": issued / t_nl / 1e12 / bf16_peak,
            "achieved_gbs": rc["bytes_nl"] * band_apps / t_nl / 1e9, "hbm_frac": rc["bytes_nl"] * band_apps / t_nl / 1e9 / hbm_peak,
            "traffic": traffic, "traffic_source": "constant: one cold-cache ncu capture of a 32-band block",
            "dram_gbs_from_traffic": traffic / t_nl / 1e9 if traffic else None,
            "seconds_per_block": t_nl}


def measure_fma_peak(dtype_code: int) -> float:
    """FP64 / FP32 CUDA-core FMA peak in TFLOP/s (best of 5)."""
    import torch

    from qimpy_gb300 import _lib

    lib = _lib.aux()
    blocks, threads, iters = 152 * 8, 256, 4096
    out = torch.empty(blocks, dtype=torch.float64, device="cuda")
    st = torch.cuda.current_stream()
    best = 0.0
    for _ in range(6):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(st)
        _lib.check(lib.qgb_fma_burn(dtype_code, blocks, threads, iters, out.data_ptr(), st.cuda_stream), "fma")
        e1.record(st)
        e1.synchronize()
        sec = e0.elapsed_time(e1) * 1e-3
        best = max(best, blocks * threads * iters * 128 / sec / 1e12)
    return best


def run_gb300(args, rank, ws, local):
    import torch

    from qimpy_gb300 import _lib, ops, sphere as sp

    dev = torch.device(f"cuda:{local}")
    torch.cuda.set_device(dev)
    p, b, beta_np, C_np = make_workload(args.workload)
    tables = sp.build_tables(b.fft_index, b.n, p.grid_shape)
    nb = C_np.shape[1]
    block = p.block_size or nb
    blocks = [(s, min(s + block, nb)) for s in range(0, nb, block)]
    flush = torch.empty(512 * 1024 * 1024 // 4, dtype=torch.float32, device=dev)
    results = {}
    forms = [f for f in (("fp64", torch.complex128), ("mixed", torch.complex64)) if f[0] in args.forms.split(",")]
    from qimpy_gb300 import autotune

    for form, cdt in forms:
        ds = sp.DeviceSphere(tables, b.ke, dev, cdt)
        ds.set_potential(torch.from_numpy(p.V_r))
        # Optionally the autotuner's FFT radix schedule (tuned outside the measured
        # region); the batched workload always uses it.
        fac = autotune.tune_shape(p.grid_shape, cdt, dev, nb=block, reps=5) if args.autotune else None
        if fac is not None:
            ds.set_factors(fac)
        C = torch.from_numpy(C_np).to(dev, cdt)
        beta = torch.from_numpy(beta_np).to(dev, cdt)
        D = torch.from_numpy(p.D_atom).to(dev, cdt)
        HC = torch.empty_like(C)
        projT = torch.empty((p.nk, block, p.n_projectors), dtype=cdt, device=dev)
        projT_all = torch.empty((p.nk, nb, p.n_projectors), dtype=cdt, device=dev)
        work = torch.empty_like(projT)
        # Slab planes for one FFT block of bands: the one call over all bands
        # then runs the local potential block by block, each block's planes in L2.
        ds.plane_budget_bytes = (args.plane_budget_mb << 20) if args.plane_budget_mb else ds.workspace_bytes(1) * block
        wsp = ops.workspace(ds.workspace_bytes(block), dev)
        mixed = cdt == torch.complex64
        if mixed:  # tensor-core nonlocal: projector operands split once per basis
            split = ops.beta_split(beta)
            ws_nl = ops.workspace(int(_lib.lib().qgb_nonlocal_tc_workspace_bytes(p.nk, p.n_projectors, block,
                                                                                 b.n_tot)), dev)
            ws_ham = ops.workspace(ds.hamiltonian_mixed_workspace_bytes(nb, p.n_projectors), dev)
        st = torch.cuda.current_stream()

        C_blk = [C[:, s0:s1].contiguous() for (s0, s1) in blocks]
        H_blk = [torch.empty_like(c) for c in C_blk]

        def step(ev=None):
            for j, (s0, s1) in enumerate(blocks):
                Cb, Hb = C_blk[j], H_blk[j]
                if ev is not None:
                    ev[0].record(st)
                ops.apply_potential(ds, Cb, out=Hb, add_ke=True, ws=wsp)
                if ev is not None:
                    ev[1].record(st)
                pT = projT[:, : s1 - s0]
                if mixed:
                    ops.apply_nonlocal_tc(split, D, Cb, Hb, pT, ws_nl)
                else:
                    ops.project(beta, Cb, pT)
                    ops.apply_nonlocal(beta, D, pT, Hb, work[:, : s1 - s0])
                if ev is not None:
                    ev[2].record(st)
                    ev = ev[3:]

        # The timed step: H.psi of all bands through one public C-ABI call
        # (qgb_hamiltonian_mixed / qgb_hamiltonian), buffers and workspaces preallocated.
        if not mixed:
            ws_ham = ops.workspace(ds.hamiltonian_workspace_bytes(nb, p.n_projectors), dev)

        def hamiltonian(Cin, Hout):
            if mixed:
                ops.hamiltonian_mixed(ds, Cin, split, D, out=Hout, projT=projT_all, ws=ws_ham)
            else:
                ops.hamiltonian(ds, Cin, beta, D, out=Hout, projT=projT_all, ws=ws_ham)

        # Device-resident inputs: the mixed form is fastest as one call over all
        # bands (its nonlocal term then streams beta twice per step, hidden beside
        # the first FFT block); the FP64 form, bound by the FP64 pipe, is fastest
        # block by block (measured: 3.94k against 3.49k band-applications/s).
        one_call = mixed
        H_out = [torch.empty_like(c) for c in C_blk]

        def fused_step():
            if one_call:
                hamiltonian(C, HC)
                return
            for j, (s0, s1) in enumerate(blocks):
                if mixed:
                    ops.hamiltonian_mixed(ds, C_blk[j], split, D, out=H_out[j], projT=projT[:, : s1 - s0],
                                          ws=ws_ham)
                else:
                    ops.hamiltonian(ds, C_blk[j], beta, D, out=H_out[j], projT=projT[:, : s1 - s0], ws=ws_ham)

        for _ in range(args.warmup):
            step()
            fused_step()
        torch.cuda.synchronize()
        # Stage breakdown (local potential and nonlocal term timed apart, one stream).
        t_loc, t_nl = [], []
        for _ in range(args.steps):
            flush.zero_()
            evs = [torch.cuda.Event(enable_timing=True) for _ in range(3 * len(blocks))]
            step(evs)
            torch.cuda.synchronize()
            for j in range(len(blocks)):
                t_loc.append(evs[3 * j].elapsed_time(evs[3 * j + 1]) * 1e-3)
                t_nl.append(evs[3 * j + 1].elapsed_time(evs[3 * j + 2]) * 1e-3)
        dist_barrier(ws)
        clock = ClockSampler(local)
        clock.start()
        times = []
        for _ in range(args.steps):
            flush.zero_()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record(st)
            fused_step()
            e1.record(st)
            torch.cuda.synchronize()
            times.append(e0.elapsed_time(e1) * 1e-3)
        clocks = clock.stop()
        if not one_call:
            HC = torch.cat(H_out, dim=1)
        # The block-by-block stage form computes the same H.psi.
        res_blocks = float((torch.cat(H_blk, dim=1) - HC).abs().max() / HC.abs().max())
        dist_barrier(ws)
        total = dist_max(float(np.sum(times)), ws)
        res = dict(value=replica_value(nb * p.nk * args.steps, total, ws), ms_per_step=1e3 * total / args.steps,
                   t_loc_block=float(np.median(t_loc)), t_nl_block=float(np.median(t_nl)),
                   clocks=clocks, stage_form_rel_diff=res_blocks,
                   call_form=(f"one call over {nb} bands (FFT blocks of {block})" if one_call
                              else f"{len(blocks)} calls of {block} bands"))
        # End-to-end through the public API with host buffers (pinned), every step:
        # each block's host->device copy, its qgb_hamiltonian(_mixed) call and its
        # device->host copy, pipelined over the blocks on an upload stream, the
        # compute stream and a download stream (a host-side caller streams blocks;
        # one call over all bands would have to wait for every band's upload).
        if not args.no_e2e:
            Ch_blk = [torch.from_numpy(np.ascontiguousarray(C_np[:, s0:s1])).to(cdt).pin_memory() for (s0, s1) in blocks]
            Hh_blk = [torch.empty_like(c).pin_memory() for c in Ch_blk]
            Cd_blk = [torch.empty_like(c, device=dev) for c in Ch_blk]
            Hd_blk = [torch.empty_like(c) for c in Cd_blk]
            up, down = torch.cuda.Stream(device=dev), torch.cuda.Stream(device=dev)
            ev_in = [torch.cuda.Event() for _ in blocks]
            ev_out = [torch.cuda.Event() for _ in blocks]
            ws_e2e = ops.workspace(ds.hamiltonian_mixed_workspace_bytes(block, p.n_projectors) if mixed
                                   else ds.hamiltonian_workspace_bytes(block, p.n_projectors), dev)

            def e2e_step():
                up.wait_stream(st)
                for j in range(len(blocks)):
                    with torch.cuda.stream(up):
                        Cd_blk[j].copy_(Ch_blk[j], non_blocking=True)
                    ev_in[j].record(up)
                for j in range(len(blocks)):
                    st.wait_event(ev_in[j])
                    pT = projT[:, : blocks[j][1] - blocks[j][0]]
                    if mixed:
                        ops.hamiltonian_mixed(ds, Cd_blk[j], split, D, out=Hd_blk[j], projT=pT, ws=ws_e2e)
                    else:
                        ops.hamiltonian(ds, Cd_blk[j], beta, D, out=Hd_blk[j], projT=pT, ws=ws_e2e)
                    ev_out[j].record(st)
                for j in range(len(blocks)):
                    down.wait_event(ev_out[j])
                    with torch.cuda.stream(down):
                        Hh_blk[j].copy_(Hd_blk[j], non_blocking=True)
                st.wait_stream(down)
            for _ in range(max(1, args.warmup)):
                e2e_step()
            torch.cuda.synchronize()
            e2e_times = []
            for _ in range(args.steps):
                flush.zero_()
                e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                e0.record(st)
                e2e_step()
                e1.record(st)
                torch.cuda.synchronize()
                e2e_times.append(e0.elapsed_time(e1) * 1e-3)
            tot = dist_max(float(np.sum(e2e_times)), ws)
            nbytes = sum(c.numel() * c.element_size() for c in Ch_blk)
            res["e2e"] = dict(value=replica_value(nb * p.nk * args.steps, tot, ws), unit=UNIT, h2d_bytes_per_step=nbytes,
                              d2h_bytes_per_step=nbytes, call_form=f"{len(blocks)} calls of {block} bands, copies pipelined")
            Hh = torch.cat(Hh_blk, dim=1)
            err = float((Hh.to(dev) - HC).abs().max() / HC.abs().max())
            res["e2e_matches_device_result"] = err
        # our kernels per step: 3 local-potential kernels per FFT block, plus the
        # nonlocal term once per call: 5 tensor-core chain kernels (mixed), or slices
        # and digit GEMMs of 3 panels, their sum, D, the projectors' scales, D proj's
        # slices, and slices and GEMMs of 2 panels (FP64)
        res["launches_per_step"] = 3 * len(blocks) + (5 if mixed else 14) * (1 if one_call else len(blocks))
        res["nonlocal_error_word"] = int(ops.device_error_word(dev).item()) if mixed else 0
        res["real_bytes"] = 8 if cdt == torch.complex128 else 4
        res["fft_schedule"] = [list(f) for f in ds.tables.fac]
        res["block"] = block
        results[form] = res
        del ds, C, beta, HC, wsp
        torch.cuda.empty_cache()
    peaks = {"fp64": measure_fma_peak(_lib.QGB_F64), "fp32": measure_fma_peak(_lib.QGB_F32)}
    return p, b, tables, results, peaks


def run_eigensolves(args, local):
    """Eigensolves/s on si2 (Si primitive cell, 8 k, 16 bands), FP64 and mixed,
    with both of the reference's eigensolvers.

    One eigensolve = Davidson (or CheFSI: Davidson warm-up to 0.1 Ha, then
    Chebyshev filters of order 8) from the seeded start vectors to
    max |d eig| < 1e-11 (Davidson FP64) / 1e-10 (CheFSI FP64) / 1e-6 (mixed,
    then FP64 refinement sweeps), every k-point, timed end to end with CUDA
    events (host syncs per iteration included).  Eigenvalue errors are against
    the reference's own FP64 eigenvalues (its Davidson, and its CheFSI run on the
    same inputs)."""
    import torch

    from qimpy_gb300 import chefsi as cf, davidson as dv, electrons as E, workloads as wl

    dev = torch.device(f"cuda:{local}")
    p = wl.get("si2")
    gold = np.load(os.path.join(ROOT, "tests", "golden", "si2.npz"))
    gold_cf = np.load(os.path.join(ROOT, "tests", "golden", "chefsi_si2.npz"))
    el64, C0 = E.from_problem(p, dev, torch.complex128)
    el32, _ = E.from_problem(p, dev, torch.complex64)
    out = {"chefsi": {}}
    runs = [("davidson", "fp64", el64, 1e-11), ("davidson", "mixed", el32, 1e-6),
            ("chefsi", "fp64", el64, float(gold_cf["eig_threshold"])), ("chefsi", "mixed", el32, 1e-6)]
    for solver, form, el, thr in runs:
        times, stats = [], None
        for rep in range(1 + max(1, args.eig_reps)):
            el.C = E.Wavefunction(el.basis, coeff=C0.to(dev, el.basis.dtype)).orthonormalize()
            torch.cuda.synchronize()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            el.deig_max = np.inf
            if solver == "davidson":
                stats = dv.Davidson(el, n_iterations=300, eig_threshold=thr)()
            else:
                stats = cf.CheFSI(el, n_iterations=100, eig_threshold=thr, filter_order=int(gold_cf["filter_order"]),
                                  init_threshold=float(gold_cf["init_threshold"]))()
            eig = el.eig
            if form == "mixed":
                eig, _ = dv.refine_fp64(el, el64)
            e1.record()
            torch.cuda.synchronize()
            if rep:  # first solve is warm-up
                times.append(e0.elapsed_time(e1) * 1e-3)
        e = eig.cpu().numpy()[:, : p.n_bands]
        res = dict(eigensolves_per_s=1.0 / float(np.median(times)), seconds=float(np.median(times)),
                   p50_s=float(np.percentile(times, 50)), p99_s=float(np.percentile(times, 99)),
                   iterations=stats.iterations, converged=stats.converged, stalled=stats.stalled,
                   hpsi_bands=stats.hpsi_bands,
                   max_eig_error_ha_vs_reference=float(np.abs(e - gold["eig"][:, : p.n_bands]).max()))
        if solver == "chefsi":
            res["max_eig_error_ha_vs_reference_chefsi"] = float(np.abs(e - gold_cf["eig"][:, : p.n_bands]).max())
            out["chefsi"][form] = res
        else:
            out[form] = res
    return out


def run_eigensolve_si64(args, local):
    """Davidson eigensolve of the 64-atom Si cell (96^3, Gamma, n = 37073,
    160 + 16 bands, P = 256), FP64 and mixed, one solve each from the seeded
    start vectors.  FP64: to max |d eig| < 1e-9 Ha (the reference's run);
    mixed: FP32 H.psi and subspace products to the FP32 floor (or 1e-6 Ha),
    then FP64 Rayleigh-Ritz refinement sweeps to 1e-9 Ha.  Errors are against
    the reference's own converged eigenvalues, the mixed one before and after
    the refinement; times by CUDA events, host syncs included."""
    import torch

    from qimpy_gb300 import davidson as dv, electrons as E, workloads as wl

    dev = torch.device(f"cuda:{local}")
    p = wl.get("si64")
    gold = np.load(os.path.join(ROOT, "tests", "golden", "si64.npz"))
    ref = gold["eig"][:, : p.n_bands]
    out = {"workload": "si64: 160 + 16 bands, eig_threshold 1e-9 Ha, one solve per form",
           "reference_cpu_seconds": float(gold["davidson_seconds"]),
           "reference_iterations": int(gold["davidson_iterations"])}
    el64, C0 = E.from_problem(p, dev, torch.complex128)
    for form in ("fp64", "mixed"):
        el = el64 if form == "fp64" else E.from_problem(p, dev, torch.complex64)[0]
        el.C = E.Wavefunction(el.basis, coeff=C0.to(dev, el.basis.dtype)).orthonormalize()
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        stats = dv.Davidson(el, n_iterations=300, eig_threshold=1e-9 if form == "fp64" else 1e-6)()
        res = dict(iterations=stats.iterations, converged=stats.converged, stalled=stats.stalled)
        if form == "mixed":
            res["max_eig_error_ha_before_refinement"] = float(np.abs(el.eig.cpu().numpy()[:, : p.n_bands] - ref).max())
            eig, _ = dv.refine_fp64(el, el64, eig_threshold=1e-9, max_sweeps=150)
            res["refinement_sweeps"] = el64.last_refine.iterations
        else:
            eig = el.eig
        e1.record()
        torch.cuda.synchronize()
        sec = e0.elapsed_time(e1) * 1e-3
        res.update(seconds=sec, eigensolves_per_s=1.0 / sec,
                   max_eig_error_ha_vs_reference=float(np.abs(eig.cpu().numpy()[:, : p.n_bands] - ref).max()))
        out[form] = res
        del el
        torch.cuda.empty_cache()
    out["mixed_over_fp64"] = out["fp64"]["seconds"] / out["mixed"]["seconds"]
    out["fp64_over_reference_cpu"] = out["reference_cpu_seconds"] / out["fp64"]["seconds"]
    return out


def run_real_hpsi(args, local):
    """H.psi of real (Gamma-point) wavefunctions on the half basis of the
    64-atom Si cell (96^3, n_half = 18,561 of the 37,073-point sphere,
    P = 256), 160 bands in blocks of 32, FP64 (qgb_hamiltonian_real) and mixed
    (qgb_hamiltonian_real_mixed: FP32 local potential, tensor-core nonlocal);
    two real bands per complex transform.  Same timing
    rules as the headline: CUDA events per step, 512 MB L2 flush between steps."""
    import torch

    import ctypes as ct

    from qimpy_gb300 import _lib, ops, real_basis as rbm, workloads as wl

    dev = torch.device(f"cuda:{local}")
    p = wl.get("si64")
    half, full = rbm.gamma_bases(p.Gbasis, p.ke_cutoff, p.grid_shape)
    beta_np = wl.make_projectors(p, half)
    nb, block = p.n_bands, p.block_size or p.n_bands
    C_np = wl.make_wavefunctions(p, half, nb)
    flush = torch.empty(512 * 1024 * 1024 // 4, dtype=torch.float32, device=dev)
    out = {"workload": f"si64 Gamma, real wavefunctions: n_half {int(half.n[0])}, {nb} bands in blocks of {block}"}
    for form, cdt in (("fp64", torch.complex128), ("mixed", torch.complex64)):
        rb = rbm.DeviceRealBasis(half, full, dev, cdt)
        rb.set_potential(torch.from_numpy(p.V_r))
        C = torch.from_numpy(C_np).to(dev, cdt)
        beta = torch.from_numpy(beta_np).to(dev, cdt)
        D = torch.from_numpy(p.D_atom).to(dev, cdt)
        blocks = [C[:, s:s + block].contiguous() for s in range(0, nb, block)]
        outs = [torch.empty_like(c) for c in blocks]
        P = beta.shape[1]
        projT = torch.empty((1, block, P), dtype=cdt, device=dev)
        mixed = cdt == torch.complex64
        if mixed:  # tensor-core nonlocal (qgb_hamiltonian_real_mixed)
            split = ops.beta_split(beta)
            ws = ops.workspace(_lib.lib().qgb_hamiltonian_real_mixed_workspace_bytes(
                ct.byref(rb.sphere.struct), ct.byref(rb.struct), block, P), dev)
        else:
            ws = ops.workspace(rb.workspace_bytes(block, P), dev)

        def step():
            for c, o in zip(blocks, outs):
                if mixed:
                    ops.hamiltonian_real_mixed(rb, c, split, D, out=o, projT=projT[:, : c.shape[1]], ws=ws)
                else:
                    ops.hamiltonian_real(rb, c, beta, D, out=o, projT=projT[:, : c.shape[1]], ws=ws)

        for _ in range(args.warmup):
            step()
        torch.cuda.synchronize()
        times = []
        for _ in range(args.steps):
            flush.zero_()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            step()
            e1.record()
            torch.cuda.synchronize()
            times.append(e0.elapsed_time(e1) * 1e-3)
        t = float(np.sum(times))
        out[form] = {"value": nb * args.steps / t, "unit": UNIT, "ms_per_step": 1e3 * t / args.steps}
        del rb, C, beta, blocks, outs, ws
        torch.cuda.empty_cache()
    out["mixed_over_fp64"] = out["mixed"]["value"] / out["fp64"]["value"]
    return out


def run_batch(args, local):
    """Batched uneven instances: `args.batch` independent problems (cubic sides
    10/14/18/22 bohr, 2-16 atoms, Ecut 15-25 Ha, 8-64 bands, 1-8 k-points),
    FP32 H.psi with the tensor-core nonlocal term, FFT radix schedule per grid
    from the autotuner, the whole batched H.psi captured in one CUDA graph and
    replayed.  Reference point: the same instances applied one after another
    with the single-problem C-ABI call (no batching, no graph)."""
    import torch

    from qimpy_gb300 import autotune, batch as bt, ops

    dev = torch.device(f"cuda:{local}")
    t0 = time.perf_counter()
    specs = bt.make_batch_specs(count=args.batch)
    shapes = sorted({(s.grid,) * 3 for s in specs})
    sched = {sh: autotune.tune_shape(sh, torch.complex64, dev) for sh in shapes}
    t_tune = time.perf_counter() - t0
    insts = [bt.Instance(s, dev, fft_factors=sched[(s.grid,) * 3]) for s in specs]
    bh = bt.BatchedHamiltonian(insts, dev, plane_chunk_bytes=args.batch_chunk_mb << 20)
    bh.capture()
    t_setup = time.perf_counter() - t0
    flush = torch.empty(512 * 1024 * 1024 // 4, dtype=torch.float32, device=dev)
    for _ in range(args.warmup):
        bh.replay()
    torch.cuda.synchronize()
    times = []
    for _ in range(args.steps):
        flush.zero_()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        bh.replay()
        e1.record()
        torch.cuda.synchronize()
        times.append(e0.elapsed_time(e1) * 1e-3)
    # Unbatched reference point: per-instance calls, eager.
    ws = [ops.workspace(i.sphere.hamiltonian_mixed_workspace_bytes(i.nb, i.beta.shape[1]), dev) for i in insts]
    outs = [torch.empty_like(i.C) for i in insts]

    def sequential():
        for i, w, o in zip(insts, ws, outs):
            ops.hamiltonian_mixed(i.sphere, i.C, i.split, i.D, out=o, ws=w)

    sequential()
    torch.cuda.synchronize()
    seq = []
    for _ in range(max(1, args.steps // 2)):
        flush.zero_()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        sequential()
        e1.record()
        torch.cuda.synchronize()
        seq.append(e0.elapsed_time(e1) * 1e-3)
    agree = max(float((a - b).abs().max() / b.abs().max()) for a, b in zip(bh.outputs, outs))
    n_sh = len(shapes)
    return dict(instances=len(insts), band_apps_per_step=bh.band_apps, grids=f"{n_sh} shapes "
                f"{shapes[0][0]}^3..{shapes[-1][0]}^3", value=bh.band_apps / float(np.median(times)),
                unit=UNIT, ms_per_step=1e3 * float(np.median(times)),
                sequential_value=bh.band_apps / float(np.median(seq)),
                batched_over_sequential=float(np.median(seq)) / float(np.median(times)),
                max_rel_diff_batched_vs_sequential=agree, launches_per_step=bh.launches(),
                solo_instances=len(bh.solo), solo_units=bh.solo_units,
                setup_s=t_setup, autotune_s=t_tune,
                schedule={f"{k[0]}": [list(f) for f in v] for k, v in sched.items()},
                error_word=int(ops.device_error_word(dev).item()))


def run_serving(args, local):
    """Continuous-batching eigensolve server: a Poisson stream (mean 200 req/s)
    of requests for the lowest N_bands in {8..160} eigenpairs (eigenvalue change
    below 1e-6 Ha; mixed requests then refined in FP64 to 1e-8 Ha),
    cells drawn from the batched-instance distribution plus 5% 64-atom Si-like
    cells (side 20.52 bohr, 96^3, Ecut 20 Ha).  Mixed precision (FP32 H.psi,
    tensor-core nonlocal, FP64 subspace and refinement) and plain FP64 on the
    same bounded sample of the stream (`--serve` requests each), which keeps
    the run within minutes.  Gamma-only requests run with real wavefunctions."""
    import torch

    from qimpy_gb300 import batch as bt, serve as sv, workloads as wl

    dev = torch.device(f"cuda:{local}")
    out = {}
    for precision, count in (("mixed", args.serve), ("fp64", args.serve)):
        specs = bt.make_batch_specs(count=count, seed=41)
        u = wl.splitmix_uniform(41, 900, count)
        for i in range(count):
            if u[i] < 0.05:  # 64-atom Si-like cell
                pos = wl.supercell_positions(wl._DIAMOND_BASIS, 2)
                specs[i] = bt.InstanceSpec(i, 20.52, pos, 20.0, 160, np.zeros((1, 3)), 41 * 100003 + i, grid=96)
        reqs = sv.poisson_stream(specs, rate_hz=200.0, seed=41)
        with sv.EigenServer(dev, precision=precision, eig_threshold=1e-6, residual_threshold=1e-6) as srv:
            rep = srv.run(reqs, realtime=True, max_wall_s=args.serve_wall)
        res = [r.residual for r in reqs if r.status == "done"]
        rep["residual_max"] = float(np.max(res)) if res else None
        rep["residual_target"] = 1e-6
        rep["sample"] = f"{count} requests of the 200 req/s stream ({sum(u < 0.05)} Si64-like)"
        out[precision] = rep
    out["mixed_over_fp64_eigensolves"] = out["mixed"]["eigensolves_per_s"] / max(out["fp64"]["eigensolves_per_s"], 1e-12)
    return out


def cpu_baseline(args, p=None, b=None, beta=None, C=None, threads=None):
    """The reference's FP64 H.psi restated with torch CPU operations (the
    reference's own library and steps: scatter, ifftn, *V, fftn, gather per
    band; nonlocal as complex matmuls) on a bounded band sample, timed on every
    host core.  The reference itself is not installed where the bench runs; on
    one x86 host the port runs at the reference's speed (REFERENCE_OVER_PORT)."""
    import torch

    from oracle import hpsi_torch as oht

    threads = threads or os.cpu_count()
    oht.set_threads(threads)
    if p is None:
        p, b, beta, C = make_workload(args.workload)
    nbs = max(1, args.cpu_sample_bands)
    Cs = np.ascontiguousarray(C[:, :nbs])
    H = oht.Hamiltonian(b.ke, p.V_r, b.fft_index, b.n, beta, p.D_all())
    H(Cs)  # warm-up
    t0 = time.perf_counter()
    reps = 0
    while True:
        H(Cs)
        reps += 1
        if (time.perf_counter() - t0 > 10.0 and reps >= 3) or reps >= 20:
            break
    sec = (time.perf_counter() - t0) / reps
    return dict(value=nbs * p.nk / sec, unit=UNIT, cores=threads, kind="port",
                sample=f"{nbs} bands x {p.nk} k of {args.workload} (one block), {reps} H.psi calls, "
                       f"torch {torch.__version__} CPU with {threads} threads",
                reference_over_port_measured=REFERENCE_OVER_PORT)


def profile_davidson() -> None:
    """Kernel time tables of Davidson solves (torch.profiler, CPU and CUDA
    activities): si2 to convergence and si64 for 12 iterations, FP64 and
    mixed; an unprofiled si2 solve of each form runs first as a warm-up."""
    import torch
    from torch.profiler import ProfilerActivity, profile

    from qimpy_gb300 import davidson as dv, electrons as E, workloads as wl

    def solve(name, dtype, threshold, iters, prof):
        p = wl.get(name)
        el, C0 = E.from_problem(p, "cuda:0", dtype)
        el.C = E.Wavefunction(el.basis, coeff=C0.to("cuda:0", dtype)).orthonormalize()
        torch.cuda.synchronize()
        d = dv.Davidson(el, n_iterations=iters, eig_threshold=threshold)
        if not prof:
            d()
            return
        with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as pr:
            t0 = time.perf_counter()
            st = d()
            torch.cuda.synchronize()
            wall = time.perf_counter() - t0
        print(f"== {name} {dtype} iterations {st.iterations} wall {wall:.3f}s "
              f"per-iteration {1e3 * wall / st.iterations:.2f} ms")
        print(pr.key_averages().table(sort_by="cuda_time_total", row_limit=25, max_name_column_width=60))

    for dt, thr in ((torch.complex128, 1e-11), (torch.complex64, 1e-6)):
        solve("si2", dt, thr, 300, False)
        solve("si2", dt, thr, 300, True)
    for dt, thr in ((torch.complex128, 1e-9), (torch.complex64, 1e-6)):
        solve("si64", dt, thr, 12, True)


def main():
    args = parse_args()
    if args.profile_davidson:
        profile_davidson()
        return
    if args.impl == "reference":
        rank = int(os.environ.get("RANK", "0"))
        if rank != 0:
            return
        cb = cpu_baseline(args)
        out = {"metric": METRIC, "value": cb["value"], "unit": UNIT, "impl": "reference",
               "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup, "higher_is_better": True,
               "dtype": "f64", "data": "synthetic", "config": workload_config(args, args.gpus),
               "cpu_baseline": cb, "e2e": {"value": cb["value"], "unit": UNIT, "h2d_bytes_per_step": 0,
                                           "d2h_bytes_per_step": 0}}
        print(json.dumps(out))
        return
    rank, ws, local = dist_init()
    p, b, tables, results, peaks = run_gb300(args, rank, ws, local)
    if set(results) != {"fp64", "mixed"}:  # profiling run of one form: no JSON line
        print(json.dumps({k: {"value": v["value"], "ms_per_step": v["ms_per_step"]} for k, v in results.items()}))
        return
    mixed, f64 = results["mixed"], results["fp64"]
    # Roofline of the dominant stage of the mixed form (local potential, 3 kernels).
    rc = roofline_counts(p, b, tables, mixed["block"], mixed["real_bytes"])
    band_apps_block = mixed["block"] * p.nk
    t_loc = mixed["t_loc_block"]
    import json as _j

    peaks_file = os.path.join(ROOT, "MEASURED_PEAKS.json")
    measured = _j.load(open(peaks_file)) if os.path.exists(peaks_file) else {}
    hbm_peak = measured.get("hbm_gbs", 6800.0)
    bf16_peak = measured.get("bf16_tflops", 1900.0)
    out = {
        "metric": METRIC, "value": mixed["value"], "unit": UNIT, "n_gpus": ws, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": mixed["ms_per_step"], "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "c64 (f32)", "data": "synthetic",
        "config": workload_config(args, ws),
        "call_form": mixed["call_form"],
        "fp64": {"value": f64["value"], "ms_per_step": f64["ms_per_step"], "e2e": f64.get("e2e"),
                 "clocks": f64["clocks"], "fft_schedule": f64["fft_schedule"], "call_form": f64["call_form"],
                 "stage_form_rel_diff": f64["stage_form_rel_diff"],
                 "e2e_matches_device_result": f64.get("e2e_matches_device_result")},
        "stage_form_rel_diff": mixed["stage_form_rel_diff"],
        "e2e_matches_device_result": mixed.get("e2e_matches_device_result"),
        "fft_schedule": mixed["fft_schedule"],
        "mixed_over_fp64": mixed["value"] / f64["value"],
        "e2e": mixed.get("e2e"),
        "stages_ms_per_block": {"mixed": {"local": 1e3 * mixed["t_loc_block"], "nonlocal": 1e3 * mixed["t_nl_block"]},
                                "fp64": {"local": 1e3 * f64["t_loc_block"], "nonlocal": 1e3 * f64["t_nl_block"]}},
        "roofline": local_roofline(rc, band_apps_block, t_loc, hbm_peak, peaks),
        "nonlocal_roofline": nonlocal_roofline(rc, band_apps_block, mixed["t_nl_block"], hbm_peak, bf16_peak),
        "measured_fma_peaks_tflops": peaks,
        "gpu_launches": mixed["launches_per_step"] * args.steps,
        "clocks": mixed["clocks"],
    }
    real = run_real_hpsi(args, local)
    real["over_complex_form"] = {"fp64": real["fp64"]["value"] / f64["value"],
                                 "mixed": real["mixed"]["value"] / mixed["value"]}
    out["real_wavefunctions_si64"] = real
    if not args.no_eigensolve:
        out["eigensolve_si2"] = run_eigensolves(args, local)
        out["eigensolve_si64"] = run_eigensolve_si64(args, local)
    if args.batch:
        out["batch"] = run_batch(args, local)
    if args.serve:
        out["serving"] = run_serving(args, local)
    if rank == 0 and not args.no_cpu_baseline:
        out["cpu_baseline"] = cpu_baseline(args)
        cb = out["cpu_baseline"]["value"]
        # The precision-matched comparison: the plain FP64 form against the FP64
        # CPU baseline (the headline `value` is the FP32/BF16x3 mixed form).
        out["fp64"]["vs_cpu"] = f64["value"] / cb
        if f64.get("e2e"):
            out["fp64"]["e2e_vs_cpu"] = f64["e2e"]["value"] / cb
    if rank == 0:
        print(json.dumps(out))


if __name__ == "__main__":
    main()
