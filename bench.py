"""Benchmark of the attention forward path.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference|sdpa-flash|sdpa-cudnn|flash-attn]
                    [--workload NAME] [--scaling strong|weak]

One "step" is one forward pass of `flash_attn_cute` over the rank's share of the workload.  The default
workload is the shape the headline metric is quoted on: non-causal B=4, H=32, S=4096, D=128, i.e. 128
independent (batch, head) units, 1.0995 TFLOP per pass.

N = 1: the whole workload on one GPU.  N > 1 (launched by torchrun, one rank per GPU): the SAME 128 units
are cut into contiguous blocks, one per rank (`fray_b200.multi_gpu.shard_units`), each rank runs its block
as a `[1, units, S, D]` problem, there is no collective on the data path, and `value` is the workload's
FLOPs over the slowest rank's device time ("scaling": "strong").  `--scaling weak` gives every rank the
whole workload instead.  After the timed region every rank compares sampled units of its output with the
CPU oracle, the shards are all-gathered over NCCL and rank 0 checks the assembled tensor (`verify` in the
JSON line).

Prints ONE JSON line (rank 0).  `--impl reference` instead times the CPU oracle (torch CPU attention, the
comparison the reference's own test uses) on a bounded sample of the same workload, on rank 0 only.  The
`sdpa-*` / `flash-attn` arms time library attention kernels of the image on the same shapes with the same
protocol: comparison bars only, never part of the product path.
"""
import argparse
import json
import os
import statistics
import sys
import threading
import time

import torch

ROOT = os.path.dirname(os.path.abspath(__file__))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

NOMINAL_FP16_TFLOPS = 2250.0
# DRAM traffic of the kernel with two softmax threads per row from the ncu captures summarised in
# profiles/attn_fwd_duo_small_ncu.md (32 (b,h) units of S=4096, D=128, non-causal): dram__bytes_read.sum of a
# launch on a flushed L2, dram__bytes_write.sum of a launch behind others of its kind (a single launch leaves
# most of its output in L2).  Units are independent, so a launch with more units of the same shape moves
# proportionally more.
NCU_DRAM_BYTES_PER_UNIT_S4096_D128 = (100.742656e6 + 33.277184e6) / 32
FALLBACK_PEAKS = {"bf16_tflops": 1590.0, "bf16_tflops_sustained": 1400.0, "hbm_gbs": 6650.0}

WORKLOADS = {
    # name: (B, H, S, D, causal)
    "headline": (4, 32, 4096, 128, False),
    "c1": (1, 4, 256, 64, False),
    "c2": (2, 16, 2048, 128, False),
    "c3": (4, 32, 4096, 128, True),
    "c4": (1, 32, 16384, 128, True),
    "c5": (16, 16, 1024, 64, False),
    # one batch of the headline shape: 134 MB of operands (> L2), small enough for profiler captures
    "small": (1, 32, 4096, 128, False),
    "small_causal": (1, 32, 4096, 128, True),
}
ORACLE_CONFIG = {"c1": 0, "c2": 1, "c3": 2, "c4": 3, "c5": 4, "headline": 5}  # index into the oracle module's CONFIGS


def flops_of(B, H, S, D, causal):
    f = 4.0 * B * H * S * S * D
    return f / 2 if causal else f


def load_peaks():
    path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    try:
        with open(path) as f:
            peaks = json.load(f)
        return peaks, "measured"
    except (OSError, ValueError):
        return dict(FALLBACK_PEAKS), "fallback"


class ClockSampler:
    """Samples SM clock and throttle reasons through NVML from a thread while the timed region runs."""

    def __init__(self, gpu_index: int, period_s: float = 0.002):
        self.gpu_index = gpu_index
        self.period_s = period_s
        self.samples = []       # (sm_mhz, reasons bitmask, board power in W)
        self.sm_max = None
        self._stop = threading.Event()
        self.thread = None
        self.error = None

    def start(self):
        try:
            import pynvml
            pynvml.nvmlInit()
            visible = os.environ.get("CUDA_VISIBLE_DEVICES")
            index = self.gpu_index
            if visible:
                entry = visible.split(",")[self.gpu_index].strip()
                index = int(entry) if entry.isdigit() else self.gpu_index
            self.handle = pynvml.nvmlDeviceGetHandleByIndex(index)
            self.sm_max = float(pynvml.nvmlDeviceGetMaxClockInfo(self.handle, pynvml.NVML_CLOCK_SM))
            self.nvml = pynvml
        except Exception as exc:  # NVML missing: report it, do not fail the benchmark
            self.error = repr(exc)
            return
        self.thread = threading.Thread(target=self._loop, daemon=True)
        self.thread.start()

    def _loop(self):
        nv = self.nvml
        while not self._stop.is_set():
            try:
                clk = nv.nvmlDeviceGetClockInfo(self.handle, nv.NVML_CLOCK_SM)
                why = nv.nvmlDeviceGetCurrentClocksEventReasons(self.handle)
                try:
                    watts = nv.nvmlDeviceGetPowerUsage(self.handle) / 1000.0
                except Exception:
                    watts = None
                self.samples.append((float(clk), int(why), watts))
            except Exception as exc:
                self.error = repr(exc)
                return
            time.sleep(self.period_s)

    def stop(self):
        self._stop.set()
        if self.thread is not None:
            self.thread.join(timeout=2)
        if not self.samples:
            return {"sm_mhz": None, "sm_max_mhz": self.sm_max, "reasons": [f"no samples: {self.error}"], "samples": 0}
        nv = self.nvml
        names = {
            "hw_slowdown": nv.nvmlClocksEventReasonHwSlowdown,
            "hw_thermal_slowdown": nv.nvmlClocksEventReasonHwThermalSlowdown,
            "sw_thermal_slowdown": nv.nvmlClocksEventReasonSwThermalSlowdown,
            "sw_power_cap": nv.nvmlClocksEventReasonSwPowerCap,
        }
        seen = 0
        for _, why, _ in self.samples:
            seen |= why
        reasons = sorted(n for n, bit in names.items() if seen & bit)
        clocks = [c for c, _, _ in self.samples]
        watts = [w for _, _, w in self.samples if w is not None]
        return {"sm_mhz": statistics.median(clocks), "sm_min_mhz": min(clocks), "sm_max_mhz": self.sm_max,
                "power_w": statistics.median(watts) if watts else None,
                "reasons": reasons, "samples": len(self.samples)}


def _all_host_threads():
    # torchrun pins OMP_NUM_THREADS=1; the CPU legs are meant to use every core this process may run on
    try:
        torch.set_num_threads(len(os.sched_getaffinity(0)))
    except (AttributeError, RuntimeError):
        pass
    return torch.get_num_threads()


def cpu_attention_sample(S, D, causal, budget_s=12.0):
    """Times torch CPU attention (fp32 math on the fp16 inputs) on successive (b,h) units until the
    budget is used; returns (TFLOP/s, units done, seconds, threads)."""
    import torch.nn.functional as F
    from oracle import attention_ref as ref
    threads = _all_host_threads()
    q, k, v = ref.make_slice(5, 0, S, D)
    q, k, v = (t.float().reshape(1, 1, S, D) for t in (q, k, v))
    F.scaled_dot_product_attention(q, k, v, is_causal=causal)  # warm-up
    done, t0 = 0, time.perf_counter()
    while (time.perf_counter() - t0) < budget_s:
        F.scaled_dot_product_attention(q, k, v, is_causal=causal)
        done += 1
    dt = time.perf_counter() - t0
    return flops_of(1, done, S, D, causal) / dt / 1e12, done, dt, threads


def workload_config(args, B, H, S, D, causal, world):
    """The `config` object both arms print: same keys, same meaning."""
    return {"workload": args.workload, "B": B, "H": H, "S": S, "D": D, "causal": causal, "units": B * H,
            "scaling": args.scaling if world > 1 else "single GPU",
            "flops_per_pass": flops_of(B, H, S, D, causal)}


def run_reference(args, B, H, S, D, causal, rank, world):
    """CPU arm: torch CPU attention on a bounded sample of the workload, rank 0 only."""
    if rank != 0:
        return
    import torch.nn.functional as F
    from oracle import attention_ref as ref
    threads = _all_host_threads()
    units_per_step = 2
    ci = ORACLE_CONFIG.get(args.workload)
    q, k, v = ref.make_inputs(ci, range(units_per_step)) if ci is not None else tuple(
        torch.randn(units_per_step, S, D).half() for _ in range(3))
    q, k, v = (t.float().unsqueeze(0) for t in (q, k, v))
    for _ in range(max(args.warmup, 1)):
        F.scaled_dot_product_attention(q, k, v, is_causal=causal)
    t0 = time.perf_counter()
    for _ in range(args.steps):
        F.scaled_dot_product_attention(q, k, v, is_causal=causal)
    dt = time.perf_counter() - t0
    value = flops_of(1, units_per_step, S, D, causal) * args.steps / dt / 1e12
    sample = f"{units_per_step} of {B * H} (b,h) units per step, torch CPU scaled_dot_product_attention in fp32"
    line = {
        "impl": "reference", "metric": "flash_attn_fwd_tflops", "value": value, "unit": "TFLOP/s",
        "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup, "ms_per_step": dt / args.steps * 1e3,
        "higher_is_better": True, "scaling": "strong" if world > 1 and args.scaling == "strong" else "weak",
        "vs_baseline": None, "dtype": "f32", "data": "synthetic",
        "config": {**workload_config(args, B, H, S, D, causal, world), "sample": sample},
        "cpu_baseline": {"value": value, "unit": "TFLOP/s", "cores": threads, "kind": "port", "sample": sample},
        "e2e": {"value": value, "unit": "TFLOP/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "gpu_launches": 0,
    }
    print(json.dumps(line), flush=True)


def run_library_bar(args, B, H, S, D, causal):
    """Comparison bars: a library attention kernel of the image on the same shape, same timing protocol
    (inputs resident, W warm-ups, K back-to-back launches between CUDA events).  Reported, never shipped."""
    import torch.nn.functional as F
    assert torch.cuda.is_available()
    q, k, v = (torch.randn(B, H, S, D, device="cuda", dtype=torch.half) for _ in range(3))
    try:
        if args.impl in ("sdpa-flash", "sdpa-cudnn"):
            from torch.nn.attention import SDPBackend, sdpa_kernel
            backend = SDPBackend.FLASH_ATTENTION if args.impl == "sdpa-flash" else SDPBackend.CUDNN_ATTENTION

            def step():
                with sdpa_kernel(backend):
                    return F.scaled_dot_product_attention(q, k, v, is_causal=causal)
        else:
            from flash_attn import flash_attn_func
            qt, kt, vt = (t.transpose(1, 2).contiguous() for t in (q, k, v))   # [B, S, H, D]

            def step():
                return flash_attn_func(qt, kt, vt, causal=causal)
        for _ in range(max(args.warmup, 3)):
            step()
        torch.cuda.synchronize()
        sampler = ClockSampler(torch.cuda.current_device())
        sampler.start()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(args.steps):
            step()
        e1.record()
        torch.cuda.synchronize()
        clocks = sampler.stop()
        ms = e0.elapsed_time(e1) / args.steps
        line = {"impl": args.impl, "metric": "flash_attn_fwd_tflops", "value": flops_of(B, H, S, D, causal) / ms / 1e9,
                "unit": "TFLOP/s", "ms_per_step": ms, "steps": args.steps, "warmup": args.warmup,
                "config": workload_config(args, B, H, S, D, causal, 1), "clocks": clocks,
                "note": "library kernel, comparison bar only"}
    except Exception as exc:  # backend not available for this shape / build
        line = {"impl": args.impl, "unavailable": f"{type(exc).__name__}: {str(exc)[:200]}"}
    print(json.dumps(line), flush=True)


def verify_shard(out_local, q, k, v, lo, H, causal, dist, n_units, rank):
    """Sampled units of this rank's output against the CPU oracle; then (N > 1) all-gather of the shards
    over the process group and, on rank 0, the same check on units of other ranks in the assembled
    tensor.  Returns a short verdict string."""
    from oracle import attention_ref as ref
    from fray_b200.multi_gpu import gather_units

    def check_unit(out_u, q_u, k_u, v_u):
        out_u, q_u, k_u, v_u = (t.cpu().unsqueeze(0) for t in (out_u, q_u, k_u, v_u))
        max_abs = (out_u.float() - ref.sdpa_cpu(q_u, k_u, v_u, causal).float()).abs().max().item()
        diff = ref.calc_diff(out_u, ref.attention_fp32(q_u, k_u, v_u, causal))
        return max_abs <= 1e-2 and diff <= 1e-5, max_abs, diff

    n_local = out_local.shape[0]
    worst = (0.0, 0.0)
    ok = True
    for u in sorted({0, n_local // 2, n_local - 1}):
        good, a, d = check_unit(out_local[u], q[u], k[u], v[u])
        ok &= good
        worst = (max(worst[0], a), max(worst[1], d))
    gathered = "single GPU"
    if dist is not None:
        full = gather_units(out_local, n_units)                      # NCCL all-gather of the shards
        fq, fk, fv = (gather_units(t, n_units) for t in (q, k, v))
        flags = torch.tensor([1.0 if ok else 0.0], device="cuda")
        if rank == 0:
            assert full.shape[0] == n_units
            for u in sorted({n_units // 2 + 1, n_units - 1}):       # units other ranks computed
                good, a, d = check_unit(full[u], fq[u], fk[u], fv[u])
                ok &= good
                worst = (max(worst[0], a), max(worst[1], d))
            ok &= bool(torch.equal(full[lo:lo + n_local], out_local))
            flags[0] = 1.0 if ok else 0.0
        dist.all_reduce(flags, op=dist.ReduceOp.MIN)
        ok = bool(flags.item() == 1.0)
        gathered = f"{n_units} units gathered over NCCL"
    return f"{'ok' if ok else 'FAILED'} (max|d| {worst[0]:.1e}, calc_diff {worst[1]:.1e}; {gathered})", ok


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference", "sdpa-flash", "sdpa-cudnn", "flash-attn"])
    ap.add_argument("--workload", default="headline", choices=sorted(WORKLOADS))
    ap.add_argument("--scaling", default="strong", choices=["strong", "weak"],
                    help="N > 1: shard the workload's (b,h) units over the ranks (strong) or give each rank all of them")
    ap.add_argument("--settle", type=float, default=1.0,
                    help="idle seconds between the one-off kernel search and the warm-up steps")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-verify", action="store_true")
    ap.add_argument("--kernel-only", action="store_true", help="skip the end-to-end, verification and CPU legs (profiler runs)")
    args = ap.parse_args()
    args.warmup = max(args.warmup, 3) if args.impl == "ours" else args.warmup

    rank = int(os.environ.get("RANK", "0"))
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    B, H, S, D, causal = WORKLOADS[args.workload]

    if args.impl == "reference":
        run_reference(args, B, H, S, D, causal, rank, world)
        return
    if args.impl != "ours":
        if rank == 0:
            run_library_bar(args, B, H, S, D, causal)
        return

    assert torch.cuda.is_available(), "bench.py needs a GPU: the attention path has no CPU fallback"
    torch.cuda.set_device(local_rank)
    dist = None
    if world > 1:
        import torch.distributed as dist
        os.environ.setdefault("MASTER_ADDR", "127.0.0.1")
        dist.init_process_group("nccl", device_id=torch.device("cuda", local_rank))

    from fray_b200.jit_kernels import flash_attn_cute, flash_attn_cute_host, flash_attn_status
    from fray_b200.jit_kernels.tuner import jit_tuner
    from fray_b200.multi_gpu import shard_units
    # This rank's (b,h) units.  Synthetic N(0,1) inputs: every rank draws the whole workload from the same
    # seed (three launches) and keeps its block, so a unit holds the same data whichever rank owns it.
    n_units = B * H
    strong = world > 1 and args.scaling == "strong"
    lo, hi = shard_units(n_units, rank, world) if strong else (0, n_units)
    n_local = hi - lo
    gen = torch.Generator(device="cuda").manual_seed(42 * 1000)
    q, k, v = (torch.randn(n_units, S, D, generator=gen, device="cuda", dtype=torch.float32)[lo:hi].half().contiguous()
               for _ in range(3))
    out = torch.zeros_like(q)
    # the op sees [B, H, S, D] on one GPU (the reference's call), [1, units, S, D] for a shard
    shape4 = (B, H, S, D) if not strong else (1, n_local, S, D)
    q4, k4, v4, out4 = (t.view(shape4) for t in (q, k, v, out))
    flops_local = flops_of(1, n_local, S, D, causal)
    flops_total = flops_of(B, H, S, D, causal) * (1 if strong or world == 1 else world)

    def step():
        flash_attn_cute(q4, k4, v4, out4, causal=causal)

    def barrier():
        torch.cuda.synchronize()
        if dist is not None:
            dist.barrier()
        torch.cuda.synchronize()

    step()  # JIT lookup + tuning happen here, outside every timed region
    # The candidate search keeps the GPU at its power limit for several hundred launches; the board needs a
    # moment off the limit before the warm-up, or the timed steps measure the tuner's heat, not the kernel.
    barrier()
    if args.settle > 0:
        time.sleep(args.settle)
    for _ in range(args.warmup):
        step()
    barrier()

    sampler = ClockSampler(local_rank)
    if rank == 0:
        sampler.start()
    stream = torch.cuda.current_stream()
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    ev0.record(stream)
    for _ in range(args.steps):
        step()
    ev1.record(stream)
    barrier()
    ms_total = ev0.elapsed_time(ev1)
    clocks = sampler.stop() if rank == 0 else None
    status = flash_attn_status()
    assert status[0] == 0, f"device status {status}"

    if args.kernel_only:
        if rank == 0:
            value = flops_total / (ms_total / args.steps * 1e-3) / 1e12
            print(json.dumps({"metric": "flash_attn_fwd_tflops", "value": value, "unit": "TFLOP/s", "n_gpus": world,
                              "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms_total / args.steps,
                              "config": {"workload": args.workload}, "kernel_only": True, "clocks": clocks}), flush=True)
        return

    # ---- verification (after the timed region): this rank's units against the CPU oracle, then the gather
    verdict, verified = ("skipped", True) if args.no_verify else verify_shard(
        out, q, k, v, lo, H, causal, dist if strong else None, n_units, rank)

    # ---- end to end: pinned host inputs -> device, op, result -> pinned host, every step
    hq, hk, hv = (t.view(shape4).cpu().pin_memory() for t in (q, k, v))
    hout = torch.empty_like(hq).pin_memory()
    e2e_steps = max(3, min(args.steps, 10))

    def e2e_step():
        # the package's host-buffer call: slices staged through the device on three streams, every step
        # copies all inputs in and the whole result out
        flash_attn_cute_host(hq, hk, hv, hout, causal=causal)

    for _ in range(2):
        e2e_step()
    barrier()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for _ in range(e2e_steps):
        e2e_step()
    e1.record(stream)
    barrier()
    e2e_ms_total = e0.elapsed_time(e1)

    mine = torch.tensor([ms_total / args.steps, e2e_ms_total / e2e_steps], device="cuda", dtype=torch.float64)
    per_rank = [mine.clone() for _ in range(world)]
    if dist is not None:
        dist.all_gather(per_rank, mine)
    ms_step = max(t[0].item() for t in per_rank)          # slowest rank
    e2e_ms_step = max(t[1].item() for t in per_rank)

    if rank == 0:
        peaks, peak_src = load_peaks()
        value = flops_total / (ms_step * 1e-3) / 1e12
        per_gpu = value / world
        e2e_value = flops_total / (e2e_ms_step * 1e-3) / 1e12
        # A timed region of tens of milliseconds is a burst measurement: the denominator is the measured
        # burst bf16 GEMM figure, always; the sustained ratio is carried beside it.
        peak = float(peaks.get("bf16_tflops", FALLBACK_PEAKS["bf16_tflops"]))
        sustained = float(peaks.get("bf16_tflops_sustained", FALLBACK_PEAKS["bf16_tflops_sustained"]))
        traffic = NCU_DRAM_BYTES_PER_UNIT_S4096_D128 * n_local if (S, D, causal) == (4096, 128, False) else None
        tuned = {str(sig[1]): keys for sig, keys in jit_tuner.tuned_keys.items()}
        in_bytes = 3 * q.numel() * 2
        line = {
            "metric": "flash_attn_fwd_tflops", "value": value, "unit": "TFLOP/s", "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms_step, "higher_is_better": True,
            "scaling": "strong" if strong else "weak", "vs_baseline": None, "dtype": "f16", "data": "synthetic",
            "config": {**workload_config(args, B, H, S, D, causal, world), "units_per_gpu": n_local,
                       "l2": f"inputs per pass and GPU ({in_bytes / 1e6:.0f} MB) larger than the 126 MB L2"
                       if in_bytes > 126e6 else f"inputs per pass and GPU ({in_bytes / 1e6:.0f} MB) fit the 126 MB L2: "
                       "K/V are re-read from L2 by design, Q/K/V/O each cross HBM once",
                       "kernel": tuned,
                       "settle_s": args.settle},
            "per_rank_ms": [round(t[0].item(), 4) for t in per_rank],
            "verify": verdict,
            "roofline": {"bound": "tensor", "achieved": per_gpu, "peak": peak, "unit": "TFLOP/s",
                         "frac": per_gpu / peak, "traffic": traffic,
                         "traffic_note": "bytes per launch per GPU: ncu captures of the one-batch case "
                                         "(profiles/attn_fwd_duo_small_ncu.md) scaled by the units launched",
                         "algorithmic_bytes": 4 * n_local * S * D * 2,
                         "peak_source": f"{peak_src} burst bf16 GEMM (MEASURED_PEAKS.json bf16_tflops)",
                         "frac_of_nominal_2250": per_gpu / NOMINAL_FP16_TFLOPS,
                         "frac_of_sustained_gemm": per_gpu / sustained},
            "e2e": {"value": e2e_value, "unit": "TFLOP/s", "ms_per_step": e2e_ms_step,
                    "h2d_bytes_per_step": 3 * n_units * S * D * 2 * (1 if strong or world == 1 else world),
                    "d2h_bytes_per_step": n_units * S * D * 2 * (1 if strong or world == 1 else world)},
            "gpu_launches": args.steps * world,
            "clocks": clocks,
        }
        if world == 1 and not args.no_cpu_baseline:
            cpu_v, cpu_units, cpu_s, cpu_threads = cpu_attention_sample(S, D, causal)
            line["cpu_baseline"] = {
                "value": cpu_v, "unit": "TFLOP/s", "cores": cpu_threads, "kind": "port",
                "sample": f"{cpu_units} single-(b,h)-unit passes (the workload has {B * H} units) in {cpu_s:.1f} s, torch CPU "
                          f"scaled_dot_product_attention in fp32, host has {os.cpu_count()} logical cores"}
        print(json.dumps(line), flush=True)

    if dist is not None:
        dist.barrier()
        dist.destroy_process_group()
    if not verified:
        sys.exit(3)


if __name__ == "__main__":
    main()
