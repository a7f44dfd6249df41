"""Helpers shared by the benchmark scripts at the repository root (`bench.py`, `bench_kernels.py`,
`bench_stack.py`): measured roofline denominators, clock sampling during a timed region, the
process-group set-up of a `torchrun` launch, and the timing loop (warm-up, barrier + synchronise
on both sides, CUDA events on the launching stream, maximum over ranks)."""
from __future__ import annotations

import json
import os
import statistics
import subprocess
import sys
import threading
import time
from pathlib import Path

import torch

ROOT = Path(__file__).resolve().parent

ROWS = COLS = 8192                        # the NVFP4 quantize configuration: bf16 [8192, 8192]
ALG_BYTES_PER_ELEM = 2 + 0.5 + 1.0 / 16  # bf16 read, packed code write, block-scale write
REQUIRED_KEYS = ("impl", "metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling", "vs_baseline",
                 "dtype", "data", "config", "clocks", "e2e", "gpu_launches", "roofline", "device_status", "error")
L2_ROTATION = 4                           # distinct input tensors cycled through (4 x 134 MB > 126 MB L2)


# ----------------------------------------------------------------------------- helpers
def measured_peaks():
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        d = json.loads(p.read_text())
        return {"hbm_gbs": d["hbm_gbs"], "bf16_tflops": d["bf16_tflops"],
                "bf16_tflops_sustained": d.get("bf16_tflops_sustained", d["bf16_tflops"]), "source": "measured"}
    return {"hbm_gbs": 6650.0, "bf16_tflops": 1590.0, "bf16_tflops_sustained": 1400.0, "source": "fallback"}


class ClockSampler:
    """Samples SM clocks and throttle reasons with nvidia-smi while the timed region runs."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index: int):
        self.index = index
        self.proc = None
        self.lines: list[str] = []
        self.thread = None

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits",
                                          "-lms", "100", "-i", str(self.index)], stdout=subprocess.PIPE,
                                         stderr=subprocess.DEVNULL, text=True)
            self.thread = threading.Thread(target=self._read, daemon=True)
            self.thread.start()
        except OSError:
            self.proc = None
        return self

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def __exit__(self, *exc):
        if self.proc is not None:
            time.sleep(0.15)
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def summary(self):
        sm, mx, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in self.lines:
            f = [t.strip() for t in line.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                mx.append(float(f[2]))
            except ValueError:
                continue
            for name, val in zip(names, f[5:9]):
                if val.lower().startswith("active"):
                    reasons.add(name)
        if not sm:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": [], "samples": 0}
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": max(mx), "reasons": sorted(reasons), "samples": len(sm)}


def make_input(seed: int, rows: int = ROWS, cols: int = COLS) -> torch.Tensor:
    """bf16 [rows, cols] ~ N(0,1), 1 % of the elements x50; generated on the CPU so the oracle
    and the device see identical bits."""
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(rows, cols, generator=g)
    x[torch.rand(rows, cols, generator=g) < 0.01] *= 50
    return x.bfloat16()


def _short(v):
    if isinstance(v, float):
        return float(f"{v:.6g}")
    if isinstance(v, dict):
        return {k: _short(x) for k, x in v.items()}
    return [_short(x) for x in v] if isinstance(v, (list, tuple)) else v


def print_line(line: dict, details: dict | None = None, limit: int = 2600) -> None:
    """The result as ONE JSON line on stdout, floats at six digits and short enough (`limit` characters) for a reader that keeps
    the end of the output only.  `details` (per-shape tables) go to stderr with everything else, at full precision; what would
    still be too long leaves the line from its end."""
    if details:
        print(json.dumps({**line, **details}), file=sys.stderr, flush=True)
    line = _short(line)
    optional = [k for k in line if k not in REQUIRED_KEYS]
    while len(json.dumps(line)) > limit and optional:
        line.pop(optional.pop())
    print(json.dumps(line), flush=True)


def dist_setup(n_gpus: int):
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if world > 1:
        import torch.distributed as dist

        torch.cuda.set_device(local)
        dist.init_process_group("nccl", device_id=torch.device("cuda", local))
    else:
        torch.cuda.set_device(0)
    return rank, world, local


def barrier(world):
    if world > 1:
        import torch.distributed as dist

        dist.barrier()
    torch.cuda.synchronize()


def max_over_ranks(ms: float, world: int) -> float:
    if world == 1:
        return ms
    import torch.distributed as dist

    t = torch.tensor([ms], device="cuda", dtype=torch.float64)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def timed(fn, steps, warmup, world):
    """W warm-up calls, then exactly `steps` calls between CUDA events on the current stream,
    bracketed by barrier + synchronize; returns max-over-ranks milliseconds for all steps."""
    for i in range(warmup):
        fn(i)
    barrier(world)
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    for i in range(steps):
        fn(warmup + i)
    e1.record()
    barrier(world)
    return max_over_ranks(e0.elapsed_time(e1), world)
