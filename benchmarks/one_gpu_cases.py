"""Times the cases of `perf/cases.py` on one GPU, and launches the one-GPU kernels once each for a profiler.

    python benchmarks/one_gpu_cases.py               # all listed cases: microseconds per pass, and its bytes at the copy rate
    python benchmarks/one_gpu_cases.py --only "mean of 8, 64 MiB bf16"
    python benchmarks/one_gpu_cases.py --launch              # 96 Mi bf16 elements through the linear kernels, for ncu
    python benchmarks/one_gpu_cases.py --launch-general      # 32 Mi bf16 elements through the general kernels

A pass is timed with CUDA events over `--passes` passes in a row that go round `--states` states prepared from different
seeds (so inputs and outputs change from pass to pass), after 2 rounds of warm-up; the median of 7 such runs.
"""

from __future__ import annotations

import argparse
import os
import statistics
import sys

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))

import torch  # noqa: E402

from benchmarks.kernel_bench import peak_gbs  # noqa: E402
from perf import cases  # noqa: E402


def microseconds(case: dict, states: int, passes: int, runs: int = 7) -> float:
    held = [cases.prepare(case, seed) for seed in range(states)]
    for state in held * 2:
        cases.run(state)
    torch.cuda.synchronize()
    out = []
    for _ in range(runs):
        start, stop = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        start.record()
        for i in range(passes):
            cases.run(held[i % states])
        stop.record()
        torch.cuda.synchronize()
        out.append(start.elapsed_time(stop) / passes * 1e3)
    return statistics.median(out)


def launch_once(n: int = 96 << 20) -> None:
    """Linear profile: encode and the one-rank passes with and without error feedback, decode, and the mean of four payloads."""

    from lowbit_comm_b200 import (CompressionConfig, compressed_all_reduce, dequantize_tensor,
                                  inplace_dequantize_reduce_mean_update_error_feedback, quantize_tensor)
    from lowbit_comm_b200.parallel.communicator import get_communicator

    cases._join_group()
    config = CompressionConfig(error_feedback=True)
    x = torch.randn(n, device="cuda", dtype=torch.bfloat16)
    r = torch.randn(n, device="cuda", dtype=torch.bfloat16)
    out = torch.empty_like(x)
    payloads = [quantize_tensor(x, config) for _ in range(3)] + [quantize_tensor(x, config, residual=r, prepared_out=r)]
    dequantize_tensor(payloads[0], (n,), config, dtype="bf16", output=out)
    inplace_dequantize_reduce_mean_update_error_feedback(payloads, r, out, r, config, reduce="mean")
    compressed_all_reduce(x, config=config, op="mean", strategy="auto")
    get_communicator(None).all_reduce(x, config=config, residual=r)
    torch.cuda.synchronize()


def launch_general_once(n: int = 32 << 20) -> None:
    """Encode, decode and the one-rank pass of the 4-bit code-book and of one and two kept values."""

    from lowbit_comm_b200 import CompressionConfig, compressed_all_reduce, dequantize_tensor, quantize_tensor

    cases._join_group()
    x = torch.randn(n, device="cuda", dtype=torch.bfloat16)
    for kw in ({"bit": 4, "quant_type": "e2m1"}, {"topk": 1}, {"topk": 2}):
        config = CompressionConfig(allow_experimental=True, **kw)
        dequantize_tensor(quantize_tensor(x, config), (n,), config, dtype="bf16")
        compressed_all_reduce(x.clone(), config=config, op="mean", strategy="auto")
    torch.cuda.synchronize()


def main() -> None:
    ap = argparse.ArgumentParser(description=__doc__, formatter_class=argparse.RawDescriptionHelpFormatter)
    ap.add_argument("--only", nargs="*", default=None, help="names of listed cases")
    ap.add_argument("--states", type=int, default=3)
    ap.add_argument("--passes", type=int, default=20)
    ap.add_argument("--launch", action="store_true")
    ap.add_argument("--launch-general", action="store_true")
    args = ap.parse_args()
    if args.launch:
        launch_once()
    elif args.launch_general:
        launch_general_once()
    else:
        peak, kind = peak_gbs()
        for case in cases.listed():
            if args.only and case["name"] not in args.only:
                continue
            us, moved = microseconds(case, args.states, args.passes), cases.work(case)["bytes"]
            print(f"{case['name']:30s} {us:9.2f} us   its bytes at {peak:.0f} GB/s ({kind}) {moved / peak / 1e3:8.2f} us",
                  flush=True)
            torch.cuda.empty_cache()
    if torch.distributed.is_initialized():
        torch.distributed.destroy_process_group()


if __name__ == "__main__":
    main()
