"""The work this library is timed on, on one GPU: what a training job has it do, through its public entry points.

A case is a dict of plain values.  `kind` names the entry point:

all_reduce  `compressed_all_reduce` of one gradient tensor, in place, on the job's process group (one rank here)
hook        the DDP communication hook over every bucket of one backward pass, error feedback on
ddp         a whole `DistributedDataParallel` step (forward, backward, the hook's reductions) of the synthetic MLP
shard       `compressed_reduce_scatter_shard` of a gradient bucket and `compressed_all_gather` of the shard that
            a sharded optimizer then owns
encode      `quantize_tensor`, with or without an error-feedback residual
decode      `dequantize_tensor`
mean        `inplace_dequantize_reduce_mean_update_error_feedback`: what a rank does with the payloads it gathered
            from all ranks (the reduction of every strategy that runs over torch.distributed)
codec       `Quantizer.quantize` and `.dequantize` one after the other: a tensor sent and received point to point,
            in any profile (top-k outliers, 4-bit codes and code-books, either payload layout)

Gradients are N(0, 1e-3) with one element in a thousand a hundred times larger, the distribution of the
all-reduce sweep; residuals are the size of one quantization step.
"""

from __future__ import annotations

import math

import torch

from lowbit_comm_b200 import (CompressionConfig, Quantizer, compressed_all_gather, compressed_all_reduce,
                              compressed_reduce_scatter_shard, create_ddp_comm_hook, dequantize_tensor,
                              estimate_quantized_size, inplace_dequantize_reduce_mean_update_error_feedback,
                              quantize_tensor)

MIB = 1 << 20
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
WIDTH = {"bf16": 2, "fp16": 2, "fp32": 4}


def listed() -> list[dict]:
    return [
        # a bias-sized bucket, or the tail bucket of a model: launches and host time are all there is
        {"name": "all_reduce 32 KiB bf16", "kind": "all_reduce", "dtype": "bf16", "numel": 16 * 1024},
        # one 25 MB DDP bucket reduced by hand (an odd size: buckets end where a parameter ends)
        {"name": "all_reduce 25 MB bf16", "kind": "all_reduce", "dtype": "bf16", "numel": 13_117_441},
        # the top of the all-reduce sweep
        {"name": "all_reduce 1 GiB bf16", "kind": "all_reduce", "dtype": "bf16", "numel": 512 * MIB},
        # the sweep's top-k arm: one outlier per group kept verbatim
        {"name": "all_reduce 64 MiB top-k 1", "kind": "all_reduce", "dtype": "bf16", "numel": 32 * MIB, "topk": 1},
        # the gradient exchange of one GPT-2 small step: 25 MB buckets, the embedding last, error feedback
        {"name": "hook gpt2-small bf16", "kind": "hook", "dtype": "bf16", "layers": 12, "width": 768, "vocab": 50257,
         "bucket_mib": 25},
        # the CPU example's MLP (1024 -> 4096 -> 4096 -> 1024, batch 32, fp32) as a GPU job, a whole step
        {"name": "ddp mlp fp32", "kind": "ddp", "dtype": "fp32", "inputs": 1024, "hidden": 4096, "hidden_layers": 2,
         "outputs": 1024, "batch": 32},
        # sharded optimizer: 32 MiB buckets through the reduced-shard interface
        {"name": "shard 32 MiB bf16", "kind": "shard", "dtype": "bf16", "numel": 16 * MIB},
        # encode with error feedback, as the torch.distributed path does per bucket
        {"name": "encode 64 MiB bf16 feedback", "kind": "encode", "dtype": "bf16", "numel": 32 * MIB, "feedback": True},
        # decode of a large payload (a dense checkpoint shard, a gathered tensor)
        {"name": "decode 256 MiB bf16", "kind": "decode", "dtype": "bf16", "numel": 128 * MIB},
        # eight ranks' payloads of one 64 MiB bucket into mean and residual
        {"name": "mean of 8, 64 MiB bf16", "kind": "mean", "dtype": "bf16", "numel": 32 * MIB, "payloads": 8},
        # a small odd-sized activation sent point to point, fp16, the per-group record layout
        {"name": "codec 99 k fp16 compact", "kind": "codec", "dtype": "fp16", "numel": 99_991, "group": 32,
         "compact": True},
        # the 4-bit code-book profile on a ragged fp32 tensor
        {"name": "codec 5 M fp32 e2m1", "kind": "codec", "dtype": "fp32", "numel": 5_000_001, "bit": 4,
         "quant": "e2m1"},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sizes(rng, lo: int, hi: int) -> int:
    """An element count spread over its logarithm: half of them odd, half whole rows."""

    n = _log_int(rng, lo, hi)
    return n | 1 if rng.random() < 0.5 else max(4096, n // 4096 * 4096)


def draw(rng) -> dict:
    kind = rng.choice(("all_reduce", "all_reduce", "all_reduce", "hook", "ddp", "shard", "encode", "decode", "mean",
                       "codec", "codec"))
    dtype = rng.choice(("bf16", "bf16", "fp16", "fp32"))
    case: dict = {"kind": kind, "dtype": dtype}
    if kind == "hook":
        case.update(layers=rng.randint(1, 12), width=64 * rng.randint(4, 12), vocab=rng.randint(1000, 50257),
                    bucket_mib=rng.choice((1, 10, 25, 50)))
        return case
    if kind == "ddp":
        case.update(inputs=rng.choice((512, 1000, 2048)), hidden=rng.choice((1024, 2048, 3000, 4096)),
                    hidden_layers=rng.randint(1, 4), outputs=rng.choice((10, 1000, 1024)), batch=rng.randint(1, 64))
        return case
    if kind == "all_reduce":
        topk = rng.choice((0, 0, 0, 0, 1, 2))
        top = (256 if topk == 0 else 64) * MIB // WIDTH[dtype]
        case.update(numel=_sizes(rng, 1024, top), group=rng.choice((64, 64, 32, 16)))
        if topk:
            case["topk"] = topk
        return case
    if kind == "shard":
        case.update(numel=_sizes(rng, 64 * 1024, 64 * MIB // WIDTH[dtype]), group=rng.choice((64, 64, 32)))
        return case
    if kind == "codec":
        case.update(numel=_sizes(rng, 1024, 16 * MIB // WIDTH[dtype]), group=rng.choice((64, 32, 16)),
                    compact=rng.random() < 0.5, topk=rng.choice((0, 0, 1, 2)))
        if rng.random() < 0.5:
            case.update(bit=4, quant=rng.choice(("linear", "normal", "uniform", "e3m0", "e2m1")))
        return case
    case.update(numel=_sizes(rng, 4096, 128 * MIB // WIDTH[dtype]), group=rng.choice((64, 64, 32, 16)),
                compact=rng.random() < 0.25)
    if rng.random() < 0.25:
        case["bit"] = 4
    if kind == "encode":
        case["feedback"] = rng.random() < 0.5
    if kind == "mean":
        case["payloads"] = rng.choice((2, 3, 4, 8))
    return case


def _config(case: dict) -> CompressionConfig:
    return CompressionConfig(bit=case.get("bit", 8), group_size=case.get("group", 64), topk=case.get("topk", 0),
                             quant_type=case.get("quant", "linear"), compact=case.get("compact", False),
                             error_feedback=True, allow_experimental=True)


def _join_group() -> None:
    """The job's process group: one rank on this GPU, as `torchrun --nproc-per-node 1` would set it up."""

    import torch.distributed as dist

    if not dist.is_initialized():
        dist.init_process_group("nccl", store=dist.HashStore(), rank=0, world_size=1,
                                device_id=torch.device("cuda", torch.cuda.current_device()))


def _gradient(n: int, dtype: torch.dtype, gen: torch.Generator, scale: float = 1e-3) -> torch.Tensor:
    x = torch.randn(n, generator=gen, device="cuda", dtype=dtype).mul_(scale)
    x[torch.randint(n, (max(1, n // 1000),), generator=gen, device="cuda")] *= 100
    return x


def _residual(n: int, dtype: torch.dtype, gen: torch.Generator) -> torch.Tensor:
    return (torch.rand(n, generator=gen, device="cuda", dtype=dtype) - 0.5) * 3e-5


class _Bucket:
    """One bucket of a backward pass, with the methods of `torch.distributed.GradBucket` (which Python cannot build)."""

    def __init__(self, index: int, last: bool, sizes: list[int], flat: torch.Tensor) -> None:
        self._index, self._last, self._flat = index, last, flat
        self._parameters = [torch.empty(n, device="meta") for n in sizes]

    def index(self) -> int:
        return self._index

    def is_last(self) -> bool:
        return self._last

    def buffer(self) -> torch.Tensor:
        return self._flat

    def parameters(self) -> list[torch.Tensor]:
        return self._parameters

    def gradients(self) -> list[torch.Tensor]:
        return list(self._flat.split([p.numel() for p in self._parameters]))


def _bucket_sizes(case: dict) -> list[list[int]]:
    """Parameter sizes of a decoder-only transformer, in the order the backward pass finishes them, cut into
    buckets as DDP cuts them: the first closes at 1 MiB, the others at `bucket_mib`."""

    d = case["width"]
    sizes = [d, d]
    for _ in range(case["layers"]):
        sizes += [d, 4 * d * d, 4 * d, 4 * d * d, d, d, d, d * d, 3 * d, 3 * d * d, d, d]
    sizes += [1024 * d, case["vocab"] * d]
    buckets, current, limit = [], [], MIB
    for n in sizes:
        current.append(n)
        if sum(current) * WIDTH[case["dtype"]] >= limit:
            buckets.append(current)
            current, limit = [], case["bucket_mib"] * MIB
    return buckets + ([current] if current else [])


def _mlp_widths(case: dict) -> list[int]:
    return [case["inputs"]] + [case["hidden"]] * case["hidden_layers"] + [case["outputs"]]


def _mlp_weights(case: dict) -> int:
    widths = _mlp_widths(case)
    return sum(a * b + b for a, b in zip(widths[:-1], widths[1:]))


def prepare(case: dict, seed: int) -> dict:
    kind, config = case["kind"], _config(case)
    dtype = DTYPES[case["dtype"]]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    state: dict = {"kind": kind, "config": config, "dtype": case["dtype"]}
    if kind in ("all_reduce", "hook", "ddp", "shard"):
        _join_group()
    if kind in ("all_reduce", "shard"):
        state["grad"] = _gradient(case["numel"], dtype, gen)
    elif kind == "hook":
        hook = create_ddp_comm_hook(config.evolve(target="ddp_gradient_bucket"), strategy="auto",
                                    max_bucket_numel=max(sum(b) for b in _bucket_sizes(case)))
        plan = _bucket_sizes(case)
        state["hook"] = hook
        state["buckets"] = [_Bucket(i, i == len(plan) - 1, sizes, _gradient(sum(sizes), dtype, gen))
                            for i, sizes in enumerate(plan)]
        for bucket in state["buckets"]:             # the residual an earlier step left behind
            hook.feedback.set(bucket.index(), _residual(bucket.buffer().numel(), dtype, gen))
    elif kind == "ddp":
        from lowbit_comm_b200.models.mlp import SyntheticMLP

        widths = _mlp_widths(case)
        with torch.device("cuda"):
            model = SyntheticMLP(widths, dtype=dtype)
        with torch.no_grad():
            for p in model.parameters():
                p.copy_(torch.randn(p.shape, generator=gen, device="cuda", dtype=dtype) / math.sqrt(p.shape[-1]))
        ddp = torch.nn.parallel.DistributedDataParallel(model, device_ids=[torch.cuda.current_device()],
                                                        bucket_cap_mb=25, gradient_as_bucket_view=True)
        ddp.register_comm_hook(state=None, hook=create_ddp_comm_hook(
            config.evolve(target="ddp_gradient_bucket"), strategy="auto", module=model))
        state["ddp"] = ddp
        state["x"] = torch.randn(case["batch"], widths[0], generator=gen, device="cuda", dtype=dtype)
        state["y"] = torch.randn(case["batch"], widths[-1], generator=gen, device="cuda", dtype=dtype)
    elif kind == "encode":
        state["grad"] = _gradient(case["numel"], dtype, gen)
        state["payload"] = torch.empty(_payload_bytes(case), dtype=torch.uint8, device="cuda")
        if case["feedback"]:
            state["residual"] = _residual(case["numel"], dtype, gen)
            state["prepared"] = torch.empty_like(state["grad"])
    elif kind == "decode":
        state["payload"] = quantize_tensor(_gradient(case["numel"], dtype, gen), config)
        state["out"] = torch.empty(case["numel"], dtype=dtype, device="cuda")
    elif kind == "mean":
        grads = [_gradient(case["numel"], dtype, gen) for _ in range(case["payloads"])]
        state["payloads"] = [quantize_tensor(g, config) for g in grads]
        state["prepared"] = grads[0]
        state["out"], state["residual"] = torch.empty_like(grads[0]), torch.empty_like(grads[0])
    else:
        state["quantizer"] = Quantizer(config, dtype=case["dtype"])
        state["x"] = _gradient(case["numel"], dtype, gen)
    return state


def run(state: dict):
    kind, config = state["kind"], state["config"]
    if kind == "all_reduce":
        return compressed_all_reduce(state["grad"], config=config, op="mean", strategy="auto")
    if kind == "hook":
        hook, buckets = state["hook"], state["buckets"]
        futures = [hook(None, bucket) for bucket in buckets]
        for future in futures:                      # DDP waits for every bucket at the end of the backward pass
            future.wait()
        return [f.value() for f in futures], [hook.feedback.get(b.index()) for b in buckets]
    if kind == "ddp":
        ddp = state["ddp"]
        ddp.zero_grad()
        loss = torch.nn.functional.mse_loss(ddp(state["x"]), state["y"])
        loss.backward()
        return loss.detach(), [p.grad for p in ddp.module.parameters()]
    if kind == "shard":
        shard = compressed_reduce_scatter_shard(state["grad"], config=config, op="mean")
        return shard.shard, compressed_all_gather(shard.shard, config=config)
    if kind == "encode":
        quantize_tensor(state["grad"], config, output=state["payload"], residual=state.get("residual"),
                        prepared_out=state.get("prepared"))
        return state["payload"], state.get("prepared")
    if kind == "decode":
        return dequantize_tensor(state["payload"], state["out"].shape, config, dtype=state["dtype"],
                                 output=state["out"])
    if kind == "mean":
        inplace_dequantize_reduce_mean_update_error_feedback(state["payloads"], state["prepared"], state["out"],
                                                             state["residual"], config, reduce="mean")
        return state["out"], state["residual"]
    payload = state["quantizer"].quantize(state["x"])
    return payload, state["quantizer"].dequantize(payload, state["x"].shape)


def _payload_bytes(case: dict) -> int:
    return estimate_quantized_size(case["numel"], dtype=case["dtype"], config=_config(case)).quantized_bytes


def work(case: dict) -> dict:
    """Bytes: each input read once and each output written once; a payload counts where it is an input or an output."""

    kind, width = case["kind"], WIDTH[case["dtype"]]
    if kind == "hook":
        n = sum(sum(sizes) for sizes in _bucket_sizes(case))
        return {"bytes": 4 * n * width, "flops": 0}            # gradient and residual, in and out
    if kind == "ddp":
        n = _mlp_weights(case)
        return {"bytes": 6 * n * width, "flops": 6 * n * case["batch"]}   # weights twice, gradient, residual in and out, result
    dense = case["numel"] * width
    if kind == "all_reduce":
        return {"bytes": 2 * dense, "flops": 0}
    if kind == "shard":
        return {"bytes": 4 * dense, "flops": 0}
    payload = _payload_bytes(case)
    if kind == "encode":
        return {"bytes": (3 if case["feedback"] else 1) * dense + payload, "flops": 0}
    if kind == "decode":
        return {"bytes": dense + payload, "flops": 0}
    if kind == "mean":
        return {"bytes": 3 * dense + case["payloads"] * payload, "flops": 0}
    return {"bytes": 2 * dense + 2 * payload, "flops": 0}


def tolerance(case: dict):
    """The wire format fixes every rounding, so payloads and what is decoded from one payload are the same bytes in
    any correct implementation.  A mean of several payloads may be summed in another order (fp32 sums, one rounding to
    the result's type): reversing the order of eight payloads moves it by 5e-5 (bf16), 9e-6 (fp16) and 8e-8 (fp32).
    The gradients of a training step come out of matrix products: with float64 products in front of the same codec
    they move by 1.6e-4 in fp32 (a few values fall to the neighbouring code), one rounding of the type in 16 bits."""

    if case["kind"] == "ddp":
        return {"rel": 7e-4, "max": 0.25} if case["dtype"] == "fp32" else {"rel": 1e-2, "max": 0.5}
    if case["kind"] == "mean":
        return {"bf16": {"rel": 2e-4, "max": 3e-2}, "fp16": {"rel": 4e-5, "max": 4e-3},
                "fp32": {"rel": 3e-7, "max": 3e-6}}[case["dtype"]]
    return "exact"
