"""Outputs that are not contiguous, at the codec's entry points: the caller's tensor gets the result."""

import pytest
import torch

from lowbit_comm_b200 import CompressionConfig
from lowbit_comm_b200.ops import codec


@pytest.mark.parametrize("device", ["cpu", pytest.param("cuda", marks=pytest.mark.gpu)])
@pytest.mark.parametrize("kw", [{}, {"topk": 1}, {"compact": True}, {"bit": 4, "quant_type": "e2m1"}])
@pytest.mark.parametrize("make", [lambda new: new(30, 50).t(), lambda new: new(50, 60)[:, 7:37]])
def test_strided_outputs_hold_what_dense_ones_do(request, device, kw, make):
    """Transposed and sliced outputs (their flattened form is a copy) in every place that takes one."""

    if device == "cuda":
        request.getfixturevalue("ext")
    config = CompressionConfig(allow_experimental=True, **kw)
    base = torch.randn(30, 50, generator=torch.Generator().manual_seed(3)).to(torch.bfloat16).to(device)
    x, feedback = base.t(), (base * 0.01).t()

    def new(*shape):
        return torch.full(shape, 999.0, dtype=x.dtype, device=device)

    payloads = [codec.quantize_tensor(base.flip(k).t(), config) for k in (0, 1)]
    outputs = []
    for fresh in (lambda: new(50, 30), lambda: make(new)):
        out = []
        for residual in (None, feedback):
            prepared = fresh()
            out += [codec.quantize_tensor(x, config, residual=residual, prepared_out=prepared), prepared]
        dense, shared = prepared.clone(), fresh().copy_(prepared)
        result, left = fresh(), fresh()
        if codec.inplace_dequantize_reduce_mean(payloads, result, config, reduce="mean"):
            out.append(result)
            result = fresh()
            assert codec.inplace_dequantize_reduce_mean_update_error_feedback(payloads, dense, result, left, config)
            out += [result, left]
            result = fresh()
            assert codec.inplace_dequantize_reduce_mean_update_error_feedback(payloads, shared, result, shared, config)
            out += [result, shared]
        left = fresh()
        restored = codec.dequantize_reduce_update_error_feedback(payloads, dense, left, (50, 30), config, dtype="bf16")
        out += [restored, left]
        left = fresh()
        assert codec.update_error_feedback_residual(dense, restored, left) is left
        outputs.append(out + [left])
    for want, got in zip(*outputs, strict=True):
        assert torch.equal(got, want)
        assert want.dtype == torch.uint8 or not (want == 999.0).any()
