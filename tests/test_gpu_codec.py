"""sm_100a codec kernels against the bit-exact torch oracle (plain fp32 math on CPU).

Mirrors the intent of the reference's tests/cuda/test_fused_quant_pack.py and
tests/test_cuda_extension_smoke.py: uneven lengths, every dtype x bit x group
size, residual add, unaligned views, empty tensors, zero steady-state
allocation.
"""

import itertools

import numpy as np
import pytest
import torch

from lowbit_comm_b200.config import CompressionConfig
from lowbit_comm_b200.ops import codec, oracle
from lowbit_comm_b200.parallel.fused import FusedWorkspace
from lowbit_comm_b200.parallel.peer_memory import PeerGroup

pytestmark = pytest.mark.gpu

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def _cfg(**kw):
    return CompressionConfig(allow_experimental=True, **kw)


def _data(n, dtype, seed=0, outliers=True):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(n, generator=g) * 1e-2
    if outliers and n > 10:
        idx = torch.randint(0, n, (max(1, n // 100),), generator=g)
        x[idx] *= 50
    return x.to(dtype)


@pytest.mark.parametrize("dtype", list(DTYPES))
@pytest.mark.parametrize("bit,group", list(itertools.product((8, 4), (16, 32, 64))))
@pytest.mark.parametrize("compact", (False, True))
def test_fast_quantize_matches_oracle(ext, dtype, bit, group, compact):
    cfg = _cfg(bit=bit, group_size=group, compact=compact)
    for n in (group + 7, 1, group, 5 * group - 1, 4096 + 3 * group + 5):
        x = _data(n, DTYPES[dtype], seed=n)
        r = _data(n, DTYPES[dtype], seed=n + 1, outliers=False)
        for residual in (None, r):
            want = oracle.encode(x, cfg, residual=residual)
            got = codec.quantize_tensor(x.cuda(), cfg, residual=None if residual is None else residual.cuda())
            assert got.dtype == torch.uint8 and got.numel() == want.numel()
            assert torch.equal(got.cpu(), want), (dtype, bit, group, compact, n, residual is not None)
            back = codec.dequantize_tensor(got, (n,), cfg, dtype=dtype)
            assert torch.equal(back.cpu().view(torch.uint8), oracle.decode(want, n, cfg, dtype).view(torch.uint8))


def test_unaligned_views_and_prepared_out(ext):
    cfg = _cfg()
    base = _data(10_000, torch.bfloat16).cuda()
    rbase = _data(10_000, torch.bfloat16, seed=3, outliers=False).cuda()
    for off in (1, 3, 8, 17):
        x, r = base[off:off + 4099], rbase[off:off + 4099]
        prepared = torch.empty_like(x)
        got = codec.quantize_tensor(x, cfg, residual=r, prepared_out=prepared)
        assert torch.equal(got.cpu(), oracle.encode(x.cpu(), cfg, residual=r.cpu()))
        assert torch.equal(prepared.cpu(), oracle.prepare(x.cpu(), r.cpu()))


def test_empty_and_zero_tensors(ext):
    cfg = _cfg()
    empty = torch.empty(0, dtype=torch.bfloat16, device="cuda")
    assert codec.quantize_tensor(empty, cfg).numel() == 0
    zeros = torch.zeros(256, dtype=torch.float16, device="cuda")
    p = codec.quantize_tensor(zeros, cfg)
    assert torch.equal(p.cpu(), oracle.encode(zeros.cpu(), cfg))
    assert codec.dequantize_tensor(p, (256,), cfg, dtype="fp16").abs().max().item() == 0


@pytest.mark.parametrize("dtype", list(DTYPES))
@pytest.mark.parametrize("bit,group,compact", [(8, 64, False), (8, 64, True), (8, 16, False), (4, 32, False), (4, 64, True)])
@pytest.mark.parametrize("world", (1, 2, 8, 16))
def test_fused_reduce_mean_and_error_feedback(ext, dtype, bit, group, compact, world):
    cfg = _cfg(bit=bit, group_size=group, compact=compact)
    n = 9 * group + 11
    xs = [_data(n, DTYPES[dtype], seed=10 + r) for r in range(world)]
    payloads = [oracle.encode(x, cfg) for x in xs]
    want, want32 = oracle.reduce_mean(payloads, n, cfg, dtype)
    dev = [p.cuda() for p in payloads]
    out = torch.empty(n, dtype=DTYPES[dtype], device="cuda")
    assert codec.inplace_dequantize_reduce_mean(dev, out, cfg, reduce="mean")
    assert torch.equal(out.cpu().view(torch.uint8), want.view(torch.uint8))
    total = codec.dequantize_reduce_tensors(dev, (n,), cfg, dtype=dtype, reduce="sum")
    assert torch.equal(total.cpu().view(torch.uint8), oracle.reduce_mean(payloads, n, cfg, dtype, 1.0)[0].view(torch.uint8))
    prepared = xs[0].cuda()
    restored = torch.empty_like(prepared)
    residual = torch.zeros_like(prepared)
    assert codec.inplace_dequantize_reduce_mean_update_error_feedback(dev, prepared, restored, residual, cfg, reduce="mean")
    assert torch.equal(restored.cpu().view(torch.uint8), want.view(torch.uint8))
    assert torch.equal(residual.cpu().view(torch.uint8), oracle.residual_update(xs[0], want32).view(torch.uint8))
    # in-place form used by the DDP hook: `prepared` lives in the residual buffer
    alias = xs[0].cuda().clone()
    assert codec.inplace_dequantize_reduce_mean_update_error_feedback(dev, alias, restored, alias, cfg, reduce="mean")
    assert torch.equal(alias.cpu().view(torch.uint8), oracle.residual_update(xs[0], want32).view(torch.uint8))


def test_unfused_sum_accumulates_in_source_dtype(ext):
    cfg = _cfg()
    n = 1000
    a, b = _data(n, torch.bfloat16, 1), _data(n, torch.bfloat16, 2)
    pa, pb = oracle.encode(a, cfg), oracle.encode(b, cfg)
    out = codec.dequantize_tensor(pa.cuda(), (n,), cfg, dtype="bf16")
    codec.dequantize_tensor(pb.cuda(), (n,), cfg, dtype="bf16", output=out, reduce_op="sum")
    want = oracle.decode_accumulate(pb, oracle.decode(pa, n, cfg, "bf16"), cfg)
    assert torch.equal(out.cpu().view(torch.uint8), want.view(torch.uint8))


@pytest.mark.parametrize("dtype", list(DTYPES))
@pytest.mark.parametrize("group", (16, 32, 64))
@pytest.mark.parametrize("bit,quant_type,topk", [(8, "linear", 1), (8, "linear", 2), (4, "linear", 2), (4, "normal", 0),
                                                  (4, "uniform", 1), (4, "e3m0", 0), (4, "e2m1", 2)])
@pytest.mark.parametrize("compact", (False, True))
def test_general_kernels_match_oracle(ext, dtype, group, bit, quant_type, topk, compact):
    cfg = _cfg(bit=bit, group_size=group, topk=topk, quant_type=quant_type, compact=compact)
    for n in (group + 7, 7 * group, 2048 + 5):
        x = _data(n, DTYPES[dtype], seed=n + topk)
        x[:group] = 0  # an all-zero group exercises the top-k fall-backs
        if n > 2 * group:
            x[group:group + 4] = x[group]  # ties
        r = _data(n, DTYPES[dtype], seed=n + 9, outliers=False)
        want = oracle.encode(x, cfg, residual=r)
        got = codec.quantize_tensor(x.cuda(), cfg, residual=r.cuda())
        assert torch.equal(got.cpu(), want), (dtype, group, bit, quant_type, topk, compact, n)
        back = codec.dequantize_tensor(got, (n,), cfg, dtype=dtype)
        assert torch.equal(back.cpu().view(torch.uint8), oracle.decode(want, n, cfg, dtype).view(torch.uint8))
        both = codec.dequantize_reduce_tensors([got, got], (n,), cfg, dtype=dtype, reduce="sum")
        want2 = oracle.decode_accumulate(want, oracle.decode(want, n, cfg, dtype), cfg)
        assert torch.equal(both.cpu().view(torch.uint8), want2.view(torch.uint8))


def test_stochastic_rounding_is_unbiased(ext):
    cfg = _cfg(stochastic=True)
    x = torch.full((64 * 4096,), 0.3, dtype=torch.float32)
    x[::64] = 1.0  # scale 1.0 -> 0.3 * 127 = 38.1: rounds up 10 % of the time
    got = codec.dequantize_tensor(codec.quantize_tensor(x.cuda(), cfg), x.shape, cfg, dtype="fp32").cpu()
    body = got.reshape(-1, 64)[:, 1:]
    assert set(torch.unique(torch.round(body * 127)).tolist()) <= {38.0, 39.0}
    assert abs(body.double().mean().item() - 0.3) < 2e-4
    det = codec.dequantize_tensor(codec.quantize_tensor(x.cuda(), _cfg()), x.shape, _cfg(), dtype="fp32").cpu()
    assert abs(det.reshape(-1, 64)[:, 1:].double().mean().item() - 38 / 127) < 1e-6


def test_round_trip_error_envelope(ext):
    cfg = _cfg()
    x = torch.randn(1 << 20, dtype=torch.float16)
    y = codec.dequantize_tensor(codec.quantize_tensor(x.cuda(), cfg), x.shape, cfg, dtype="fp16").cpu()
    rel = ((y.float() - x.float()).norm() / x.float().norm()).item()
    assert rel < 0.02 and (y.float() - x.float()).abs().max().item() <= 0.0235


def test_error_feedback_update_and_scale(ext):
    a, b = _data(5001, torch.bfloat16, 1).cuda(), _data(5001, torch.bfloat16, 2).cuda()
    res = torch.empty_like(a)
    codec.update_error_feedback_residual(a, b, res)
    assert torch.equal(res.cpu(), oracle.residual_update_from_restored(a.cpu(), b.cpu()))


def test_zero_steady_state_allocation(ext):
    cfg = _cfg()
    x = _data(1 << 16, torch.bfloat16).cuda()
    r = torch.zeros_like(x)
    out = codec.allocate_quantized_buffer(x, cfg)
    restored = torch.empty_like(x)
    codec.quantize_tensor(x, cfg, output=out, residual=r)
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    ptr = out.data_ptr()
    for _ in range(100):
        codec.quantize_tensor(x, cfg, output=out, residual=r)
        codec.inplace_dequantize_reduce_mean_update_error_feedback([out], x, restored, r, cfg, reduce="mean")
    torch.cuda.synchronize()
    assert torch.cuda.memory_allocated() == before and out.data_ptr() == ptr


def test_payload_size_is_validated(ext):
    cfg = _cfg()
    x = _data(640, torch.bfloat16).cuda()
    with pytest.raises(ValueError):
        codec.quantize_tensor(x, cfg, output=torch.empty(10, dtype=torch.uint8, device="cuda"))
    with pytest.raises(ValueError):
        codec.dequantize_tensor(torch.empty(10, dtype=torch.uint8, device="cuda"), (640,), cfg, dtype="bf16")


@pytest.mark.parametrize("quant_type", ("normal", "uniform", "e3m0", "e2m1"))
def test_codebook_codes_at_their_thresholds(ext, quant_type):
    """Values next to the middle of two entries (and on the entries), where a code changes: the kernel counts
    thresholds, the oracle searches the table."""

    table = oracle.codebook(quant_type)[:15]
    near = [table]
    for mid in (table[:-1] + (table[1:] - table[:-1]) / 2,):
        for toward in (-2.0, 2.0):
            step = mid
            for _ in range(3):
                near.append(step)
                step = torch.nextafter(step, torch.full_like(step, toward))
    values = torch.cat(near)
    for scale in (1.0, 0.7310584, 3.0e-7, 1.7e37):
        groups = torch.zeros(-(-values.numel() // 15), 16)
        flat = torch.zeros(groups.shape[0] * 15)
        flat[:values.numel()] = values
        groups[:, 1:] = flat.reshape(-1, 15)
        groups[:, 0] = 1.0
        x = (groups * scale).reshape(-1)
        cfg = _cfg(bit=4, group_size=16, quant_type=quant_type)
        assert torch.equal(codec.quantize_tensor(x.cuda(), cfg).cpu(), oracle.encode(x, cfg)), scale


@pytest.mark.parametrize("quant_type", ("normal", "uniform", "e3m0", "e2m1"))
@pytest.mark.parametrize("dtype", list(DTYPES))
@pytest.mark.parametrize("topk", (0, 2))
def test_codebook_look_up_in_every_bucket(ext, quant_type, dtype, topk):
    """Encode and the one-rank pass where the look-up changes its entry: the powers of two and their quarters, the middles of the
    entries, each with its neighbours in the type, both signs, beside what is too small for any bucket."""

    table = oracle.codebook(quant_type)[:15]
    edges = torch.cat([torch.tensor([2.0 ** -e * (1 + q / 4) for e in range(1, 10) for q in range(4)]),
                       table[:-1] + (table[1:] - table[:-1]) / 2, torch.tensor([0.0, 1e-7, 2.0 ** -20])]).to(DTYPES[dtype])
    way = torch.full_like(edges, 2.0)
    values = torch.cat([edges, torch.nextafter(edges, way), torch.nextafter(edges, -way)]).clamp(-1, 1)
    values = torch.cat([values, -values])
    for scale in (1.0, 0.7310584, 3.0e-7):
        groups = torch.zeros(-(-values.numel() // 12), 16)
        flat = torch.zeros(groups.shape[0] * 12)
        flat[:values.numel()] = values
        groups[:, 4:] = flat.reshape(-1, 12)
        groups[:, :3] = torch.tensor([1.0, 4.0, -3.0]) if topk else torch.tensor([1.0, -1.0, 0.0])
        x = (groups * scale).reshape(-1).to(DTYPES[dtype])
        cfg = _cfg(bit=4, group_size=16, topk=topk, quant_type=quant_type)
        payload = oracle.encode(x, cfg)
        assert torch.equal(codec.quantize_tensor(x.cuda(), cfg).cpu(), payload), scale
        out = torch.empty_like(x).cuda()
        assert ext.roundtrip_general(x.cuda(), None, out, None, 16, 4, topk, codec._QUANT_CODE[quant_type], False, 0, 1)
        assert torch.equal(out.cpu().view(torch.uint8), oracle.decode(payload, x.numel(), cfg, dtype).view(torch.uint8)), scale


@pytest.mark.parametrize("quant_type", ("normal", "uniform", "e3m0", "e2m1"))
def test_codebook_codes_around_the_division_limit(ext, quant_type):
    """The corrected reciprocal serves scales below 1e30, a division the others: values at every threshold with scales
    next to the limit, and 16-bit sources (whose quotients round apart from the fp32 ones) on both sides of it."""

    table = oracle.codebook(quant_type)[:15]
    mids = table[:-1] + (table[1:] - table[:-1]) / 2
    around = torch.cat([mids, torch.nextafter(mids, mids - 1), torch.nextafter(mids, mids + 1), table])
    around = around[:around.numel() // 15 * 15].reshape(-1, 15)
    groups = torch.cat([torch.ones(around.shape[0], 1), around], dim=1)
    limit = torch.tensor(1.0e30)
    below, above = torch.nextafter(limit, torch.tensor(0.0)), torch.nextafter(limit, torch.tensor(2.0e30))
    cfg = _cfg(bit=4, group_size=16, quant_type=quant_type)
    for name, scales in (("fp32", (below, limit, above)), ("bf16", (0.9e30, 1.1e30, 1.7, 3e-7)), ("fp16", (1.7, 3e-7))):
        for scale in scales:
            x = (groups * scale).to(DTYPES[name]).reshape(-1)
            assert torch.equal(codec.quantize_tensor(x.cuda(), cfg).cpu(), oracle.encode(x, cfg)), (name, scale)


@pytest.mark.parametrize("dtype", ("bf16", "fp16"))
@pytest.mark.parametrize("topk", (0, 1))
def test_codebook_codes_in_a_group_whose_scale_is_nan(ext, dtype, topk):
    """More NaN than the group keeps: the scale is NaN, the codes are those of value / 1e-6 (the floor of a scale), as
    a division gives them, also where that overflows."""

    cfg = _cfg(bit=4, group_size=16, topk=topk, quant_type="e2m1")
    top = torch.finfo(DTYPES[dtype]).max
    x = torch.zeros(6 * 16)
    x[:64] = _data(64, torch.float32, seed=1)                        # finite groups in the same warp
    nan = [float("nan")] * (topk + 1)
    for g, body in ((4, [-float("inf"), float("inf"), -top, top, -0.25 * top, 0.0, -1e-7, 1e-7]), (5, [-1.0, 1.0, -5e-7])):
        x[16 * g:16 * g + len(nan) + len(body)] = torch.tensor(nan + body)
    x = x.to(DTYPES[dtype])
    table = oracle.codebook("e2m1")
    t = x.float() / torch.tensor(1e-6)
    low = (torch.searchsorted(table[:15].contiguous(), t, right=True) - 1).clamp_(0, 14)
    want = low + ((t - table[low]) > (table[low + 1] - table[low]) / 2).to(torch.int64)
    for g in (4, 5):
        want[16 * g:16 * g + topk] = 7                               # what is kept has the code of zero
    payload = codec.quantize_tensor(x.cuda(), cfg).cpu()
    codes = oracle._unpack_words(payload[:x.numel() // 2].reshape(-1, 8), 4, 2).reshape(-1)
    assert codes[64:].tolist() == want[64:].tolist()
    finite = oracle.encode(x[:64], cfg)
    assert torch.equal(payload[:32], finite[:32])


@pytest.mark.parametrize("dtype", list(DTYPES))
@pytest.mark.parametrize("bit,group,topk", [(8, 64, 0), (8, 16, 2), (4, 32, 1), (4, 64, 0)])
def test_compact_records_through_warp_spans(ext, dtype, bit, group, topk):
    """Payloads that start on 16 bytes move as a warp's span, others word by word; whole warps, ragged last warps,
    and ends in the middle of a vector."""

    cfg = _cfg(bit=bit, group_size=group, topk=topk, compact=True, quant_type="e2m1" if bit == 4 else "linear")
    for n in (512 * 9, 512 * 8 + group + 1, 3 * group, 1):
        x = _data(n, DTYPES[dtype], seed=n)
        want = oracle.encode(x, cfg)
        back = oracle.decode(want, n, cfg, dtype)
        for skew in (0, 4, 16):
            raw = torch.full((want.numel() + 64,), 0xA5, dtype=torch.uint8, device="cuda")
            payload = raw[skew:skew + want.numel()]
            codec.quantize_tensor(x.cuda(), cfg, output=payload)
            assert torch.equal(payload.cpu(), want), (n, skew)
            assert (raw[:skew] == 0xA5).all() and (raw[skew + want.numel():] == 0xA5).all()
            got = codec.dequantize_tensor(payload, (n,), cfg, dtype=dtype)
            assert torch.equal(got.cpu().view(torch.uint8), back.view(torch.uint8)), (n, skew)


@pytest.mark.parametrize("dtype", list(DTYPES))
@pytest.mark.parametrize("bit,quant_type,topk,group", [(8, "linear", 1, 64), (4, "linear", 2, 32), (4, "e3m0", 0, 16),
                                                       (4, "normal", 1, 64), (8, "linear", 2, 16)])
@pytest.mark.parametrize("passes", (1, 2))
def test_general_one_rank_pass_matches_the_codec(ext, dtype, bit, quant_type, topk, group, passes):
    """encode + decode in registers against a payload in memory: residual, unaligned views, special values (an
    all-NaN group among them), and buffers the pass declines."""

    cfg = _cfg(bit=bit, group_size=group, topk=topk, quant_type=quant_type)
    code = {"linear": 0, "normal": 1, "e3m0": 3}[quant_type]
    for n, skew in ((20_000, 0), (4096 + 5, 1), (1, 0), (3 * group, 8)):
        base = torch.empty(n + skew, dtype=DTYPES[dtype], device="cuda").normal_(std=1e-2)
        x = base[skew:]
        if n > 8 * group:
            x[group:group + 4] = x[group]
            x[2 * group:2 * group + 3] = torch.tensor([float("inf"), -float("inf"), float("nan")]).to(x)
            x[4 * group:5 * group] = float("nan")
            x[6 * group:7 * group] = 0
        r = torch.empty(n, dtype=x.dtype, device="cuda").normal_(std=1e-4)
        for residual in (None, r):
            prepared = torch.empty_like(x)
            cur = x
            for k in range(passes):
                payload = codec.quantize_tensor(cur, cfg, residual=residual if k == 0 else None,
                                                prepared_out=prepared if k == 0 else None)
                cur = codec.dequantize_tensor(payload, (n,), cfg, dtype=dtype)
            out = x.clone() if residual is None else torch.empty_like(x)
            rout = None if residual is None else residual.clone()
            src = out if residual is None else x
            assert ext.roundtrip_general(src, rout, out, rout, group, bit, topk, code, False, 0, passes)
            assert torch.equal(out.view(torch.uint8), cur.view(torch.uint8)), (n, residual is None)
            if residual is not None:
                want = torch.empty_like(x)
                codec.update_error_feedback_residual(prepared, cur.contiguous(), want)
                assert torch.equal(rout.view(torch.uint8), want.view(torch.uint8)), n
    both = torch.zeros(1000, dtype=DTYPES[dtype], device="cuda")
    assert not ext.roundtrip_general(both[:900], None, both[100:], None, group, bit, topk, code, False, 0, passes)
    assert not ext.roundtrip_general(both[:900], both[50:950], both[:900], None, group, bit, topk, code, False, 0, passes)


@pytest.mark.parametrize("dtype", list(DTYPES))
@pytest.mark.parametrize("bit,group,compact", [(8, 64, False), (8, 32, True), (4, 16, False), (4, 64, True)])
def test_codec_kernels_at_tile_edges(ext, dtype, bit, group, compact):
    """Encode (one and two chunks per thread), decode and the reduction of 1, 3, 4, 5 and 9 payloads: whole and ragged
    tiles, unaligned tensors, payloads that start on an odd vector, accumulation into the output."""

    cfg = _cfg(bit=bit, group_size=group, compact=compact)
    large = 4096 * int(ext.default_max_blocks()) + 4097
    for n, skew in ((large, 0), (8192, 0), (8192 + 4096 + 1, 0), (4095, 3), (2 * group + 1, 8)):
        base, rbase = _data(n + skew, DTYPES[dtype], seed=n).cuda(), _data(n + skew, DTYPES[dtype], seed=n + 1).cuda()
        x, r = base[skew:], rbase[skew:]
        for residual in (None, r):
            want = oracle.encode(x.cpu(), cfg, residual=None if residual is None else residual.cpu())
            raw = torch.full((want.numel() + 16,), 0xA5, dtype=torch.uint8, device="cuda")
            payload = raw[skew // 2 * 2:][:want.numel()] if dtype != "fp32" else raw[skew // 4 * 4:][:want.numel()]
            prepared = torch.empty_like(base)[skew:]
            codec.quantize_tensor(x, cfg, output=payload, residual=residual, prepared_out=prepared)
            assert torch.equal(payload.cpu(), want), (n, skew)
            assert torch.equal(prepared, oracle.prepare(x.cpu(), None if residual is None else residual.cpu()).cuda())
        if n == large:
            got = codec.dequantize_tensor(payload, (n,), cfg, dtype=dtype)
            assert torch.equal(got.cpu().view(torch.uint8), oracle.decode(want, n, cfg, dtype).view(torch.uint8))
            continue
        for count in (1, 3, 4, 5, 9):
            payloads = [oracle.encode(_data(n, DTYPES[dtype], seed=40 + k), cfg) for k in range(count)]
            dev = [p.cuda() for p in payloads[:-1]] + [payload.copy_(payloads[-1])]
            y, y32 = oracle.reduce_mean(payloads, n, cfg, dtype)
            out, rout = torch.empty_like(base)[skew:], torch.empty_like(base)[skew:]
            codec.inplace_dequantize_reduce_mean_update_error_feedback(dev, x, out, rout, cfg, reduce="mean")
            assert torch.equal(out.cpu().view(torch.uint8), y.view(torch.uint8)), (n, skew, count)
            assert torch.equal(rout.cpu().view(torch.uint8), oracle.residual_update(x.cpu(), y32).view(torch.uint8))
        total = x.clone()
        codec.dequantize_tensor(payload, (n,), cfg, dtype=dtype, output=total, reduce_op="sum")
        assert torch.equal(total.cpu(), oracle.decode_accumulate(payloads[-1], x.cpu(), cfg)), (n, skew)


@pytest.mark.parametrize("kw", [{}, {"topk": 1}, {"compact": True}])
def test_codec_takes_tensors_of_any_shape(ext, kw):
    """Shapes and strides at the entry points: the kernels see the elements in order, results have the asked shape."""

    cfg = _cfg(**kw)
    base = _data(48 * 130, torch.bfloat16).cuda()
    dense, strided = base.reshape(48, 130), base.reshape(130, 48).t()
    for x in (dense, strided, dense.reshape(4, 12, 130)):
        want = oracle.encode(x.cpu().contiguous(), cfg)
        payload = codec.quantize_tensor(x, cfg, residual=torch.zeros_like(x))
        assert torch.equal(payload.cpu(), want)
        back = oracle.decode(want, x.numel(), cfg, "bf16").reshape(x.shape)
        got = codec.dequantize_tensor(payload, x.shape, cfg, dtype="bf16")
        assert got.shape == x.shape and torch.equal(got.cpu(), back)
        into = torch.zeros(x.numel(), dtype=x.dtype, device="cuda")
        got = codec.dequantize_tensor(payload, x.shape, cfg, dtype="bf16", output=into, reduce_op="sum")
        assert got.shape == x.shape and got.data_ptr() == into.data_ptr() and torch.equal(got.cpu(), back)
        got = codec.dequantize_reduce_tensors([payload], x.shape, cfg, dtype="bf16", reduce="mean")
        assert got.shape == x.shape and torch.equal(got.cpu(), back)


@pytest.mark.parametrize("kw", [{}, {"topk": 1}, {"compact": True}, {"bit": 4, "quant_type": "normal"}])
def test_codec_takes_views_with_one_stride(ext, kw):
    """Every other element, one element repeated, a column: views whose flattened form is a view again."""

    cfg = _cfg(**kw)
    base = _data(6000, torch.bfloat16).cuda()
    for x in (base[::2], base[3::7], base[:1].expand(200), base.reshape(60, 100)[:, :1]):
        want = oracle.encode(x.cpu().contiguous(), cfg)
        assert torch.equal(codec.quantize_tensor(x, cfg).cpu(), want)
        assert torch.equal(codec.quantize_tensor(x, cfg, residual=torch.zeros(x.shape, dtype=x.dtype, device="cuda")).cpu(),
                           want)


@pytest.mark.parametrize("dtype", list(DTYPES))
@pytest.mark.parametrize("bit,group,compact", [(8, 64, False), (8, 16, True), (4, 32, False)])
@pytest.mark.parametrize("which", ("input", "residual", "prepared", "payload", "output", "all"))
def test_each_tensor_on_its_own_boundary(ext, dtype, bit, group, compact, which):
    """Encode, decode, reduction and the one-rank pass where one tensor starts 1 element, 4, 8 or 16 bytes past a
    32-byte boundary and the others on it: same results, and nothing written beside the outputs."""

    cfg = _cfg(bit=bit, group_size=group, compact=compact)
    T = DTYPES[dtype]
    width, edge = T.itemsize, 32 // T.itemsize
    sizes = (2 * 4096 + group + 5, 4096, 15)
    ranks = PeerGroup.loopback(1, FusedWorkspace.required_bytes(1, dtype, cfg, sizes[0], True) + (1 << 20))
    ws = FusedWorkspace(ranks[0], dtype=dtype, config=cfg, max_numel=sizes[0], engine="pipe")
    for n in sizes:
        x, r = _data(n, T, seed=n), _data(n, T, seed=n + 1, outliers=False)
        payload = oracle.encode(x, cfg, residual=r)
        prepared = oracle.prepare(x, r)
        y, y32 = oracle.reduce_mean([payload, payload, payload], n, cfg, dtype)
        once, once32 = oracle.reduce_mean([payload], n, cfg, dtype)
        left = oracle.residual_update(prepared, y32)
        for off in sorted({1, 4 // width, 8 // width, 16 // width}):
            held = []

            def place(values, name):
                at = edge + (off if which in (name, "all") else 0)
                raw = torch.full((n + 3 * edge,), 7.0, dtype=T, device="cuda")
                view = raw[at:at + n]
                if values is not None:
                    view.copy_(values)
                held.append((raw, at))
                return view

            def wire(values):
                at = 32 + (max(off * width, width) if which in ("payload", "all") else 0)
                raw = torch.full((payload.numel() + 96,), 0xA5, dtype=torch.uint8, device="cuda")
                if values is not None:
                    raw[at:at + payload.numel()] = values.cuda()
                return raw, raw[at:at + payload.numel()], at

            raw, to, at = wire(None)
            keep = place(None, "prepared")
            codec.quantize_tensor(place(x, "input"), cfg, output=to, residual=place(r, "residual"), prepared_out=keep)
            assert torch.equal(to.cpu(), payload) and torch.equal(keep.cpu(), prepared), (n, off)
            assert (raw[:at] == 0xA5).all() and (raw[at + payload.numel():] == 0xA5).all()
            out, res = place(None, "output"), place(None, "residual")
            codec.inplace_dequantize_reduce_mean_update_error_feedback(
                [wire(payload)[1], payload.cuda(), wire(payload)[1]], place(prepared, "prepared"), out, res, cfg,
                reduce="mean")
            assert torch.equal(out.cpu(), y) and torch.equal(res.cpu(), left), (n, off)
            out = place(None, "output")
            codec.dequantize_tensor(wire(payload)[1], (n,), cfg, dtype=dtype, output=out)
            assert torch.equal(out.cpu(), once), (n, off)
            if which != "payload":
                out, res = place(None, "output"), place(r, "residual")
                ws.all_reduce(place(x, "input"), out, residual=res)
                assert torch.equal(out.cpu(), once), (n, off)
                assert torch.equal(res.cpu(), oracle.residual_update(prepared, once32)), (n, off)
                same = place(x, "input")
                ws.all_reduce(same)
                assert torch.equal(same.cpu(), oracle.decode(oracle.encode(x, cfg), n, cfg, dtype)), (n, off)
            for raw, at in held:
                assert (raw[:at] == 7.0).all() and (raw[at + n:] == 7.0).all(), (n, off)
    PeerGroup.close_loopback(ranks)


def _repeated(base, n):
    """`base` over and over, n elements: a tensor of any size whose payload is the oracle's payload of `base`, repeated."""

    return base.repeat(-(-n // base.numel()))[:n]


def _repeated_payload(base, n, cfg, dtype):
    """The oracle's payload of `_repeated(base, n)`; `base` is whole groups."""

    groups, tail = n // cfg.group_size, n % cfg.group_size
    values, metas = oracle._split(oracle.encode(base, cfg), base.numel(), cfg, dtype)
    times = -(-groups // values.shape[0])
    values, metas = values.repeat(times, 1)[:groups], metas.repeat(times, 1)[:groups]
    if tail:
        at = groups * cfg.group_size % base.numel()
        last = oracle._split(oracle.encode(base[at:at + tail], cfg), tail, cfg, dtype)
        values, metas = torch.cat([values, last[0]]), torch.cat([metas, last[1]])
    if cfg.compact:
        return torch.cat([values, metas], dim=1).reshape(-1)
    return torch.cat([values.reshape(-1), metas.reshape(-1)])


@pytest.mark.parametrize("dtype", ("bf16", "fp32"))
@pytest.mark.parametrize("bit,quant_type,topk,group,compact", [
    (8, "linear", 1, 64, True), (8, "linear", 2, 16, False), (4, "linear", 2, 32, True), (4, "e2m1", 0, 64, True),
    (4, "normal", 1, 32, False)])
def test_general_kernels_on_a_grid_that_loops(ext, dtype, bit, quant_type, topk, group, compact):
    """Above four default grids the general kernels loop over one: the warp's staging area is used again and offsets grow.
    Whole result against the oracle, for the default grid and for three blocks; the last tile is ragged."""

    cfg = _cfg(bit=bit, group_size=group, topk=topk, quant_type=quant_type, compact=compact)
    code = codec._QUANT_CODE[quant_type]
    base = _data(group * 997, DTYPES[dtype], seed=11)
    base_dev = base.cuda()
    full = 4 * 4096 * int(ext.default_max_blocks())
    n = full + 5 * 4096 * 37 + group + 3
    x = _repeated(base_dev, n)
    want = _repeated_payload(base, n, cfg, dtype).cuda()
    once = oracle.decode(oracle.encode(base, cfg), base.numel(), cfg, dtype)
    decoded = _repeated(once.cuda(), n)
    # the last group is ragged: its scale is that of the elements it has
    tail = n % group
    at = (n - tail) % base.numel()
    ends = oracle.decode(oracle.encode(base[at:at + tail], cfg), tail, cfg, dtype)
    decoded[n - tail:] = ends.cuda()
    assert torch.equal(codec.quantize_tensor(x, cfg), want)
    back = codec.dequantize_tensor(want, (n,), cfg, dtype=dtype)
    assert torch.equal(back.view(torch.uint8), decoded.view(torch.uint8))
    total = codec.dequantize_tensor(want, (n,), cfg, dtype=dtype, output=back, reduce_op="sum")
    assert torch.equal(total, (decoded.float() * 2).to(decoded.dtype))
    small = 3 * 4096 * 5 + group + 3
    for numel, blocks in ((n, 0), (small, 3)):
        expect = decoded[:numel].clone()
        ragged = numel % group
        at = (numel - ragged) % base.numel()
        expect[numel - ragged:] = oracle.decode(oracle.encode(base[at:at + ragged], cfg), ragged, cfg, dtype).cuda()
        out = torch.empty_like(x[:numel])
        assert ext.roundtrip_general(x[:numel].clone(), None, out, None, group, bit, topk, code, False, 0, 1, blocks)
        assert torch.equal(out.view(torch.uint8), expect.view(torch.uint8))
        payload = codec.quantize_tensor(x[:numel], cfg)
        ext.reduce_general([payload.data_ptr()] * 2, out, group, bit, topk, code, compact, 0.5, None, None, None, blocks)
        half = ((expect.float() * 2).to(out.dtype).float() * 0.5).to(out.dtype)
        assert torch.equal(out, half)


@pytest.mark.parametrize("dtype", list(DTYPES))
@pytest.mark.parametrize("bit,quant_type,topk,group", [(8, "linear", 0, 64), (8, "linear", 1, 32), (4, "linear", 2, 16),
                                                       (4, "normal", 0, 64), (4, "e3m0", 1, 32), (4, "uniform", 2, 16)])
def test_stochastic_one_rank_pass_matches_the_codec(ext, dtype, bit, quant_type, topk, group):
    """The same seed gives the same numbers in registers and through a payload; another seed gives others; and the payload
    is the oracle's, bit for bit, for the counter-based numbers of `uniform01`."""

    cfg = _cfg(bit=bit, group_size=group, topk=topk, quant_type=quant_type, stochastic=True)
    code = codec._QUANT_CODE[quant_type]
    # (a fused product and sum would give another code for one value in 2^17: the first size has several of those)
    for n, skew in ((2_000_000 // group * group, 0), (4096 + 5, 1), (group, 8)):
        x = torch.empty(n + skew, dtype=DTYPES[dtype], device="cuda").normal_(std=1e-2)[skew:]
        r = torch.empty(n, dtype=x.dtype, device="cuda").normal_(std=1e-4)
        results = []
        for seed in (12345, 2**61 + 7):
            payload, prepared = codec.allocate_quantized_buffer(x, cfg), torch.empty_like(x)
            ext.quant_general(x, r, prepared, payload, group, bit, topk, code, True, False, seed)
            want = codec.dequantize_tensor(payload, (n,), cfg, dtype=dtype)
            out, rout = torch.empty_like(x), r.clone()
            assert ext.roundtrip_general(x, rout, out, rout, group, bit, topk, code, True, seed, 1)
            assert torch.equal(out.view(torch.uint8), want.view(torch.uint8))
            left = torch.empty_like(x)
            codec.update_error_feedback_residual(prepared, want, left)
            assert torch.equal(rout.view(torch.uint8), left.view(torch.uint8))
            results.append(out)
            if n % group == 0:
                noise = torch.from_numpy(_uniform01(seed, n)) - 0.5
                expect = oracle.encode(x.cpu(), cfg, residual=r.cpu(), noise=noise)
                assert torch.equal(payload.cpu(), expect)
        assert n < 1000 or not torch.equal(*results)


def _uniform01(seed, n):
    """The kernels' uniform numbers in (0, 1] by element index."""

    z = np.uint64(seed) + np.uint64(0x9E3779B97F4A7C15) * np.arange(1, n + 1, dtype=np.uint64)
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    z ^= z >> np.uint64(31)
    return ((z >> np.uint64(40)).astype(np.float32) + np.float32(1)) * np.float32(2.0**-24)


@pytest.mark.parametrize("dtype", list(DTYPES))
@pytest.mark.parametrize("bit,quant_type,topk,group", [(8, "linear", 1, 64), (4, "linear", 2, 32), (4, "e3m0", 0, 16),
                                                       (4, "uniform", 1, 64), (8, "linear", 2, 16)])
def test_general_one_rank_pass_matches_the_oracle(ext, dtype, bit, quant_type, topk, group):
    """Both pass counts and the residual against the oracle, beside groups with infinities and NaN (which the oracle does
    not define; the finite groups of the same warp are compared)."""

    cfg = _cfg(bit=bit, group_size=group, topk=topk, quant_type=quant_type)
    code = codec._QUANT_CODE[quant_type]
    n = 40 * group + 7
    x, r = _data(n, DTYPES[dtype], seed=2), _data(n, DTYPES[dtype], seed=3, outliers=False)
    finite = torch.ones(n, dtype=torch.bool)
    special = x.clone()
    special[2 * group:2 * group + 3] = torch.tensor([float("inf"), -float("inf"), float("nan")]).to(x)
    special[4 * group:5 * group] = float("nan")
    finite[2 * group:3 * group] = finite[4 * group:5 * group] = False
    for passes in (1, 2):
        y = prepared = oracle.prepare(x, r)
        for _ in range(passes):
            y = oracle.decode(oracle.encode(y, cfg), n, cfg, dtype)
        left = oracle.residual_update_from_restored(prepared, y)
        for source, mask in ((x, torch.ones_like(finite)), (special, finite)):
            out, rout = torch.empty_like(x).cuda(), r.cuda()
            assert ext.roundtrip_general(source.cuda(), rout, out, rout, group, bit, topk, code, False, 0, passes)
            assert torch.equal(out.cpu()[mask].view(torch.uint8), y[mask].view(torch.uint8)), passes
            assert torch.equal(rout.cpu()[mask].view(torch.uint8), left[mask].view(torch.uint8)), passes


@pytest.mark.parametrize("dtype", list(DTYPES))
@pytest.mark.parametrize("bit,group,compact", [(8, 64, False), (8, 32, True), (4, 16, True)])
@pytest.mark.parametrize("skew", (0, 1))
def test_codec_kernels_on_a_capped_grid(ext, dtype, bit, group, compact, skew):
    """`max_blocks` below the tiles: every block goes round several times, aligned and unaligned, whole and ragged ends."""

    cfg = _cfg(bit=bit, group_size=group, compact=compact)
    code = codec._DTYPE_CODE[dtype]
    for n in (7 * 4096 + group + 3, 6 * 4096):
        base, rbase = _data(n + skew, DTYPES[dtype], seed=n), _data(n + skew, DTYPES[dtype], seed=n + 1, outliers=False)
        x, r = base.cuda()[skew:], rbase.cuda()[skew:]
        groups = -(-n // group)
        want = oracle.encode(base[skew:], cfg, residual=rbase[skew:])
        plain = oracle.encode(base[skew:], cfg)
        for residual, expect in ((r, want), (None, plain)):
            payload = torch.zeros(want.numel(), dtype=torch.uint8, device="cuda")
            ext.quant_push(x, residual, None, None, [payload.data_ptr()],
                           ext.PUSH_COMPACT_LOCAL if compact else ext.PUSH_BROADCAST, 0, groups, 0, group, bit, None, 2)
            assert torch.equal(payload.cpu(), expect)
        for count in (1, 5):
            dev = [want.cuda() if k % 2 else plain.cuda() for k in range(count)]
            y, y32 = oracle.reduce_mean([d.cpu() for d in dev], n, cfg, dtype)
            out, res = torch.empty_like(rbase).cuda()[skew:], torch.empty_like(rbase).cuda()[skew:]
            ext.reduce([d.data_ptr() for d in dev], groups, 0, compact, n, code, group, bit, 1.0 / count, out, False, x, res,
                       [], 0, 0, None, None, 2)
            assert torch.equal(out.cpu(), y) and torch.equal(res.cpu(), oracle.residual_update(base[skew:], y32))
        ext.reduce([payload.data_ptr()], groups, 0, compact, n, code, group, bit, 1.0, out, False, None, None, [], 0, 0, None,
                   None, 2)
        assert torch.equal(out.cpu(), oracle.decode(plain, n, cfg, dtype))


@pytest.mark.parametrize("dtype", list(DTYPES))
@pytest.mark.parametrize("kw", [{}, {"compact": True}, {"topk": 1}, {"bit": 4, "quant_type": "e2m1", "compact": True}])
def test_payloads_off_their_words_are_refused(ext, dtype, kw):
    """A payload view that starts between two words of the source's width: an error before any launch."""

    cfg = _cfg(**kw)
    x = _data(640, DTYPES[dtype]).cuda()
    need = codec.allocate_quantized_buffer(x, cfg).numel()
    raw = torch.zeros(need + 8, dtype=torch.uint8, device="cuda")
    for off in (1, 3) if dtype != "fp32" else (1, 2, 3):
        view, out, res = raw[off:off + need], torch.zeros_like(x), torch.zeros_like(x)
        with pytest.raises(RuntimeError, match="multiple of"):
            codec.quantize_tensor(x, cfg, output=view)
        with pytest.raises(RuntimeError, match="multiple of"):
            codec.dequantize_tensor(view, x.shape, cfg, dtype=dtype, output=out)
        with pytest.raises(RuntimeError, match="multiple of"):
            codec.dequantize_reduce_update_error_feedback([view], x, res, x.shape, cfg, dtype=dtype)
        torch.cuda.synchronize()
        assert not out.any() and not res.any() and not raw.any()
    view = raw[4:4 + need]
    codec.quantize_tensor(x, cfg, output=view)
    assert torch.equal(view.cpu(), oracle.encode(x.cpu(), cfg))


@pytest.mark.parametrize("kw", [{}, {"topk": 1}])
def test_tensors_that_the_kernels_cannot_address_are_refused(ext, kw):
    """Payloads in pageable host memory, and outputs or residuals of a collective that are not like its tensor: errors
    before any launch; pinned payloads stay served where the kernels take an address."""

    import torch.distributed as dist

    from lowbit_comm_b200.parallel.communicator import Communicator

    cfg = _cfg(**kw)
    x = _data(640, torch.bfloat16).cuda()
    payload = codec.quantize_tensor(x, cfg)
    with pytest.raises(ValueError, match="on the GPU"):
        codec.quantize_tensor(x, cfg, output=torch.empty(payload.numel(), dtype=torch.uint8))
    out, res = torch.zeros_like(x), torch.zeros_like(x)
    with pytest.raises(ValueError, match="on the GPU"):
        codec.inplace_dequantize_reduce_mean([payload.cpu(), payload], out, cfg) or codec.dequantize_reduce_update_error_feedback(
            [payload, payload.cpu()], x, res, x.shape, cfg, dtype="bf16")
    if not kw:
        pinned = torch.empty(payload.numel(), dtype=torch.uint8).pin_memory()
        codec.quantize_tensor(x, cfg, output=pinned)
        assert codec.inplace_dequantize_reduce_mean([pinned], out, cfg)
        torch.cuda.synchronize()
        assert torch.equal(pinned, payload.cpu())
        assert torch.equal(out, codec.dequantize_tensor(payload, x.shape, cfg, dtype="bf16"))
    created = not dist.is_initialized()
    if created:
        dist.init_process_group("nccl", store=dist.HashStore(), rank=0, world_size=1, device_id=torch.device("cuda", 0))
    comm = Communicator(None)
    try:
        before = x.clone()
        for wrong in (torch.zeros(640), torch.zeros(640, device="cuda"), torch.zeros(639, dtype=x.dtype, device="cuda"),
                      torch.zeros(640, 2, dtype=x.dtype, device="cuda")[:, 0]):
            if wrong.is_contiguous() or not kw:      # (general profiles: a strided out takes the torch path)
                with pytest.raises(ValueError, match="out must be"):
                    comm.all_reduce(x, config=cfg, out=wrong)
            if wrong.is_contiguous() or not kw:      # (there a strided residual is copied in and out)
                with pytest.raises(ValueError, match="residual must be"):
                    comm.all_reduce(x, config=cfg, residual=wrong)
        assert torch.equal(x, before)
        if kw:
            strided, dense = torch.zeros(640, 2, dtype=x.dtype, device="cuda")[:, 0], torch.zeros_like(x)
            strided.fill_(1e-4)
            dense.fill_(1e-4)
            out2 = torch.zeros_like(x)
            comm.all_reduce(x, config=cfg, out=out, residual=dense)
            comm.all_reduce(x, config=cfg, out=out2, residual=strided)
            assert torch.equal(out, out2) and torch.equal(strided, dense) and not torch.equal(dense, torch.full_like(dense, 1e-4))
        good = torch.zeros(32, 20, dtype=x.dtype, device="cuda")
        comm.all_reduce(x, config=cfg, out=good, residual=res)
        assert torch.equal(good.reshape(-1), codec.dequantize_tensor(payload, x.shape, cfg, dtype="bf16"))
    finally:
        comm.close()
        if created:
            dist.destroy_process_group()


@pytest.mark.parametrize("dtype", list(DTYPES))
@pytest.mark.parametrize("bit,quant_type,topk,group", [(8, "linear", 1, 64), (8, "linear", 2, 16), (4, "linear", 1, 32),
                                                       (4, "e2m1", 1, 64), (4, "normal", 2, 32)])
@pytest.mark.parametrize("case", ("ties", "sparse", "minus zero", "tiny", "all"))
def test_one_rank_pass_whichever_of_equal_magnitudes_is_kept(ext, dtype, bit, quant_type, topk, group, case):
    """The pass keeps what is above the scale and looks for the places only where that could matter: equal magnitudes around the
    last kept one, groups with fewer non-zero elements than are kept, zeros of both signs, scales below the clamp."""

    cfg = _cfg(bit=bit, group_size=group, topk=topk, quant_type=quant_type)
    n = 96 * group + 5
    x = _data(n, torch.float32, seed=9)
    for g in range(0, 96, 3):                                        # groups of every kind side by side in a warp
        part = x[g * group:(g + 1) * group]
        if case in ("ties", "all"):
            top = part.abs().max()
            part[1] = top
            part[group // 2] = -top
            if g % 2:
                part[group - 1] = top
                part[3] = top
        if case == "sparse" or (case == "all" and g % 2):
            part[:] = 0
            part[g % group] = 0.25 if g % 4 else 0.0
        if case == "minus zero" or (case == "all" and g % 5 == 0):
            part[:] = 0
            part[2 + g % 7] = -0.0
            part[9] = 1e-3 if g % 2 else -0.0
        if case == "tiny" or (case == "all" and g % 7 == 0):
            part[:] = 0
            part[4:8] = torch.tensor([2e-7, -2e-7, 1e-7, 3e-7 if g % 2 else 2e-7])
    x = x.to(DTYPES[dtype])
    y = x
    for passes in (1, 2):
        y = oracle.decode(oracle.encode(y, cfg), n, cfg, dtype)
        out = torch.empty_like(x).cuda()
        assert ext.roundtrip_general(x.cuda(), None, out, None, group, bit, topk, codec._QUANT_CODE[quant_type], False, 0, passes)
        assert torch.equal(out.cpu().view(torch.uint8), y.view(torch.uint8)), passes


@pytest.mark.parametrize("kw", [{}, {"compact": True}, {"topk": 1}, {"bit": 4, "quant_type": "e2m1"}])
@pytest.mark.parametrize("n,skew", [(4099, 0), (300_001, 1), (3 << 20, 0)])
def test_kernels_in_a_row_wait_for_each_other(ext, kw, n, skew):
    """Kernels start while the one ahead of them still runs: calls that read what the call before wrote, in place and through
    other buffers, beside kernels of torch, alone and captured in a graph, against the same calls one at a time."""

    cfg = _cfg(**kw)
    first = _data(n + skew, torch.bfloat16, seed=7).cuda()
    state = {"x": first.clone()[skew:], "r": torch.zeros(n, dtype=torch.bfloat16, device="cuda"),
             "y": torch.empty(n, dtype=torch.bfloat16, device="cuda")}
    state["p"] = codec.quantize_tensor(state["x"], cfg)

    def chain(pause):
        for _ in range(3):
            for call in (lambda: codec.quantize_tensor(state["x"], cfg, output=state["p"], residual=state["r"], prepared_out=state["r"]),
                         lambda: codec.dequantize_tensor(state["p"], (n,), cfg, dtype="bf16", output=state["y"]),
                         lambda: state["x"].add_(state["y"], alpha=0.25),
                         lambda: codec.quantize_tensor(state["x"], cfg, output=state["p"]),
                         lambda: codec.dequantize_tensor(state["p"], (n,), cfg, dtype="bf16", output=state["y"], reduce_op="sum"),
                         lambda: state["x"].copy_(state["y"])):
                call()
                if pause:
                    torch.cuda.synchronize()

    def restart():
        state["x"].copy_(first[skew:])
        state["r"].zero_()
        state["y"].zero_()

    restart()
    chain(pause=True)
    want = {name: t.clone() for name, t in state.items()}
    for _ in range(5):
        restart()
        chain(pause=False)
        assert all(torch.equal(t, want[name]) for name, t in state.items())
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.graph(graph, stream=stream):
        restart()
        chain(pause=False)
    for _ in range(5):
        graph.replay()
        assert all(torch.equal(t, want[name]) for name, t in state.items())


@pytest.mark.parametrize("dtype", list(DTYPES))
@pytest.mark.parametrize("kw", [{}, {"compact": True}, {"topk": 2}, {"bit": 4, "quant_type": "e3m0", "compact": True}])
def test_native_codec_calls_and_the_general_way(ext, dtype, kw, monkeypatch):
    """The calls that settle everything natively give what the general way gives, for every form of argument that they take, and
    leave the others to it: the same calls with the native ones taken away."""

    from lowbit_comm_b200.ops.loader import load_cuda_extension

    cfg, torch_dtype, other = _cfg(**kw), DTYPES[dtype], "fp16" if dtype == "fp32" else "fp32"
    size = lambda n: codec.estimate_quantized_size(n, dtype=dtype, config=cfg).quantized_bytes
    base = _data(3 * 4160, torch_dtype, seed=4).cuda()
    bytes_ = torch.zeros(2 * size(4160) + 8, dtype=torch.uint8, device="cuda")
    x, r = base[:4099], base[4160:8259] * 0.01
    whole = codec.quantize_tensor(x, cfg)
    around = torch.full((4099, 2), 3.0, dtype=torch_dtype, device="cuda")     # every second element belongs to nobody
    scattered = around[:, 0]
    outer, square = torch.full((64, 128), 3.0, dtype=torch_dtype, device="cuda"), base[:4096].view(64, 64)
    inner = outer[:, :64]
    encodes = {
        "plain": lambda: codec.quantize_tensor(x, cfg),
        "shaped": lambda: codec.quantize_tensor(base[:4096].view(16, 256), cfg),
        "view off its vectors": lambda: codec.quantize_tensor(base[1:4100], cfg),
        "transposed": lambda: codec.quantize_tensor(base[:4096].view(64, 64).t(), cfg),
        "one stride": lambda: codec.quantize_tensor(base[:8198:2], cfg),
        "empty": lambda: codec.quantize_tensor(base[:0], cfg),
        "residual": lambda: codec.quantize_tensor(x, cfg, residual=r),
        "strided residual": lambda: codec.quantize_tensor(x, cfg, residual=base[:8198:2]),
        "output": lambda: codec.quantize_tensor(x, cfg, output=bytes_[4:4 + size(4099)]),
        "output off its words": lambda: codec.quantize_tensor(x, cfg, output=bytes_[1:1 + size(4099)]),
        "output too small": lambda: codec.quantize_tensor(x, cfg, output=bytes_[:8]),
        "output of floats": lambda: codec.quantize_tensor(x, cfg, output=r),
        "residual of another type": lambda: codec.quantize_tensor(x, cfg, residual=r.to(DTYPES[other])),
        "residual too short": lambda: codec.quantize_tensor(x, cfg, residual=r[:-1]),
        "residual on the host": lambda: codec.quantize_tensor(x, cfg, residual=r.cpu()),
        "whole numbers": lambda: codec.quantize_tensor(torch.ones(64, dtype=torch.int32, device="cuda"), cfg),
        "strided prepared": lambda: (codec.quantize_tensor(square, cfg, residual=r[:4096], prepared_out=inner), outer.clone())[1],
        "prepared with one stride": lambda: codec.quantize_tensor(x, cfg, residual=r, prepared_out=scattered),
        "prepared": lambda: torch.cat([codec.quantize_tensor(x, cfg, residual=r, prepared_out=(p := torch.empty_like(x))).float(), p.float()]),
    }
    decodes = {
        "plain": lambda: codec.dequantize_tensor(whole, (4099,), cfg, dtype=dtype),
        "a list": lambda: codec.dequantize_tensor(whole, [4099, 1], cfg, dtype=dtype),
        "a size": lambda: codec.dequantize_tensor(whole, x.shape, cfg, dtype=dtype),
        "floats": lambda: codec.dequantize_tensor(whole, (4099.0,), cfg, dtype=dtype),
        "an iterator": lambda: codec.dequantize_tensor(whole, np.array([4099]), cfg, dtype=dtype),
        "negative": lambda: codec.dequantize_tensor(whole, (-4099, -1), cfg, dtype=dtype),
        "empty": lambda: codec.dequantize_tensor(bytes_[:0], (0, 3), cfg, dtype=dtype),
        "beyond 64 bits": lambda: codec.dequantize_tensor(whole, (1 << 70,), cfg, dtype=dtype),
        "below 64 bits": lambda: codec.dequantize_tensor(whole, [-(1 << 70), 1], cfg, dtype=dtype),
        "output": lambda: codec.dequantize_tensor(whole, (4099,), cfg, dtype=dtype, output=torch.empty_like(x)),
        "output of another shape": lambda: codec.dequantize_tensor(whole, (1, 4099), cfg, dtype=dtype, output=torch.empty_like(x)),
        "output of another type": lambda: codec.dequantize_tensor(whole, (4099,), cfg, dtype=dtype, output=torch.empty_like(x, dtype=DTYPES[other])),
        "strided output": lambda: codec.dequantize_tensor(whole, (4099,), cfg, dtype=dtype, output=scattered),
        "strided payload": lambda: codec.dequantize_tensor(torch.stack([whole, whole], 1)[:, 0], (4099,), cfg, dtype=dtype),
        "sum": lambda: codec.dequantize_tensor(whole, (4099,), cfg, dtype=dtype, output=r.clone(), reduce_op="sum"),
        "payload too short": lambda: codec.dequantize_tensor(whole[:-2], (4099,), cfg, dtype=dtype),
        "unknown type": lambda: codec.dequantize_tensor(whole, (4099,), cfg, dtype="int8"),
        "unknown reduction": lambda: codec.dequantize_tensor(whole, (4099,), cfg, dtype=dtype, reduce_op="max"),
        "type of its own": lambda: codec.dequantize_tensor(whole, (4099,), cfg, dtype="auto"),
    }

    def outcome(call):
        try:
            result = call()
        except Exception as error:  # noqa: BLE001
            return type(error)
        return result.shape, result.dtype, result.contiguous().view(torch.uint8).cpu().numpy().tobytes()

    def every_outcome():
        around.fill_(3.0)
        outer.fill_(3.0)
        got = {("encode", name): outcome(call) for name, call in encodes.items()}
        got.update({("decode", name): outcome(call) for name, call in decodes.items()})
        want = oracle.prepare(x[:4096].cpu(), r[:4096].cpu()).view(64, 64)
        assert torch.equal(inner.cpu(), want) and bool((outer[:, 64:] == 3.0).all())
        assert bool((around == 3.0).all())                       # strided outputs of one dimension are refused untouched
        assert got["decode", "strided output"] is ValueError and got["decode", "strided payload"] is ValueError
        return got

    native = every_outcome()
    taken = {"encode": 0, "decode": 0}

    class General:
        def __getattr__(self, name):
            return getattr(ext, name)

        def codec_encode(self, *args):
            taken["encode"] += ext.codec_encode(*args) is not None

        def codec_decode(self, *args):
            taken["decode"] += ext.codec_decode(*args) is not None

    monkeypatch.setattr(codec, "require_extension", lambda status=None: General())
    assert load_cuda_extension().available
    general = every_outcome()
    assert {name for name in native if native[name] != general[name]} == set()
    assert taken["encode"] >= 5 and taken["decode"] >= 4


@pytest.mark.parametrize("dtype", list(DTYPES))
@pytest.mark.parametrize("bit,quant_type,topk,group,compact", [
    (8, "linear", 1, 64, False), (8, "linear", 2, 16, True), (4, "linear", 1, 32, True), (4, "normal", 0, 16, False),
    (4, "e2m1", 2, 64, True), (4, "uniform", 1, 32, False)])
def test_general_encode_at_tile_edges(ext, dtype, bit, quant_type, topk, group, compact):
    """Sizes around a block's 4096 elements, each tensor on and off its vectors, payloads on 16, 8 and 4 bytes: the kernel of whole
    tiles, its last tile and the kernel of payloads off their vectors."""

    cfg = _cfg(bit=bit, group_size=group, topk=topk, quant_type=quant_type, compact=compact)
    for n in (4096 - 1, 4096, 4096 + 1, 3 * 4096 + group + 5, 2 * 4096 - group, 7):
        x, r = _data(n, DTYPES[dtype], seed=n), _data(n, DTYPES[dtype], seed=n + 1, outliers=False)
        want, prepared = oracle.encode(x, cfg, residual=r), oracle.prepare(x, r)
        for where, skew in ((0, (0, 0, 0)), (16, (16, 0, 0)), (8, (1, 0, 0)), (4, (0, 3, 0)), (0, (0, 0, 8)), (16, (5, 1, 2))):
            at = [torch.zeros(n + 16, dtype=DTYPES[dtype], device="cuda")[s:s + n] for s in skew]
            at[0].copy_(x)
            at[1].copy_(r)
            raw = torch.full((want.numel() + 48,), 0xAB, dtype=torch.uint8, device="cuda")
            codec.quantize_tensor(at[0], cfg, output=raw[where:where + want.numel()], residual=at[1], prepared_out=at[2])
            assert torch.equal(raw[where:where + want.numel()].cpu(), want), (n, where, skew)
            assert bool((raw[:where] == 0xAB).all()) and bool((raw[where + want.numel():] == 0xAB).all())
            assert torch.equal(at[2].cpu().view(torch.uint8), prepared.view(torch.uint8)), (n, where, skew)


@pytest.mark.parametrize("dtype", ("bf16", "fp32"))
@pytest.mark.parametrize("kw", [{}, {"compact": True}, {"bit": 4, "group_size": 16}, {"topk": 1}, {"topk": 2, "compact": True},
                                {"bit": 4, "quant_type": "e2m1"}])
@pytest.mark.parametrize("n,skew", [(2 * 4096, 0), (4099, 1), (150_001, 0)])
def test_only_codec_and_one_rank_calls_in_a_row(ext, dtype, kw, n, skew):
    """Rows of calls with no kernel of another library between them, small enough that three and more are on the GPU at once: a
    payload decoded, written anew and decoded again, one-rank passes in place, a mean of several payloads; every call
    reads what the one before it wrote.  Alone and captured in a graph, against the same calls one at a time."""

    cfg, T, rounds = _cfg(**kw), DTYPES[dtype], 4
    fast = codec.is_fast_profile(cfg)
    grads = [_data(n, T, seed=i).cuda() for i in range(rounds)]
    size = codec.estimate_quantized_size(n, dtype=dtype, config=cfg).quantized_bytes
    held = lambda: torch.empty(n + skew, dtype=T, device="cuda")[skew:]
    x, a, b, c = ([held() for _ in range(rounds)] for _ in range(4))
    residual, prepared = held(), held()
    p, q = (torch.empty(size, dtype=torch.uint8, device="cuda") for _ in range(2))
    ranks = PeerGroup.loopback(1, FusedWorkspace.required_bytes(1, dtype, cfg, n, True) + (1 << 20)) if fast else []
    ws = FusedWorkspace(ranks[0], dtype=dtype, config=cfg, max_numel=n, engine="pipe") if fast else None

    def one_rank(t):
        if fast:
            ws.all_reduce(t, t, residual=residual)
        else:
            assert ext.roundtrip_general(t, residual, t, residual, cfg.group_size, cfg.bit, cfg.topk,
                                         codec._QUANT_CODE[cfg.quant_type], False, 0, 1)

    def row(pause):
        for i in range(rounds):
            for call in (lambda: codec.quantize_tensor(x[i], cfg, output=p),
                         lambda: codec.dequantize_tensor(p, (n,), cfg, dtype=dtype, output=a[i]),
                         lambda: codec.quantize_tensor(a[i], cfg, output=p, residual=residual, prepared_out=residual),
                         lambda: codec.dequantize_tensor(p, (n,), cfg, dtype=dtype, output=b[i]),
                         lambda: one_rank(b[i]),
                         lambda: one_rank(b[i]),
                         lambda: codec.quantize_tensor(b[i], cfg, output=q, residual=residual, prepared_out=prepared),
                         lambda: codec.dequantize_tensor(q, (n,), cfg, dtype=dtype, output=x[i]),
                         lambda: codec.dequantize_tensor(p, (n,), cfg, dtype=dtype, output=c[i]),
                         lambda: codec.inplace_dequantize_reduce_mean_update_error_feedback([p, q, p], prepared, c[i], residual,
                                                                                            cfg, reduce="mean"),
                         lambda: codec.dequantize_tensor(q, (n,), cfg, dtype=dtype, output=c[i], reduce_op="sum")):
                call()
                if pause:
                    torch.cuda.synchronize()

    def restart():
        for i in range(rounds):
            x[i].copy_(grads[i])
            for t in (a[i], b[i], c[i]):
                t.zero_()
        residual.zero_()
        prepared.zero_()

    def everything():
        return [t.clone() for t in (*x, *a, *b, *c, residual, prepared, p, q)]

    restart()
    row(pause=True)
    want = everything()
    for _ in range(5):
        restart()
        row(pause=False)
        assert all(torch.equal(t, w) for t, w in zip(everything(), want))
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.graph(graph, stream=stream):
        restart()
        row(pause=False)
    for _ in range(5):
        graph.replay()
        assert all(torch.equal(t, w) for t, w in zip(everything(), want))
    # payloads and results that are allocated by the calls: the allocator gives the same addresses again and again
    alone = [codec.dequantize_tensor(codec.quantize_tensor(g, cfg), (n,), cfg, dtype=dtype).cpu() for g in grads]
    for _ in range(5):
        results = [codec.dequantize_tensor(codec.quantize_tensor(g, cfg), (n,), cfg, dtype=dtype) for g in grads * 3]
        assert all(torch.equal(r.cpu(), w) for r, w in zip(results, alone * 3))
    PeerGroup.close_loopback(ranks)


@pytest.mark.parametrize("bit,quant_type,group", [(8, "linear", 64), (4, "linear", 16), (4, "e2m1", 32)])
@pytest.mark.parametrize("past", (0, 1, 4096))
def test_fp32_one_rank_pass_where_its_blocks_per_sm_change(ext, bit, quant_type, group, past):
    """One kept value: up to three blocks per SM in all, and above, with and without a residual, against the codec."""

    cfg = _cfg(bit=bit, group_size=group, topk=1, quant_type=quant_type)
    n = int(ext.default_max_blocks()) // 8 * 3 * 4096 + past
    x = _repeated(_data(group * 997, torch.float32, seed=5).cuda(), n).clone()
    for residual in (None, torch.full_like(x, 1e-4)):
        prepared = torch.empty_like(x)
        payload = codec.quantize_tensor(x, cfg, residual=residual, prepared_out=prepared)
        want = codec.dequantize_tensor(payload, (n,), cfg, dtype="fp32")
        out, rout = torch.empty_like(x), None if residual is None else residual.clone()
        assert ext.roundtrip_general(x, rout, out, rout, group, bit, 1, codec._QUANT_CODE[quant_type], False, 0, 1)
        assert torch.equal(out.view(torch.uint8), want.view(torch.uint8))
        if residual is not None:
            left = torch.empty_like(x)
            codec.update_error_feedback_residual(prepared, want, left)
            assert torch.equal(rout.view(torch.uint8), left.view(torch.uint8))


@pytest.mark.parametrize("kw", [{"topk": 1}, {"bit": 4, "quant_type": "e2m1", "compact": True}])
@pytest.mark.parametrize("where", (0, 4))
def test_a_general_payload_of_this_gpu_raises_its_signal(ext, kw, where):
    """The C entry takes a signal without destinations too: raised once the payload is stored, wherever that starts."""

    import ctypes

    from lowbit_comm_b200.ops.build import extension_path

    class Signal(ctypes.Structure):
        _fields_ = [("remote_flags", ctypes.c_void_p * 16), ("num_remote", ctypes.c_int), ("my_slot", ctypes.c_int),
                    ("epoch", ctypes.c_uint), ("block_counter", ctypes.c_void_p)]

    class Encode(ctypes.Structure):
        _fields_ = [*((name, ctypes.c_int) for name in ("dtype", "group_size", "bit", "topk", "quant_type", "stochastic", "compact")),
                    ("x", ctypes.c_void_p), ("residual", ctypes.c_void_p), ("prepared_out", ctypes.c_void_p),
                    ("numel", ctypes.c_int64), ("out", ctypes.c_void_p), ("seed", ctypes.c_ulonglong),
                    ("dst", ctypes.c_void_p * 16), ("num_dst", ctypes.c_int), ("signal", Signal), ("max_blocks", ctypes.c_int),
                    ("shard_groups", ctypes.c_int64), ("book", ctypes.c_uint32 * 47)]

    cfg, n = _cfg(**kw), 3 * 4096 + 5
    x = _data(n, torch.bfloat16).cuda()
    want = oracle.encode(x.cpu(), cfg)
    raw = torch.zeros(want.numel() + 16, dtype=torch.uint8, device="cuda")
    flags, counter = torch.zeros(8, dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    call = Encode(dtype=1, group_size=cfg.group_size, bit=cfg.bit, topk=cfg.topk, quant_type=codec._QUANT_CODE[cfg.quant_type],
                  compact=cfg.compact, x=x.data_ptr(), numel=n, out=raw.data_ptr() + where)
    call.signal = Signal(num_remote=1, my_slot=3, epoch=7, block_counter=counter.data_ptr())
    call.signal.remote_flags[0] = flags.data_ptr()
    lib = ctypes.CDLL(str(extension_path()))
    lib.lbc_quant_general.argtypes = [ctypes.POINTER(Encode), ctypes.c_void_p]
    assert lib.lbc_quant_general(ctypes.byref(call), torch.cuda.current_stream().cuda_stream) == 0
    assert torch.equal(raw[where:where + want.numel()].cpu(), want)
    assert flags.tolist() == [0, 0, 0, 7, 0, 0, 0, 0] and counter.item() == 0


@pytest.mark.parametrize("dtype", list(DTYPES))
@pytest.mark.parametrize("bit,group,compact", [(8, 64, False), (8, 16, True), (4, 32, False)])
@pytest.mark.parametrize("n", (4096, 4096 * 3 + 513, 5_000_000))
def test_linear_codes_of_scales_that_need_the_clamp(ext, dtype, bit, group, compact, n):
    """Groups with an infinity, a NaN or a scale around 1e30 (where the quotient goes another way) between ordinary ones,
    in the first, a middle and the last tile, one and two chunks per thread: a NaN (an infinity times zero) gets the lowest
    code, as the clamp gives it.  Every operation is one rounding, so the bytes are the same."""

    cfg = CompressionConfig(bit=bit, group_size=group, compact=compact, allow_experimental=True)
    T, lim, inf = DTYPES[dtype], 127.0 if bit == 8 else 7.0, float("inf")
    x = _data(n, T, seed=11)
    edge = torch.tensor([1e30 if dtype != "fp16" else 6e4], dtype=T).view(torch.int32 if dtype == "fp32" else torch.int16)
    sizes = [(edge + k).view(T).item() for k in (-1, 0, 1)] + [torch.finfo(T).max, torch.finfo(T).smallest_normal, 1e-6]
    for at in (0, (n // 2) // 512 * 512 + 64, (n - 1) // 512 * 512 - 1024):
        for k, size in enumerate(sizes):                # one group of a warp each, its neighbours untouched
            x[at + 2 * k * group % 512:][:3] = torch.tensor([size, -size, size / 3]).to(T)
        x[at + 512:][:3] = torch.tensor([inf, 1.0, float("nan")]).to(T)
        x[at + 512 + group:][:2] = torch.tensor([float("nan"), -2.0]).to(T)
    values = oracle._grouped(x, group).float()
    stored = torch.nan_to_num(values.abs(), nan=0.0, posinf=inf).amax(1).to(T)
    t = values * (torch.tensor(lim) / stored.float().clamp_min(1e-6))[:, None]      # (a number / tensor takes two roundings)
    codes = torch.where(t.isnan(), -lim, t.round().clamp(-lim, lim)).to(torch.int64) & (255 if bit == 8 else 15)
    words = oracle._pack_words(codes, bit, x.element_size())
    scales = stored.view(torch.uint8).reshape(len(stored), -1)
    want = torch.cat([words, scales], 1).reshape(-1) if compact else torch.cat([words.reshape(-1), scales.reshape(-1)])
    finite = x.isfinite()
    assert torch.equal(codec.quantize_tensor(x.cuda(), cfg).cpu(), want)
    r = torch.zeros_like(x).cuda()
    prepared = torch.empty_like(r)
    assert torch.equal(codec.quantize_tensor(x.cuda(), cfg, residual=r, prepared_out=prepared).cpu(), want)
    assert torch.equal(prepared.cpu()[finite], x[finite]) and bool((prepared.cpu().isnan() == x.isnan()).all())
    wide = torch.empty(n + 1, dtype=T, device="cuda")    # one element in: the kernel of unaligned tensors
    wide[1:].copy_(x)
    assert torch.equal(codec.quantize_tensor(wide[1:], cfg).cpu(), want)


@pytest.mark.parametrize("dtype", list(DTYPES))
@pytest.mark.parametrize("bit,quant_type,topk,group", [(8, "linear", 1, 64), (4, "linear", 2, 16), (4, "e2m1", 0, 32), (4, "normal", 1, 64)])
def test_one_rank_pass_without_a_residual(ext, dtype, bit, quant_type, topk, group):
    """The forms of the pass that only encode and decode: a tile per block, and blocks that go round with their next tile under way,
    which a cap on the blocks and the sizes where they begin bring in; whole and ragged ends, tensors off their vectors, in
    place.  Beside them infinities, NaN and a scale above 1e30 (fp16: the largest), whose warps take the clamp: in finite groups the
    bytes are the oracle's."""

    cfg, code = _cfg(bit=bit, group_size=group, topk=topk, quant_type=quant_type), codec._QUANT_CODE[quant_type]
    edge = int(ext.default_max_blocks()) * 4096 // (2 if quant_type != "linear" and topk == 0 else 1)
    large = () if dtype == "fp16" else ((edge, 0, 0), (edge + 4099, 0, 0))
    for n, blocks, skew in ((1, 0, 0), (4096, 0, 0), (8191, 1, 0), (4096 * 3 + 17, 2, 0), (4096 * 7, 2, 0), (4096 * 5 + 1, 3, 1)) + large:
        x = _data(n, DTYPES[dtype], seed=n % 97)
        finite = torch.ones(n, dtype=torch.bool)
        if n > 2000:
            x[group:group + 3] = torch.tensor([torch.finfo(x.dtype).max, -torch.finfo(x.dtype).max / 2, 1.0]).to(x)
            x[20 * group:20 * group + 2] = torch.tensor([float("inf"), float("nan")]).to(x)
            x[n - 1] = float("nan")
            finite[20 * group:21 * group] = False
            finite[(n - 1) // group * group:] = False
        want = oracle.decode(oracle.encode(torch.where(finite, x, torch.zeros_like(x)), cfg), n, cfg, dtype)
        for in_place in (False, True):
            source = torch.empty(n + skew, dtype=x.dtype, device="cuda")[skew:]
            source.copy_(x)
            out = source if in_place else torch.empty_like(source)
            assert ext.roundtrip_general(source, None, out, None, group, bit, topk, code, False, 0, 1, blocks)
            assert torch.equal(out.cpu()[finite].view(torch.uint8), want[finite].view(torch.uint8)), (n, blocks, skew, in_place)


@pytest.mark.parametrize("dtype", ("bf16", "fp32"))
@pytest.mark.parametrize("bit,quant_type,topk,compact", [(8, "linear", 1, False), (8, "linear", 2, True), (4, "linear", 2, False), (4, "e2m1", 0, False),
                                                        (4, "e2m1", 0, True), (4, "normal", 1, True)])
def test_general_codec_where_its_kernels_change(ext, dtype, bit, quant_type, topk, compact):
    """Encode without a residual, and decode, on both sides of the sizes from which other kernels serve them (halves of the default
    grid), whole and ragged."""

    cfg = _cfg(bit=bit, quant_type=quant_type, topk=topk, compact=compact)
    half = int(ext.default_max_blocks()) // 2 * 4096
    for n in (half // 2 - 7, half // 2 + 4096, half - 1, half + 4096, 2 * half, 2 * half + 7, 3 * half, 4 * half + 1, 5 * half + 3):
        x = _data(n, DTYPES[dtype], seed=n % 89)
        want = oracle.encode(x, cfg)
        assert torch.equal(codec.quantize_tensor(x.cuda(), cfg).cpu(), want), n
        got = codec.dequantize_tensor(want.cuda(), (n,), cfg, dtype=dtype)
        assert torch.equal(got.cpu().view(torch.uint8), oracle.decode(want, n, cfg, dtype).view(torch.uint8)), n


@pytest.mark.parametrize("dtype", list(DTYPES))
@pytest.mark.parametrize("bit,group,compact", [(8, 64, False), (8, 16, True), (4, 32, False)])
def test_own_error_on_both_sides_of_one_grid(ext, dtype, bit, group, compact):
    """Encode with this rank's own quantization error (one rounding, then the rounding to the type): the kernel of small and unaligned
    tensors, and the one that takes aligned 16-bit ones above one default grid, whole, ragged and on a capped grid; the error in place of
    the residual, and an infinity whose warp takes the clamp."""

    cfg, T, lim = _cfg(bit=bit, group_size=group, compact=compact), DTYPES[dtype], 127.0 if bit == 8 else 7.0
    edge = int(ext.default_max_blocks()) * 4096
    for n, blocks in ((edge, 0), (edge + 4096, 0), (edge + 4099, 0), (edge + 8192 + 5, 700)):
        x = _data(n, T, seed=n % 83)
        r = (_data(n, T, seed=n % 79, outliers=False) * 1e-3).to(T)
        x[n // 3] = float("inf")
        prepared = oracle.prepare(x, r)
        values = oracle._grouped(prepared, group).float()
        scale = values.abs().amax(1).to(T).float()
        t = values * (torch.tensor(lim) / scale.clamp_min(1e-6))[:, None]
        codes = torch.where(t.isnan(), -lim, t.round().clamp(-lim, lim))       # (infinity times zero: the clamp's lowest code)
        words = oracle._pack_words(codes.to(torch.int64) & (255 if bit == 8 else 15), bit, x.element_size())
        scales = scale.to(T).view(torch.uint8).reshape(len(scale), -1)
        want = torch.cat([words, scales], 1).reshape(-1) if compact else torch.cat([words.reshape(-1), scales.reshape(-1)])
        left = (values.double() - codes.double() * (scale / torch.tensor(lim))[:, None].double()).float().to(T).reshape(-1)[:n]
        finite = torch.ones(n, dtype=torch.bool)
        finite[n // 3 // group * group:(n // 3 // group + 1) * group] = False
        for skew in (0, 1):
            source = torch.empty(n + skew, dtype=T, device="cuda")[skew:]
            source.copy_(x)
            residual, payload = r.cuda(), torch.zeros(want.numel(), dtype=torch.uint8, device="cuda")
            ext.quant_push(source, residual, None, residual, [payload.data_ptr()],
                           ext.PUSH_COMPACT_LOCAL if compact else ext.PUSH_BROADCAST, 0, -(-n // group), 0, group, bit, None, blocks)
            assert torch.equal(payload.cpu(), want), (n, skew)
            got = residual.cpu()
            assert torch.equal(got[finite].view(torch.uint8), left[finite].view(torch.uint8)), (n, skew)
            assert bool(got[~finite].float().isnan().any()) or bool((~got[~finite].float().isfinite()).any())


@pytest.mark.parametrize("group", (16, 32, 64))
def test_fp32_records_in_four_bits_where_their_kernels_change(ext, group):
    """Decode on both sides of a sixteenth, three eighths and the whole of a default grid, whole and ragged."""

    cfg, full = _cfg(bit=4, group_size=group, compact=True), int(ext.default_max_blocks()) * 4096
    for n in (full // 16, full // 16 + 5, full // 8 * 3 - 4096, full // 8 * 3, full // 8 * 3 + 1, full, full + 9):
        x = _data(n, torch.float32, seed=n % 73)
        payload = oracle.encode(x, cfg)
        got = codec.dequantize_tensor(payload.cuda(), (n,), cfg, dtype="fp32")
        assert torch.equal(got.cpu().view(torch.uint8), oracle.decode(payload, n, cfg, "fp32").view(torch.uint8)), n


@pytest.mark.parametrize("dtype", list(DTYPES))
@pytest.mark.parametrize("bit,group,compact", [(8, 64, False), (8, 16, True), (4, 32, True)])
def test_sums_that_are_added_to_the_output(ext, dtype, bit, group, compact):
    """One payload and several, with and without error feedback, whole and ragged ends, aligned tensors and views: T(sum) is added to what the
    output holds, one rounding; the residual is that of the sum alone."""

    cfg, T = _cfg(bit=bit, group_size=group, compact=compact), DTYPES[dtype]
    for n in (group, 4096 * 2, 4096 * 3 + group + 5):
        payloads = [oracle.encode(_data(n, T, seed=k), cfg) for k in range(5)]
        held, prepared = _data(n, T, seed=11), _data(n, T, seed=12)
        for count in (1, 2, 5):
            y, y32 = oracle.reduce_mean(payloads[:count], n, cfg, dtype)
            want = (held.float() + y.float()).to(T)
            for feedback in (False, True):
                for skew in (0, 1):
                    out = torch.empty(n + skew, dtype=T, device="cuda")[skew:]
                    out.copy_(held)
                    dev, res = [p.cuda() for p in payloads[:count]], torch.empty(n, dtype=T, device="cuda")
                    ext.reduce([d.data_ptr() for d in dev], -(-n // group), 0, compact, n, codec._DTYPE_CODE[dtype], group, bit, 1.0 / count, out, True,
                               prepared.cuda() if feedback else None, res if feedback else None, [], 0, 0, None, None, 0)
                    assert torch.equal(out.cpu(), want), (n, count, feedback, skew)
                    assert not feedback or torch.equal(res.cpu(), oracle.residual_update(prepared, y32)), (n, count, skew)


@pytest.mark.parametrize("dtype", list(DTYPES))
@pytest.mark.parametrize("bit", (8, 4))
def test_quotients_over_the_range_of_scales(ext, dtype, bit):
    """The encoder multiplies by L / scale and the decoder by scale / L, both rounded correctly without a division: every scale of the
    16-bit types from 1e-6 to 1e30 and one in 1021 of fp32, each with values whose products lie beside the halves between two codes, where a
    quotient one step off gives another code."""

    cfg, T, lim, group = _cfg(bit=bit, group_size=16), DTYPES[dtype], 127.0 if bit == 8 else 7.0, 16
    if dtype == "fp32":
        ends = torch.tensor([1e-6, 1e30]).view(torch.int32).tolist()
        scale = torch.arange(ends[0], ends[1] + 1021, 1021, dtype=torch.int32).view(T)
    else:
        scale = torch.arange(1 << 15, dtype=torch.int32).to(torch.int16).view(T)
        scale = scale[(scale.float() >= 1e-6) & (scale.float() <= 1e30)]
    mul = torch.tensor(lim) / scale.float()
    at = torch.linspace(0.0, lim - 1, 15).round() + 0.5
    values = (at * torch.tensor([1.0, -1.0]).repeat(8)[:15] / mul.double()[:, None]).float().to(T)
    x = torch.cat([scale[:, None], torch.minimum(torch.maximum(values, -scale[:, None]), scale[:, None])], 1)
    codes = (x.float() * mul[:, None]).round().clamp(-lim, lim)
    want = (codes * (scale.float() / torch.tensor(lim))[:, None]).to(T)
    payload = codec.quantize_tensor(x.reshape(-1).cuda(), cfg)
    got = codec.dequantize_tensor(payload, (x.numel(),), cfg, dtype=dtype).cpu().reshape(x.shape)
    wrong = (got + 0.0 != want + 0.0).any(1)                       # (a code 0 is +0)
    assert not bool(wrong.any()), (int(wrong.sum()), scale[wrong][:4], x[wrong][:1], got[wrong][:1], want[wrong][:1])
