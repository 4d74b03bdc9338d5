"""Whole native calls of a group of one rank against the general way through the communicator and the hook."""

import pytest
import torch
import torch.distributed as dist

from lowbit_comm_b200 import (CompressionConfig, compressed_all_gather, compressed_all_reduce,
                              compressed_reduce_scatter_shard, create_ddp_comm_hook)
from lowbit_comm_b200.parallel.communicator import Communicator, get_communicator, shutdown_communicators
from lowbit_comm_b200.parallel.fused import FusedWorkspace
from lowbit_comm_b200.parallel.fused_general import GeneralPeerWorkspace

pytestmark = pytest.mark.gpu

DT = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


@pytest.fixture(scope="module", autouse=True)
def one_rank(ext):
    created = not dist.is_initialized()
    if created:
        dist.init_process_group("nccl", store=dist.HashStore(), rank=0, world_size=1, device_id=torch.device("cuda", 0))
    yield
    shutdown_communicators()
    if created:
        dist.destroy_process_group()


class Marked(torch.Tensor):
    pass


class _Counted:
    """A native plan that notes which of its entries served a call, and which declined."""

    def __init__(self, plan, seen):
        self.plan, self.seen = plan, seen

    def __getattr__(self, name):
        def call(*args):
            result = getattr(self.plan, name)(*args)
            self.seen.append((name, result is not None and result is not False))
            return result

        return call


@pytest.fixture
def native(monkeypatch):
    """[(entry, did it serve the call?)] of all calls that the native plans saw."""

    seen = []
    for workspace in (FusedWorkspace, GeneralPeerWorkspace):
        def plans(self, plain=workspace.one_rank_plans):
            return tuple(p if p is None else _Counted(p, seen) for p in plain(self))

        monkeypatch.setattr(workspace, "one_rank_plans", plans)
    return seen


def _plain(value):
    if isinstance(value, torch.Tensor):
        return type(value), value.dtype, tuple(value.shape), value.contiguous().view(torch.uint8).cpu()
    if isinstance(value, list):
        return [_plain(v) for v in value]
    return _plain(value.shard), value.to_metadata()


def _same(a, b):
    if isinstance(a, torch.Tensor):
        return torch.equal(a, b)
    if isinstance(a, (tuple, list)):
        return len(a) == len(b) and all(_same(p, q) for p, q in zip(a, b))
    return a == b


def _outcome(call, *tensors):
    try:
        return _plain(call()), [_plain(t) for t in tensors]
    except Exception as exc:  # noqa: BLE001 - the two ways must refuse alike
        return type(exc), str(exc)


@pytest.mark.parametrize("dtype", list(DT))
@pytest.mark.parametrize("kw", [{}, {"bit": 4, "group_size": 16}, {"topk": 1}, {"bit": 4, "quant_type": "e2m1", "topk": 2}])
def test_native_one_rank_calls_and_the_general_way(dtype, kw, monkeypatch, native):
    """Sizes around a group and a tile, views, strides, outputs, residuals, overlaps, other classes, empty tensors, arguments
    that are refused: results, what is written, types and errors are the same.  The native entries serve the dense ones that fit,
    and decline or never see the others."""

    cfg = CompressionConfig(error_feedback=True, allow_experimental=True, **kw)
    comm, T = get_communicator(), DT[dtype]
    base = (torch.randn(40_000, generator=torch.Generator().manual_seed(3)) * 1e-2).to(T).cuda()
    base[700:706] = torch.tensor([float("inf"), float("nan"), 0.0, -0.0, 1e-7, -1e-7], device="cuda").to(T)
    comm.all_reduce(base.clone(), config=cfg)                      # the workspaces are there
    compressed_all_gather(base, config=cfg)

    def fresh(at, n):
        return base.clone()[at:at + n]

    inputs = [lambda n=n, at=at: fresh(at, n) for n in (1, 15, 64, 511, 512, 4096, 4097, 20_001) for at in (0, 1)]
    inputs += [lambda: fresh(0, 4096).reshape(64, 64)]
    dense = len(inputs)
    inputs += [lambda: fresh(0, 4096).reshape(64, 64).t(), lambda: fresh(0, 4096)[::2],
               lambda: fresh(0, 0), lambda: fresh(0, 640).as_subclass(Marked), lambda: fresh(0, 640).double(),
               lambda: fresh(0, 640).cpu(), lambda: base.repeat(3)]
    oversized = len(inputs) - 1                                    # its first call makes a larger workspace
    calls = [lambda x: compressed_all_reduce(x, config=cfg, strategy="auto"),
             lambda x: compressed_all_reduce(x, config=cfg, op="sum", strategy="reduce_scatter"),
             lambda x: comm.all_reduce(x, config=cfg, strategy="ring"),
             lambda x: comm.all_reduce(x, config=cfg, strategy="nowhere"),
             lambda x: compressed_reduce_scatter_shard(x, config=cfg),
             lambda x: compressed_all_gather(x, config=cfg)]
    linear = not (cfg.topk or cfg.quant_type != "linear")
    entry = ["one_rank"] * 3 + [None] + (["one_rank_shard", "one_rank_gather"] if linear else [None] * 2)
    for at, make in enumerate(inputs):
        for which, call in enumerate(calls):
            x = make()
            if x.is_cuda is False:
                continue                                            # (CPU tensors need a CPU group)
            native.clear()
            got = _outcome(lambda: call(x), x.as_subclass(torch.Tensor))
            name = entry[which]
            if name is None or (at >= dense and at != oversized):
                assert not any(ok for _, ok in native), (at, which, native)
            elif at < dense:
                assert native == [(name, True)], (at, which, native)
            elif which < 2:
                assert native == [(name, which == 1)], (which, native)
            y = make()
            with monkeypatch.context() as m:
                m.setattr(Communicator, "_one_rank_workspace", lambda *a: None)
                want = _outcome(lambda: call(y), y.as_subclass(torch.Tensor))
            assert _same(got, want), (x.shape, calls.index(call), got, want)
    pairs = [lambda x: {"out": torch.empty_like(x)}, lambda x: {"residual": torch.full_like(x, 1e-3)},
             lambda x: {"residual": torch.full_like(x, 1e-3), "update_residual": False},
             lambda x: {"residual": torch.full_like(x, 1e-3), "ef_mode": "local", "out": torch.empty_like(x)},
             lambda x: {"residual": torch.full_like(x, 1e-3), "ef_mode": "other"},
             lambda x: {"residual": torch.full((x.numel() + 1,), 1e-3, dtype=T, device="cuda")},
             lambda x: {"out": torch.empty(x.shape, dtype=torch.float64, device="cuda")},
             lambda x: {"residual": x}, lambda x: {"out": x}, lambda x: {"out": x._base[8:8 + x.numel()]},
             lambda x: {"residual": x._base[8:8 + x.numel()]}]
    for n in (1, 4097):
        for which, extra in enumerate(pairs):
            sides = []
            for general in (False, True):
                x = fresh(0, n)
                more = extra(x)
                native.clear()
                with monkeypatch.context() as m:
                    if general:
                        m.setattr(Communicator, "_one_rank_workspace", lambda *a: None)
                    sides.append(_outcome(lambda: comm.all_reduce(x, config=cfg, **more), x,
                                          *[v for v in more.values() if isinstance(v, torch.Tensor)]))
                if not general:
                    apart = which not in (9, 10) or n <= 8
                    want = [] if which == 4 else [("one_rank", which not in (5, 6, 7) and apart)]
                    assert native == want, (n, which, native)
            if which != 10 or n <= 8:              # (two results that overlap: whichever is written last)
                assert _same(*sides), (n, which, sides)


class _Bucket:
    def __init__(self, flat):
        self.flat = flat

    index = staticmethod(lambda: 0)
    is_last = staticmethod(lambda: True)
    parameters = staticmethod(lambda: [])

    def buffer(self):
        return self.flat


@pytest.mark.parametrize("dtype", list(DT))
@pytest.mark.parametrize("ef_mode", ("reference", "local"))
def test_a_bucket_in_one_native_call(dtype, ef_mode, monkeypatch, native):
    """The bucket is reduced behind what its stream holds, the future hands the buffer out on whichever stream waits for it, and
    residuals of several steps are those of the general way."""

    cfg = CompressionConfig(error_feedback=True, target="ddp_gradient_bucket")
    steps = [(torch.randn(300_001, generator=torch.Generator().manual_seed(s)) * 1e-2).to(DT[dtype]) for s in range(3)]
    results = []
    for general in (False, True):
        hook = create_ddp_comm_hook(cfg, strategy="auto", ef_mode=ef_mode)
        with monkeypatch.context() as m:
            if general:
                m.setattr(FusedWorkspace, "one_rank_plans", lambda self: (None, None))
            for step in steps:
                flat = torch.zeros(300_001, dtype=DT[dtype], device="cuda")
                torch.cuda._sleep(2_000_000)                        # the gradient arrives late on the producing stream
                flat.copy_(step, non_blocking=True)
                future = hook(None, _Bucket(flat))
                assert isinstance(future, torch.futures.Future) and future.done()
                other = torch.cuda.Stream()
                with torch.cuda.stream(other):
                    future.wait()
                    seen = future.value().clone()
                    assert future.value() is flat
                torch.cuda.current_stream().wait_stream(other)
                results.append((seen.cpu(), hook.feedback.get(0).cpu()))
        assert hook.gpu_launches() == 3 and hook.stats["peer"] == 3
        assert native == [("one_rank_bucket", True)] * 3            # (the general way sees no plan)
        torch.cuda.synchronize()
    for (a, ra), (b, rb) in zip(results[:3], results[3:]):
        assert torch.equal(a.view(torch.uint8), b.view(torch.uint8)) and torch.equal(ra.view(torch.uint8), rb.view(torch.uint8))
