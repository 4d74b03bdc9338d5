"""State that calls share: modules imported on first use, memoized sizes and geometry."""

import dataclasses
import subprocess
import sys

import numpy as np
import pytest
import torch

from lowbit_comm_b200 import CompressionConfig, estimate_quantized_size, quantize_tensor
from lowbit_comm_b200.parallel.fused import geometry

FIRST_USE = r"""
import importlib.machinery, sys, threading, time
from lowbit_comm_b200.parallel.collectives._routes import communicator_module

NAME = "lowbit_comm_b200.parallel.communicator"
started, found, failed = threading.Event(), [], []


class Slow:
    # the module's own loader, with a pause between its entry in sys.modules and its body
    def __init__(self, loader): self.loader = loader
    def __getattr__(self, name): return getattr(self.loader, name)
    def create_module(self, spec): return self.loader.create_module(spec)
    def exec_module(self, module):
        started.set()
        time.sleep(0.5)
        self.loader.exec_module(module)


class Finder:
    @staticmethod
    def find_spec(name, path, target=None):
        if name != NAME:
            return None
        spec = importlib.machinery.PathFinder.find_spec(name, path)
        spec.loader = Slow(spec.loader)
        return spec


def first_call():
    try:
        found.append(communicator_module().get_communicator)
    except Exception as exc:
        failed.append(repr(exc))


assert NAME not in sys.modules
sys.meta_path.insert(0, Finder)
threads = [threading.Thread(target=first_call) for _ in range(8)]
threads[0].start()
assert started.wait(60)
for t in threads[1:]: t.start()
for t in threads: t.join()
assert not failed, failed
assert len(found) == 8 and len(set(found)) == 1
replaced = type(sys)(NAME)
sys.modules[NAME] = replaced            # as an import statement, a later look sees what is in sys.modules
assert communicator_module() is replaced
"""


def test_threads_that_make_their_first_collective_wait_for_the_import():
    done = subprocess.run([sys.executable, "-c", FIRST_USE], capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]


@pytest.mark.parametrize("first", (float, np.int64, np.int32, np.array, bool))
def test_memoized_sizes_keep_the_types_of_each_caller(first):
    """Sizes that are equal but of another type are other keys: what one caller asks for changes nothing for the next."""

    numel = 1 if first is bool else 640 + len(first.__name__)
    config = CompressionConfig()
    estimate_quantized_size(first(numel), dtype="bf16", config=config)
    geometry(first(numel), 2, "bf16", config)
    estimate_quantized_size(numel, dtype="bf16", config=CompressionConfig(bit=8.0, group_size=np.float64(64)))
    geometry(numel, np.int64(2), "bf16", CompressionConfig(group_size=64.0))
    estimate, shape = estimate_quantized_size(numel, dtype="bf16", config=config), geometry(numel, 2, "bf16", config)
    for value in (*dataclasses.asdict(estimate).values(), *dataclasses.asdict(shape).values()):
        assert type(value) in (int, float, str), value
    assert type(estimate.quantized_bytes) is int and type(estimate.numel) is int and type(shape.shard_groups) is int
    payload = quantize_tensor(torch.randn(numel, dtype=torch.bfloat16), config)
    assert payload.numel() == estimate.quantized_bytes
