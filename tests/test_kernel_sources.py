"""Rules of the kernels that reading their source shows (no GPU, no compiler)."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "lowbit_comm_b200" / "ops" / "csrc"
CHAINED = sorted(p.name for p in CSRC.glob("*.cu") if "launch_chained(" in p.read_text())


def _code(name):
    return re.sub(r"//[^\n]*", "", (CSRC / name).read_text())


def test_the_files_with_chained_kernels_are_known():
    assert CHAINED == ["codec_kernels.cu", "general_kernels.cu", "roundtrip_kernels.cu"]


@pytest.mark.parametrize("name", CHAINED + ["codec_device.cuh"])
def test_kernels_that_start_early_read_with_plain_loads(name):
    """A chained kernel is on the GPU while the one ahead of it writes what it will read.  Loads through the read-only path are no
    part of the memory model, so its wait says nothing of what they see."""

    assert re.findall(r"ld\w*_stream|__ldg|__ldlu|\.nc\b|__restrict__", _code(name)) == []
    bodies = [b for b in re.split(r"\n__global__", _code(name))[1:] if "chain_wait();" in b.split("\n}\n")[0]]
    for body in bodies:
        assert "load16<" not in body.split("\n}\n")[0]          # (takes the read-only path where its last argument says so)


@pytest.mark.parametrize("name", CHAINED)
def test_chained_kernels_wait_before_they_touch_memory(name):
    """Every kernel that is launched early waits in its first statements, and no kernel waits without need."""

    code = _code(name)
    launched = set(re.findall(r"launch_chained\((\w+)<", code))
    kernels = {}
    for body in re.split(r"\n__global__", code)[1:]:
        head, _, rest = body.partition(") {\n")
        kernels[re.findall(r"(\w+)\(const", head)[-1]] = [line.strip() for line in rest.split("\n")[:3]]
    assert launched <= set(kernels)
    for kernel, first in kernels.items():
        waits = [i for i, line in enumerate(first) if line == "chain_wait();"]
        assert bool(waits) == (kernel in launched), kernel
        assert all(line.startswith("constexpr") for line in first[:waits[0] if waits else 0]), kernel
