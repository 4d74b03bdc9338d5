"""Rules of the kernels that their source shows, or what the compiler printed when it built them (no GPU)."""

import re
import shutil
import subprocess
from pathlib import Path

import pytest

from lowbit_comm_b200.ops import build

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
    rest = _code(name)                                     # without the kernels that are not chained: these, and what they call
    for body in re.split(r"\n__global__", rest)[1:]:
        body = body.split("\n}\n")[0]
        if "chain_wait();" not in body:
            rest = rest.replace(body, "")
    assert "load16<" not in rest                           # (takes the read-only path where its last argument says so)


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


def test_a_chained_kernel_waits_before_it_lets_the_next_one_start():
    """Otherwise a kernel two places behind starts beside the first, and what it reads ahead of its own wait may not be written yet."""

    body = _code("common.cuh").split("void chain_wait() {")[1].split("}")[0]
    assert re.findall(r"griddepcontrol\.(\w+)", body) == ["wait", "launch_dependents"]
    for path in CSRC.glob("*.cu*"):
        assert path.name == "common.cuh" or "griddepcontrol" not in _code(path.name)


def test_code_books_take_no_vote_for_linear_codes():
    """Whether linear codes may go without a clamp is one vote per chunk, and it waits for the group's scale.  The compiler keeps a vote whose
    result nobody reads, so the code-book kernels must not ask."""

    code = _code("general_kernels.cu")
    body = code.split("bool all_near(", 1)[1].split("\n}\n")[0]
    assert re.search(r"return !Kind<KIND>::book && __all_sync\(", body)
    assert len(re.findall(r"all_near<KIND>\(", code)) == 3 and "all_near(m)" not in code


def test_a_pad_that_no_tile_would_write_is_refused():
    """The one-rank pass clears a shard's pad with the tile that the tensor ends in, so behind whole tiles (and with nothing to
    encode) no block would.  Refused before anything is launched: the addresses here belong to nobody."""

    import ctypes

    torch = pytest.importorskip("torch")      # (the extension links against its libraries)
    assert torch is not None
    if not build.extension_path().exists():
        pytest.skip("the extension was not built here")

    class Roundtrip(ctypes.Structure):
        _fields_ = [*((name, ctypes.c_int) for name in ("dtype", "group_size", "bit")),
                    *((name, ctypes.c_void_p) for name in ("x", "residual", "out", "residual_out")), ("numel", ctypes.c_int64),
                    *((name, ctypes.c_int) for name in ("passes", "own_error", "max_blocks", "pad"))]

    lib = ctypes.CDLL(str(build.extension_path()))
    lib.lbc_roundtrip.argtypes = [ctypes.POINTER(Roundtrip), ctypes.c_void_p]
    invalid = 1
    for group in (16, 32, 64):
        for numel, pad in ((0, 64), (8 * group, 8), (4096, 512), (3 * 8192, 1), (8 * group, -1)):
            call = Roundtrip(dtype=1, group_size=group, bit=8, x=1 << 20, out=1 << 24, numel=numel, passes=1, pad=pad)
            assert lib.lbc_roundtrip(ctypes.byref(call), None) == invalid, (group, numel, pad)
    empty = Roundtrip(dtype=1, group_size=64, bit=8, x=1 << 20, out=1 << 24, numel=0, passes=1)
    assert lib.lbc_roundtrip(ctypes.byref(empty), None) == 0


def _plain_names(mangled):
    names = subprocess.run(["c++filt"], input="\n".join(mangled), capture_output=True, text=True, check=True).stdout.split("\n")
    return [re.sub(r"\((int|bool)\)", "", name.replace("void lbc::", "")).split("(Lbc")[0] for name in names]


def _spill_loads(source):
    """Kernel (with its template arguments) -> bytes of spill loads, from the last build."""

    report = build.ptxas_report(source)
    if not report.exists() or shutil.which("c++filt") is None:
        pytest.skip("the extension was not built here")
    pairs = re.findall(r"Function properties for (\S+)\n.*?(\d+) bytes spill loads", report.read_text())
    return {name: int(loads) for name, (_, loads) in zip(_plain_names([name for name, _ in pairs]), pairs)}


def test_decode_kernels_keep_their_registers():
    """A payload's scale is divided ahead of its sixteen codes: the other way round they live across the division, and these sums
    were 10872 and 5388 bytes.  The limits are what nvcc 12.9 gives (5840 and 352) and a quarter more."""

    loads = _spill_loads("codec_kernels.cu")
    one = [v for k, v in loads.items() if k.startswith("decode_kernel<") and k.endswith(", 1>")]
    ragged = [v for k, v in loads.items() if k.startswith("decode_ragged_kernel<")]
    assert len(one) == 36 and len(ragged) == 72
    assert sum(one) <= 7300 and sum(ragged) <= 440


def _registers(source):
    report = build.ptxas_report(source)
    if not report.exists() or shutil.which("c++filt") is None:
        pytest.skip("the extension was not built here")
    pairs = re.findall(r"Function properties for (\S+)\n.*\n.*?Used (\d+) registers", report.read_text())
    return dict(zip(_plain_names([name for name, _ in pairs]), (int(n) for _, n in pairs)))


def test_kernels_that_plain_calls_run_keep_their_registers():
    """Decodes of one payload, reductions of several, one-rank passes without a residual.  Only the decodes with eight blocks per SM (32
    registers) spill, nearly all of it for the end tile: 10460 bytes of spill loads in sum, 492 in the worst one, of which 56 and 8 are left
    when they are compiled without it.  The limits are what nvcc 12.9 gives and a quarter more."""

    loads = _spill_loads("codec_kernels.cu")
    eight = [v for k, v in loads.items() if k.startswith("decode_one_kernel<") and k.endswith(", 8>")]
    five = [v for k, v in loads.items() if k.startswith("decode_one_kernel<") and k.endswith(", 5>")]
    several = [v for k, v in loads.items() if k.startswith("decode_several_kernel<")]
    assert (len(eight), len(five), len(several)) == (36, 36, 66)
    assert sum(eight) <= 13100 and max(eight) <= 620 and not any(five) and not any(several)
    plain = [v for k, v in _spill_loads("general_kernels.cu").items() if k.startswith("roundtrip_plain_kernel<")]
    assert len(plain) == 43 and not any(plain)


def test_no_decode_kernel_that_nothing_reaches():
    """The general form of the decoder serves one payload that is added to the output, and fp32 records with error feedback."""

    names = [k for k in _spill_loads("codec_kernels.cu") if k.startswith("decode_kernel<")]
    assert len([k for k in names if k.endswith(", 1>")]) == 36
    assert sorted(k for k in names if not k.endswith(", 1>")) == sorted(
        "decode_kernel<float, %d, %d, true, 2>" % (group, bit) for group in (16, 32, 64) for bit in (4, 8))


def test_fp32_encoders_with_a_residual_have_room_for_both_tensors():
    """Sixteen values and sixteen residuals per thread: with five blocks per SM (48 registers) records took a tenth longer."""

    with_residual = [v for k, v in _registers("codec_kernels.cu").items() if re.match(r"encode_kernel<float, \d+, \d, \w+, true, ", k)]
    assert len(with_residual) == 12 and min(with_residual) > 48


def test_fp32_one_rank_kernels_with_three_blocks_do_not_spill():
    """One kept value: the kernels with four blocks per SM do, which passes with a residual and the stochastic code-book pay for
    (192 bytes of spill loads in that one)."""

    loads = {k: v for k, v in _spill_loads("general_kernels.cu").items() if k.startswith("roundtrip_general_kernel<float, 1, ")}
    assert sorted(loads) == ["roundtrip_general_kernel<float, 1, %d, %d>" % kind for kind in
                             ((0, 3), (0, 4), (1, 3), (1, 4), (2, 3), (2, 4), (3, 3))]
    assert all(v == 0 for k, v in loads.items() if k.endswith(", 3>"))
