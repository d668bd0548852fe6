"""The warps of the experts' streams that an SM has room for: what the sizes of a decode step were measured with."""
import re
import subprocess

import pytest

from delta_b200.kernels import build

# (0: a result in 32 bit, 1: gated, 2: relu squared; tiles of eight rows; warps a block; a short K of its own) -> warps an SM
ROOM = {(mode, 1, warps, 0): 32 for mode in (0, 1, 2) for warps in (4, 8)} | {(1, 1, 4, 0): 28, (0, 1, 4, 1): 32} \
    | {(mode, 2, warps, 0): 24 for mode in (0, 2) for warps in (4, 8)} | {(0, 4, warps, 0): 24 for warps in (4, 8)} \
    | {(mode, 4, warps, 0): 16 for mode in (1, 2) for warps in (4, 8)} | {(1, 2, 8, 0): 16, (1, 2, 4, 0): 12}


@pytest.fixture(scope="module")
def registers(tmp_path_factory):
    try:
        nvcc = build.find_nvcc()
    except build.BuildError as e:
        pytest.skip(str(e))
    r = subprocess.run([nvcc, *build.NVCC_FLAGS, "-Xptxas", "-v", "-I", str(build.CSRC), "-c", str(build.CSRC / "experts_stream.cu"),
                        "-o", str(tmp_path_factory.mktemp("stream") / "x.o")], capture_output=True, text=True, check=True)
    found = re.findall(r"Compiling entry function '\S*experts_stream_kernelILi(\d)ELi(\d)ELi(\d)ELb(\d)E.*?Used (\d+) registers", r.stderr, re.S)
    return {(int(a), int(b), int(c), int(d)): int(n) for a, b, c, d, n in found}


@pytest.mark.parametrize("instance", sorted(ROOM))
def test_an_sm_has_room_for_as_many_warps_as_measured(registers, instance):
    assert set(registers) == set(ROOM)
    warps = instance[2]
    # 65,536 registers an SM, handed out to warps eight a thread at a time
    blocks = 65536 // (-(-registers[instance] // 8) * 8 * 32 * warps)
    assert min(blocks * warps, 32) >= ROOM[instance], registers[instance]
