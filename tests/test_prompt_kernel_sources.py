"""What the prompt kernels' sources have to keep to and no run can show: a breach may work on one chip and hang another."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "kinetics_b200" / "csrc"
KERNELS = [CSRC / "ktk_prefill_umma.cu", CSRC / "layers" / "ktl_attn_umma.cu", CSRC / "layers" / "ktl_attn_expanded.cu"]


def _number(text, name):
    return int(re.search(rf"constexpr int {name} = (\d+);", text).group(1))


@pytest.mark.parametrize("path", KERNELS, ids=lambda p: p.stem)
def test_all_warps_of_a_warpgroup_change_their_registers_by_one_instruction(path):
    """setmaxnreg is .aligned over the warpgroup: one instruction, on a branch that whole warpgroups take."""
    lines = [line.strip() for line in path.read_text().splitlines()]
    for call, branch in (("fewer_registers();", "if (warp >= kFlSoftmaxWarps) {"), ("more_registers();", "} else {")):
        at = [i for i, line in enumerate(lines) if call in line]
        assert len(at) == 1, (call, at)
        assert lines[at[0] - 1] == branch
    assert not any("setmaxnreg" in line for line in lines)


def test_the_registers_of_the_warpgroups_are_those_of_the_launch():
    """setmaxnreg.inc waits for registers that the block was launched with: a larger sum would wait for good."""
    text = (CSRC / "ktk_flash.cuh").read_text()
    threads, softmax = _number(text, "kFlThreads"), 32 * _number(text, "kFlSoftmaxWarps")
    assert threads % 128 == 0 and softmax % 128 == 0
    more, = map(int, re.findall(r"setmaxnreg\.inc\.sync\.aligned\.u32 (\d+);", text))
    fewer, = map(int, re.findall(r"setmaxnreg\.dec\.sync\.aligned\.u32 (\d+);", text))
    launched = 65536 // threads // 8 * 8                       # registers per thread come in eights
    assert softmax * more + (threads - softmax) * fewer <= threads * launched
