"""The batched product's warps are whole where an instruction wants that: between a step
that lanes may leave one by one (a wait for a barrier, a branch on one lane's answer or on the lane) and the
next .aligned tensor-memory instruction or elect.sync stands a warp or CTA barrier or a vote."""
import re

import pytest

from test_early_start_loads import CSRC

APART = r"mbar_wait\(|mbar_test\(|lane == 0\)"
WHOLE = r"__syncwarp\(\)|__syncthreads\(\)|bar\.sync|mbar_over\("
WANTS = r"tcgen05\.[a-z_:]+[a-z0-9_.:]*\.sync\.aligned|tmem_store(?:_32)?\(|elect_one\(\)"


def _code(name):
    return re.sub(r"//[^\n]*", "", (CSRC / name).read_text())


def test_the_question_to_a_barrier_is_a_vote():
    over = re.search(r"bool mbar_over\(.*?^}\n", _code("qgemm.cu"), flags=re.M | re.S).group(0)
    assert "return __all_sync(0xffffffffu, done);" in over


@pytest.mark.parametrize("name", ["qgemm.cu", "qgemm_stream.cuh"])
def test_aligned_instructions_meet_a_whole_warp(name):
    kernel = re.search(r"__global__.*?^}\n", _code(name), flags=re.M | re.S).group(0)
    apart, seen = None, 0
    for m in re.finditer(f"(?P<apart>{APART})|(?P<whole>{WHOLE})|(?P<wants>{WANTS})", kernel):
        line = kernel[:m.start()].count("\n")
        if m["whole"]:
            apart = None
        elif m["apart"]:
            apart = m.group(0)
        else:
            assert apart is None, f"{name}, kernel line {line}: {m.group(0)} after {apart}"
            seen += 1
            if m.group(0) == "elect_one()":
                apart = m.group(0)  # its branch is one lane's
    assert seen > 10
