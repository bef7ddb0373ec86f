"""The batched product's warps are whole where an instruction wants that: between a step
that lanes may leave one by one (a wait for or a question about a barrier, a branch on the
lane) and the next .aligned tensor-memory instruction or elect.sync stands a warp or CTA barrier."""
import re

import pytest

from test_early_start_loads import CSRC

APART = r"mbar_wait\(|mbar_test\(|take_words\(|lane == 0\)"
WHOLE = r"__syncwarp\(\)|__syncthreads\(\)|bar\.sync"
WANTS = r"tcgen05\.[a-z_:]+[a-z0-9_.:]*\.sync\.aligned|tmem_store(?:_32)?\(|elect_one\(\)"


@pytest.mark.parametrize("name", ["qgemm.cu", "qgemm_stream.cuh"])
def test_aligned_instructions_meet_a_whole_warp(name):
    text = re.sub(r"//[^\n]*", "", (CSRC / name).read_text())
    kernel = re.search(r"__global__.*?^}\n", text, flags=re.M | re.S).group(0)
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
