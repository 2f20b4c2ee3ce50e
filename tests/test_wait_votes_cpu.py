"""Warps that vote or meet in a loop leave it together.  A bounded wait may run out in some lanes of a warp only; lanes that went on alone would
never meet the others at the loop's next vote.  Such a wait cannot be made to run out in a test without a stalled GPU, so this reads the source."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "insignia_b200", "csrc")
WAIT = r"\b(?:mbar_wait|mbar_wait_cluster|g_wait<CL>)\("


def roles(name):
    """The kernel's per-warp branches: what follows each \"if (warp ...)\" of its outermost chain."""
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    text = re.sub(r"//[^\n]*", "", text)
    parts = re.split(r"\n    (?:\} else )?if \((warp[^)]*)\) \{\n", text)
    return list(zip(parts[1::2], parts[2::2]))


def loops(body):
    """Bodies of the branch's outermost loops."""
    for m in re.finditer(r"\n( +)(?:for|while) \([^\n]*\{\n(.*?)\n\1\}", body, re.S):
        yield m.group(2)


@pytest.mark.parametrize("name", ["umma_gemm.cu"])
def test_loops_that_vote_are_left_together(name):
    seen = 0
    for warp, body in roles(name):
        for loop in loops(body):
            if not re.search(r"__all_sync\(|__syncwarp\(\)", loop) or "bar.red" in loop:  # the epilogue's warps vote through a named barrier
                continue
            for m in re.finditer(WAIT, loop):
                seen += 1
                assert loop[:m.start()].endswith("__all_sync(0xffffffffu, "), (warp, loop[m.start():m.start() + 60])
    assert seen >= 3
