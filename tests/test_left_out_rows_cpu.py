"""A plain product has no error flag: rows whose sums a bounded wait left out are NaN.  Such a wait cannot be made to run out without a stalled GPU, so
this reads the source."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "insignia_b200", "csrc")


def test_rows_left_out_are_nan():
    with open(os.path.join(CSRC, "umma_gemv.cu")) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    owner = text[text.index("int i = group;"):]
    loop = re.match(r"int i = group;\n#pragma unroll 1\n        for \(; i < nun && ok; i \+= kGroups\) \{\n(.*?)\n        \}\n", owner, re.S)
    # the unit that is given up is the one `i` still names: the loop is left behind the wait, ahead of the unit's stores
    assert loop.group(1).index("if (!ok) break;\n            if (!delta") < loop.group(1).index("out[(t0 + u) * ld] = v[u];")
    rest = owner[loop.end():]
    nan = re.match(r"\s*if constexpr \(records\)\s*if \(!ok\)\n#pragma unroll 1\n\s*for \(; i < nun; i \+= kGroups\) \{(.*?)\n                \}", rest, re.S).group(1)
    assert "min(t0 + TN, p.tokens)" in nan and "row < p.seg[0].rows" in nan and "__int_as_float(0x7fc00000)" in nan
