"""CTAs of a cluster that write into one another's shared memory: a CTA whose wait for its peers' parts ran out neither leaves while they may still
send nor passes what it has for a result.  Such a wait cannot be made to run out without a stalled GPU, so this reads the source."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "insignia_b200", "csrc")


def splitk():
    with open(os.path.join(CSRC, "attention.cu")) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    start = text.index("attn_splitk_kernel(const __grid_constant__")
    return text[start:text.index("\ntemplate", start)]


def test_decode_attention_leaves_behind_its_exchange():
    body = splitk()
    send = body.index("st.async.shared::cluster")
    wait = re.search(r"if \(!mbar_wait_cluster\(&s_there, 0, &(\w+)\)\) \{(.*?)\n    \}", body[send:], re.S)
    flag, poison = wait.groups()
    # a flag of its own: set by another role, it would cut the wait short
    assert flag not in body[:send].replace("__shared__ int s_abort, " + flag, "").replace("s_abort = " + flag + " = 0", "")
    assert "s_in[c][tid] = kNan" in poison and "s_ml[c] = make_float2(-3.0e38f, kNan)" in poison
    after = body[send + wait.end():]
    leave = re.search(r"auto leave = \[&\] \{(.*?)\n    \};", after, re.S)
    assert re.search(r"lost\b[^;]*barrier\.cluster\.arrive[^;]*;[^;]*barrier\.cluster\.wait.*mbar_wait_cluster\(&s_there", leave.group(1), re.S)
    # every way out goes through it
    rest = after[leave.end():]
    assert all(rest[:m.start()].rstrip().endswith("leave();") for m in re.finditer(r"\breturn;", rest))
    assert rest.rstrip().rstrip("}").rstrip().endswith("leave();")


def test_rows_that_a_wait_left_out_make_no_result():
    body = splitk()
    assert re.search(r"if \(kMma && s_abort\) l0 = kNan;.*st\.async", body, re.S)
