"""The tokens of a short chunk have the bits of single steps at every length: where one cluster holds the rows, where several do,
where the rows reach the bf16 tensor-core loop, on caches of small and large capacity."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), ".."))
from tests.test_kernels_gpu import bf16, dev, host  # noqa: E402

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# 384 rows fill a cluster of eight CTAs and 192 one of four; eight tokens on a small cache take pairs of clusters while one holds the rows
@pytest.mark.parametrize("kv_bf16", [False, True])
@pytest.mark.parametrize("tokens,start,ctx", [(2, 383, 400), (8, 370, 400), (8, 385, 600), (3, 800, 1024), (2, 700, 2560), (2, 800, 2560), (5, 800, 2560),
                                              (2, 1535, 2560), (5, 1600, 2560), (2, 2047, 2560), (32, 1590, 2560)])
def test_chunk_equals_steps_bitwise(cuda, kv_bf16, tokens, start, ctx):
    from insignia_b200 import ops

    rng = np.random.default_rng(start + tokens)
    dt = torch.bfloat16 if kv_bf16 else torch.float32
    kc, vc = (torch.randn(ctx * 1024, device="cuda").to(dt) for _ in range(2))
    qw, kw = dev(bf16(rng, 256)), dev(bf16(rng, 256))
    qraw, kraw, v = (dev(rng.standard_normal((tokens, n)).astype(np.float32)) for n in (8192, 1024, 1024))
    pos, one = torch.full((1,), start, dtype=torch.int32, device="cuda"), ops.gqa_scratch("cuda")
    got = []
    for hint in (0, start + tokens):  # without and with the host's knowledge of the length
        kc2, vc2, big = kc.clone(), vc.clone(), torch.zeros(tokens * one.numel(), dtype=torch.uint8, device="cuda")
        got.append(host(ops.attention_chunk(qraw, kraw, v, qw, kw, kc2, vc2, pos, ctx, big, tokens, rows_hint=hint)))
    want = []
    for m in range(tokens):
        pos.fill_(start + m)
        want.append(host(ops.attention_step(qraw[m], kraw[m], v[m], qw, kw, kc, vc, pos, ctx, one)))
    assert np.array_equal(got[0], np.stack(want)) and np.array_equal(got[1], np.stack(want))
    assert torch.equal(kc, kc2) and torch.equal(vc, vc2)
