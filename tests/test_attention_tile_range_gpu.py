"""A prompt pass that starts before the cache or runs past its end: the tokens with a place in it are served, the others left alone."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), ".."))
from tests.test_kernels_gpu import bf16, dev, host  # noqa: E402

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("kv_bf16", [False, True])
@pytest.mark.parametrize("start,tokens,ctx", [(60, 64, 100), (0, 50, 40), (-20, 64, 100), (-3, 40, 30), (90, 48, 90), (-40, 40, 90)])
def test_tokens_outside_the_cache(cuda, kv_bf16, start, tokens, ctx):
    from insignia_b200 import ops

    rng = np.random.default_rng(tokens)
    dt = torch.bfloat16 if kv_bf16 else torch.float32
    kc, vc = (torch.randn(ctx * 1024, device="cuda").to(dt) for _ in range(2))
    qw, kw = dev(bf16(rng, 256)), dev(bf16(rng, 256))
    qraw, kraw, v = (dev(rng.standard_normal((tokens, n)).astype(np.float32)) for n in (8192, 1024, 1024))
    pos, one = torch.full((1,), start, dtype=torch.int32, device="cuda"), ops.gqa_scratch("cuda")
    scratch = torch.zeros(tokens * one.numel(), dtype=torch.uint8, device="cuda")
    got = host(ops.attention_chunk(qraw, kraw, v, qw, kw, kc.clone(), vc.clone(), pos, ctx, scratch, tokens))
    k2, v2 = kc.clone(), vc.clone()
    for m in range(tokens):
        if 0 <= start + m < ctx:
            pos.fill_(start + m)
            want = host(ops.attention_step(qraw[m], kraw[m], v[m], qw, kw, k2, v2, pos, ctx, one))
            assert np.max(np.abs(got[m] - want)) <= 1e-5, m  # two orders of fp32 sums
