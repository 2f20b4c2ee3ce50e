"""The query-tile attention of prompt passes (more than 32 tokens) against a float64 softmax over the same cached rows."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), ".."))
from tests.test_kernels_gpu import bf16, dev, host  # noqa: E402

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# tokens: the first count that takes tiles, full tiles, one past them, a ragged long pass; start: rows before the pass
@pytest.mark.parametrize("kv_bf16", [False, True])
@pytest.mark.parametrize("tokens,start,spread", [(33, 0, 1.0), (48, 15, 1.0), (65, 31, 300.0), (256, 33, 1.0), (301, 1000, 1e-3)])
def test_attention_tiles_vs_float64(cuda, kv_bf16, tokens, start, spread):
    from insignia_b200 import ops

    rng = np.random.default_rng(tokens)
    ctx = start + tokens + 3
    dt = torch.bfloat16 if kv_bf16 else torch.float32
    kc, vc = torch.randn(ctx * 1024, device="cuda").to(dt), torch.randn(ctx * 1024, device="cuda")
    # value rows of very different magnitudes, growing along the context: the running scale has to follow
    vc = (vc.view(ctx, 1024) * torch.logspace(0, float(np.log10(spread)), ctx, device="cuda")[:, None]).reshape(-1).to(dt)
    qw, kw = bf16(rng, 256), bf16(rng, 256)
    qraw, kraw, v = (dev(rng.standard_normal((tokens, n)).astype(np.float32)) for n in (8192, 1024, 1024))
    v = v * spread
    pos = torch.full((1,), start, dtype=torch.int32, device="cuda")
    one = ops.gqa_scratch("cuda")
    scratch = torch.zeros(tokens * one.numel(), dtype=torch.uint8, device="cuda")
    got = host(ops.attention_chunk(qraw, kraw, v, dev(qw), dev(kw), kc, vc, pos, ctx, scratch, tokens, fast_trig=False)).reshape(tokens, 16, 256)
    # normalised, rotated queries in float64 (src/ops.cu:9); the keys as the launch stored them
    q = host(qraw).astype(np.float64).reshape(tokens, 16, 512)[:, :, :256]
    w = (qw.astype(np.uint32) << 16).view(np.float32).astype(np.float64)
    q = q / np.sqrt((q * q).mean(-1, keepdims=True) + 1e-6) * w
    ang = (start + np.arange(tokens))[:, None] * 1e7 ** (-2.0 * np.arange(32) / 64)
    c, s = np.cos(ang)[:, None], np.sin(ang)[:, None]
    lo, hi = q[..., :32].copy(), q[..., 32:64].copy()
    q[..., :32], q[..., 32:64] = lo * c - hi * s, hi * c + lo * s
    K = host(kc.float()).astype(np.float64).reshape(ctx, 4, 256)
    V = host(vc.float()).astype(np.float64).reshape(ctx, 4, 256)
    for m in sorted({0, 1, 15, 16, 31, 32, tokens // 2, tokens - 2, tokens - 1}):
        n = start + m + 1
        for h in (0, 5, 15):
            x = K[:n, h >> 2] @ q[m, h] / 16
            p = np.exp(x - x.max())
            want = (p / p.sum()) @ V[:n, h >> 2]
            # fp16 pieces round every operand to 23 bits; scores of a few units turn their error into the same relative error
            # of a weight, and the fp32 rotation angle of position 1300 is good to 1300 * 2^-24: 5e-5 as for the split kernel
            assert np.max(np.abs(got[m, h] - want)) <= 5e-5 * np.abs(V[:n, h >> 2]).max(), (m, h)
