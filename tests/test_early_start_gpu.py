"""Operator calls start before the launch ahead of them has ended and wait before they read: whatever that launch wrote, weights, states, caches and
inputs among it, is seen, and the results are those of calls with the device idle in between."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), ".."))
from tests.test_kernels_gpu import host  # noqa: E402

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _calls(ops, gen, between):
    """Each call's operands are written by the launch right before it."""
    randn = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    weights = [(torch.randint(-2**31, 2**31, (rows, cols // 8), generator=gen, device="cuda", dtype=torch.int64).to(torch.int32),
                torch.randint(118, 124, (rows, cols // 32), generator=gen, device="cuda", dtype=torch.uint8)) for rows, cols in ((3200, 4096), (512, 4096))]
    x, qkv, g, beta = randn(40, 4096), randn(40, 8192), -randn(40, 32).abs(), torch.sigmoid(randn(40, 32))
    state0, caches = 0.1 * randn(32 * 128 * 128), [randn(300 * 1024) for _ in range(2)]
    scratch, gemm = ops.gqa_scratch("cuda"), ops.umma_gemm_scratch(4096, 40)
    norm, pos, qraw, raw = torch.ones(256, device="cuda").to(torch.bfloat16).view(torch.int16), torch.full((1,), 299, dtype=torch.int32, device="cuda"), randn(1, 8192), randn(2, 1, 1024)
    got = []

    def step(fn, *a, **kw):
        between()
        r = fn(*a, **kw)
        between()
        return r

    for w, s in weights:  # packed by the launch before; large enough for tcgen05, and not
        packed = step(ops.repack, w, s)
        y = step(ops.gemv_packed, packed, x[:1])
        got += [y, step(ops.gemv_packed, packed, y[:, :512].repeat(3, 8).contiguous())]  # the input by a copy that reads the result
    image = step(ops.repack_umma, *weights[0])
    y = step(ops.gemm_umma, image, x, scratch=gemm)
    got += [y, step(ops.gemm_umma, image, torch.cat([y, y], 1)[:, :4096].contiguous(), scratch=gemm), step(ops.gemm_umma, image, x[:2], scratch=gemm)]
    state, flat = torch.empty_like(state0), qkv.view(-1)
    for n in (1, 40):
        step(state.copy_, state0)
        got.append(step(ops.deltanet_decode_tokens, state, flat, flat[2048:], flat[4096:], g, beta, n, 8192))
        got += [step(ops.deltanet_decode_tokens, state, flat, flat[2048:], flat[4096:], g, beta, n, 8192), state.clone()]
    kc, vc = (torch.empty_like(c) for c in caches)
    step(kc.copy_, caches[0])
    step(vc.copy_, caches[1])
    got.append(step(ops.gqa_decode, y.view(-1)[:4096], kc, vc, 300, scratch=scratch))
    step(kc.copy_, caches[1])
    got.append(step(ops.attention_batch, qraw, raw[0], raw[1], norm, norm, kc.view(1, -1), vc.view(1, -1), pos, 300, scratch, 1))
    got.append(step(ops.gqa_decode, got[-1].view(-1), kc, vc, 300, scratch=scratch))
    torch.cuda.synchronize()
    return [host(t) for t in got]


def test_calls_one_behind_the_other_see_what_was_written_before(cuda):
    from insignia_b200 import ops

    for seed in range(6):
        make = lambda: torch.Generator(device="cuda").manual_seed(seed)  # noqa: E731
        apart = _calls(ops, make(), torch.cuda.synchronize)
        for _ in range(3):
            for a, b in zip(_calls(ops, make(), lambda: None), apart):
                assert np.array_equal(a, b)
