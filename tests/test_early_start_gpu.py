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


def _rows_then_step(ops, gen, between, tokens, alone):
    """The rows of `tokens` tokens, alone or with their attention, and the next token's step, which fetches rows ahead of its wait."""
    import ctypes as C

    from insignia_b200 import _lib

    L, ctx = _lib.lib(), tokens + 1
    randn = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    kc, vc, raw, last = randn(ctx * 1024), randn(ctx * 1024), (randn(tokens, 8192), randn(tokens, 1024), randn(tokens, 1024)), (randn(1, 8192), randn(1, 1024), randn(1, 1024))
    norm = torch.ones(256, device="cuda").to(torch.bfloat16).view(torch.int16)
    first, next_ = (torch.full((1,), at, dtype=torch.int32, device="cuda") for at in (0, tokens))
    scratch = torch.zeros(max(1, min(tokens, 32)) * ops.gqa_scratch("cuda").numel(), dtype=torch.uint8, device="cuda")
    between()
    if alone:
        op = _lib.AttnOp()
        op.k_raw, op.v, op.k_norm_w, op.k_cache, op.v_cache, op.position = (t.data_ptr() for t in (raw[1], raw[2], norm, kc, vc, first))
        op.max_context, op.kv_dtype, op.fast_trig = ctx, ops.KV_F32, 1
        _lib.check(L.insg_attention_rows(C.byref(op), tokens, torch.cuda.current_stream().cuda_stream))
        got = []
    else:
        got = [ops.attention_chunk(*raw, norm, norm, kc, vc, first, ctx, scratch, tokens)]
    between()
    got += [ops.attention_step(*last, norm, norm, kc, vc, next_, ctx, scratch, pdl=True), kc, vc]
    torch.cuda.synchronize()
    return [host(t) for t in got]


@pytest.mark.parametrize("tokens,alone", [(3, True), (1500, True), (3, False), (20, False), (300, False)])
def test_a_step_that_reads_ahead_sees_the_rows_of_the_call_before(cuda, tokens, alone):
    from insignia_b200 import ops

    for seed in range(4):
        make = lambda: torch.Generator(device="cuda").manual_seed(seed)  # noqa: E731
        apart = _rows_then_step(ops, make(), torch.cuda.synchronize, tokens, alone)
        for _ in range(4):
            for a, b in zip(_rows_then_step(ops, make(), lambda: None, tokens, alone), apart):
                assert np.array_equal(a, b)
