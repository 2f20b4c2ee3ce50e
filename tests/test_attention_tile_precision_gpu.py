"""The query tiles of a prompt pass are as close to float64 as the token-by-token form of the same attention."""
import ctypes as C
import os
import sys

import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), ".."))

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("kv_bf16", [False, True])
@pytest.mark.parametrize("tokens,start", [(64, 0), (100, 50), (256, 0), (301, 1000), (512, 512)])
def test_tiles_are_as_precise_as_single_tokens(cuda, kv_bf16, tokens, start):
    from insignia_b200 import _lib, ops

    torch.manual_seed(tokens)
    ctx, dt = start + tokens, torch.bfloat16 if kv_bf16 else torch.float32
    kc, vc = (torch.randn(ctx * 1024, device="cuda").to(dt) for _ in range(2))
    qw, kw = ((1 + 0.1 * torch.randn(256, device="cuda")).to(torch.bfloat16).view(torch.int16) for _ in range(2))
    qraw, kraw, v = (torch.randn(tokens, n, device="cuda") for n in (8192, 1024, 1024))
    pos, out, q = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.empty(tokens, 4096, device="cuda"), torch.empty(tokens, 4096, device="cuda")
    scratch = torch.zeros(tokens * ops.gqa_scratch("cuda").numel(), dtype=torch.uint8, device="cuda")

    def run(first, count):  # `count` tokens from `first` on in one call
        op = _lib.AttnOp()
        for name, t in dict(qraw=qraw[first:], k_raw=kraw[first:], v=v[first:], q_norm_w=qw, k_norm_w=kw, k_cache=kc, v_cache=vc, out=out[first:], position=pos,
                            scratch=scratch).items():
            setattr(op, name, t.data_ptr())
        op.max_context, op.kv_dtype, op.scratch_bytes = ctx, int(kv_bf16), scratch.numel()
        pos.fill_(start + first)
        _lib.check(_lib.lib().insg_attention_chunk(C.byref(op), count, q[first:].data_ptr(), start + first + count, torch.cuda.current_stream().cuda_stream))

    error = []
    for step in (tokens, 32):
        for first in range(0, tokens, step):
            run(first, min(step, tokens - first))
        K, V = (c.double().view(ctx, 4, 256).repeat_interleave(4, 1) for c in (kc, vc))
        x = torch.einsum("thd,nhd->thn", q.double().view(tokens, 16, 256), K) / 16  # the queries as the call normalised and rotated them
        seen = torch.arange(ctx, device="cuda")[None, :] <= (start + torch.arange(tokens, device="cuda"))[:, None]
        want = torch.einsum("thn,nhd->thd", torch.softmax(x.masked_fill(~seen[:, None], float("-inf")), -1), V)
        error.append(float((out.double().view(tokens, 16, 256) - want).norm() / want.norm()))
    # two orders of the same fp32 arithmetic differ by chance: a sixth of sums that are 1.0e-7 to 1.9e-7 off
    assert error[0] <= 1.17 * error[1], error
