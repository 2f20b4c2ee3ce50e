"""What one launch leaves by ordinary stores and the next fetches by bulk copies (digits of the activations, rows of the bf16 cache):
launches queued back to back give the bits of launches that are waited for one by one."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), ".."))
from tests.fixtures import pair_tokens  # noqa: E402
from tests.test_kernels_gpu import bf16, dev, host, rand_matrix  # noqa: E402

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("tokens", [9, 49, 300, "pairs"])
@pytest.mark.parametrize("pdl", [False, True])
def test_queued_products_read_their_own_digits(cuda, tokens, pdl):
    from insignia_b200 import ops

    rows, cols, calls = 384, 1152, 24
    if tokens == "pairs":  # the GEMM on pairs of CTAs, whose digits have a producer warp of their own
        rows = 2432
        tokens = pair_tokens(rows, cols)
    rng = np.random.default_rng(tokens)
    packed = ops.repack_umma(*(dev(a) for a in rand_matrix(rng, rows, cols)))
    xs = [torch.randn(tokens, cols, device="cuda") for _ in range(calls)]

    def product(x, out, scratch):
        ops.gemv_fused(x, [dict(packed=packed, out=out, rows=rows, epilogue="store")], layout=1, tokens=tokens, cols=cols, umma_scratch=scratch, pdl=pdl)

    alone, queued = torch.zeros(calls, tokens, rows, device="cuda"), torch.zeros(calls, tokens, rows, device="cuda")
    for x, out in zip(xs, alone):
        product(x, out, ops.umma_gemm_scratch(cols, tokens))
        torch.cuda.synchronize()
    scratch = ops.umma_gemm_scratch(cols, tokens)
    for x, out in zip(xs, queued):  # one scratch: every call overwrites the digits of the one before
        product(x, out, scratch)
    assert torch.equal(alone, queued)


def test_queued_steps_read_the_rows_before_them(cuda):
    """Steps around the length from which the bf16 cache is fetched by bulk copies."""
    from insignia_b200 import ops

    first, steps, ctx = 2030, 40, 2080
    rng = np.random.default_rng(3)
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    q, k, v = (torch.randn(steps, n, generator=g, device="cuda") for n in (8192, 1024, 1024))
    kc0, vc0 = (torch.randn(ctx * 1024, generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    w = dev(bf16(rng, 256))
    position = torch.full((1,), first, dtype=torch.int32, device="cuda")

    def run(wait):
        kc, vc, scratch, outs = kc0.clone(), vc0.clone(), ops.gqa_scratch("cuda"), []
        torch.cuda.synchronize()
        for i in range(steps):
            outs.append(ops.attention_step(q[i], k[i], v[i], w, w, kc, vc, position, ctx, scratch, position_offset=i, pdl=not wait))
            if wait:
                torch.cuda.synchronize()
        return host(torch.stack(outs)), kc, vc

    alone, ka, va = run(True)
    for _ in range(3):
        queued, kq, vq = run(False)
        assert np.array_equal(alone, queued)
        assert torch.equal(ka, kq) and torch.equal(va, vq)
