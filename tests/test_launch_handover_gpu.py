"""What one launch leaves by ordinary stores and the next fetches by bulk copies (the digits of the activations): launches queued back to back give the bits of launches that are waited for one by one."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), ".."))
from tests.test_kernels_gpu import dev, rand_matrix  # noqa: E402

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("tokens", [9, 49, 300])
@pytest.mark.parametrize("pdl", [False, True])
def test_queued_products_read_their_own_digits(cuda, tokens, pdl):
    from insignia_b200 import ops

    rng = np.random.default_rng(tokens)
    rows, cols, calls = 384, 1152, 24
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
