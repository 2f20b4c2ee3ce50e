"""A segment whose epilogue has no such number leaves its output as it is, in every variant of the tcgen05 products."""
import ctypes as C
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), ".."))
from tests.test_kernels_gpu import dev, host, rand_matrix  # noqa: E402

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# 8 k-blocks: whole octets (the variant that leaves nothing prepared); 9: the general one
@pytest.mark.parametrize("cols", [1024, 1152])
@pytest.mark.parametrize("tokens,prologue", [(1, "plain"), (1, "prepared"), (2, "plain"), (2, "prepared"), (3, "prepared"), (8, "plain"), (8, "prepared"), (16, "plain")])
def test_output_stays(cuda, tokens, prologue, cols):
    from insignia_b200 import _lib, ops

    rng = np.random.default_rng(cols + tokens)
    P = ops.repack_umma(*(dev(a) for a in rand_matrix(rng, 256, cols)))
    x = dev(rng.standard_normal((tokens, cols)).astype(np.float32))
    if prologue == "prepared":
        x = torch.zeros(_lib.lib().insg_mxfp4_digit_image_bytes(cols, tokens), dtype=torch.uint8, device="cuda")
    out = torch.full((tokens, 256), 7.0, device="cuda")
    op = ops._gemv_op(x, [dict(packed=P, out=out, rows=256, epilogue="store")], prologue=prologue, layout=1, tokens=tokens, cols=cols,
                      umma_scratch=ops.umma_gemm_scratch(cols, tokens) if tokens > 8 else None)
    op.seg[0].epilogue = 99
    _lib.check(_lib.lib().insg_gemv_fused(C.byref(op), ops._stream()))
    assert np.all(host(out) == 7.0)
