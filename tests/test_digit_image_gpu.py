"""Products that hand their results on as digit images (layout 1, one to eight tokens) against the same chain in fp32 vectors."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), ".."))
from tests.test_kernels_gpu import bf16, dev, host, rand_matrix  # noqa: E402

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# inter: 128 = one k-block for four CTAs (three have none), 1152 = nine (ragged quarters), 3200 = 25
@pytest.mark.parametrize("tokens,inter", [(1, 1152), (2, 128), (3, 3200), (8, 1152)])
def test_prepared_chain_equals_fp32_chain(cuda, tokens, inter):
    """gate|up + SwiGLU -> down + residual -> RMSNorm'd product: the second and third take prepared inputs in one chain and
    convert for themselves in the other.  An image holds 25 bits of every value relative to its 32-element group, as the
    in-kernel conversion does, so the two differ by the rounding of one fp32 factor (2^-23) through three products."""
    from insignia_b200 import _lib, ops

    rng = np.random.default_rng(tokens * inter)
    P = {n: ops.repack_umma(*(dev(a) for a in rand_matrix(rng, r, c))) for n, r, c in
         (("g", inter, 4096), ("u", inter, 4096), ("d", 4096, inter), ("n", 256, 4096))}
    nw, nw2 = dev(bf16(rng, 4096)), dev(bf16(rng, 4096))
    hidden0 = (rng.standard_normal((tokens, 4096)) * rng.uniform(0.1, 30, (tokens, 1))).astype(np.float32)
    got = {}
    for prepared in (False, True):
        h, act, out = dev(hidden0.copy()), torch.zeros(tokens, inter, device="cuda"), torch.zeros(tokens, 256, device="cuda")
        image = [torch.zeros(_lib.lib().insg_mxfp4_digit_image_bytes(c, tokens), dtype=torch.uint8, device="cuda") for c in (inter, 4096)]
        sums, err = torch.zeros(tokens * 128, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
        kw = dict(layout=1, tokens=tokens, error_flag=err)
        for _ in range(2):
            a, b = (dict(prep=image[0]), dict(prep=image[1], prep_w=nw2, prep_partials=sums)) if prepared else ({}, {})
            ops.gemv_fused(h, [dict(packed=P["g"], packed2=P["u"], out=act, rows=inter, epilogue="swiglu", **a)], prologue="rmsnorm", norm_w=nw, cols=4096, **kw)
            ops.gemv_fused(image[0] if prepared else act, [dict(packed=P["d"], out=h, rows=4096, epilogue="residual", **b)],
                           prologue="prepared" if prepared else "plain", cols=inter, **kw)
            ops.gemv_fused(image[1] if prepared else h, [dict(packed=P["n"], out=out, rows=256, epilogue="store")], cols=4096,
                           **(dict(prologue="prepared", prep_partials=sums, prep_rms=True) if prepared else dict(prologue="rmsnorm", norm_w=nw2)), **kw)
        assert int(err.item()) == 0
        got[prepared] = [host(x) for x in (act, h, out)]
    for x, y in zip(*got.values()):
        for m in range(tokens):
            assert np.max(np.abs(x[m] - y[m])) <= 2e-6 * np.abs(x[m]).max(), m
