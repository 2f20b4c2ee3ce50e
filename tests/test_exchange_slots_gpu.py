"""tcgen05 GEMV: the exchange slots of a cluster used over and over (many row tiles, hardly any K) against float64."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), ".."))
from oracle import oracle as orc  # noqa: E402
from tests.test_kernels_gpu import dev, host, rand_matrix  # noqa: E402

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# 300 tiles are nine or ten a cluster, whose slots hold one, two or four; one k-block leaves three CTAs of a cluster without any
@pytest.mark.parametrize("cols", [128, 640])
@pytest.mark.parametrize("tokens", [1, 2, 3, 8])
def test_slots_are_reused_in_order(cuda, tokens, cols):
    from insignia_b200 import ops

    rng = np.random.default_rng(tokens + cols)
    rows = 300 * 128 - 5
    (w, s), (w2, s2) = rand_matrix(rng, rows, cols), rand_matrix(rng, rows, cols)
    x = rng.standard_normal((tokens, cols)).astype(np.float32)
    P, P2, xd = ops.repack_umma(dev(w), dev(s)), ops.repack_umma(dev(w2), dev(s2)), dev(x)
    want = [np.stack([orc.gemv_mlx_f64(a, b, v) for v in x]) for a, b in ((w, s), (w2, s2))]
    err, first = torch.zeros(1, dtype=torch.int32, device="cuda"), {}
    for _ in range(10):
        for epilogue in ("store", "swiglu"):
            out = torch.zeros(tokens, rows, device="cuda")
            seg = dict(packed=P, out=out, rows=rows, epilogue=epilogue, **(dict(packed2=P2) if epilogue == "swiglu" else {}))
            ops.gemv_fused(xd, [seg], layout=1, tokens=tokens, cols=cols, error_flag=err)
            got = host(out)
            assert np.array_equal(got, first.setdefault(epilogue, got)), epilogue
    assert int(err.item()) == 0
    # sums of up to 640 fp32 products of 25-bit operands; fast_silu (a reciprocal and an exponential of 2^-22 each)
    assert np.max(np.abs(first["store"] - want[0])) <= 4e-6 * np.abs(want[0]).max()
    glu = want[0] / (1 + np.exp(-want[0])) * want[1]
    assert np.max(np.abs(first["swiglu"] - glu)) <= 1e-5 * np.abs(glu).max()
