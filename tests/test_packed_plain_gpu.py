"""The packed GEMV's plain vectors around the width up to which all tokens are prepared at once: a token's bits do not depend on the
tokens beside it, and the product is the oracle's."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), ".."))
from oracle import oracle as orc  # noqa: E402
from tests.test_kernels_gpu import dev, host, rand_matrix  # noqa: E402

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("cols", [128, 2176, 4096, 4224])
@pytest.mark.parametrize("tokens", [1, 2, 3, 4])
def test_plain_tokens(cuda, cols, tokens):
    from insignia_b200 import ops

    rng = np.random.default_rng(cols + tokens)
    rows = 48
    w, s = rand_matrix(rng, rows, cols)
    x = (rng.standard_normal((tokens, cols)) * 10.0 ** rng.uniform(-6, 4, (tokens, 1))).astype(np.float32)
    if tokens > 1:
        x[-1] = 0
    P = ops.repack(dev(w), dev(s))
    y = host(ops.gemv_packed(P, dev(x)))
    for m in range(tokens):
        y64 = orc.gemv_mlx_f64(w, s, x[m])
        # two fp16 pieces of the vector's largest element: 22 bits, and fp32 sums
        assert np.max(np.abs(y[m] - y64)) <= 4e-6 * np.abs(y64).max(), m
        assert np.array_equal(y[m], host(ops.gemv_packed(P, dev(x[m])))), m
