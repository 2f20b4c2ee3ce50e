"""Packed GEMV of two to four tokens: the bits of one token at a time, whatever the tokens that travel along."""
import numpy as np
import pytest

from oracle import oracle as orc
from tests.test_kernels_gpu import dev, host, rand_matrix

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# one record a warp and less, a run shared by several warps, several runs a warp, an uneven last tile count, widest columns
@pytest.mark.parametrize("rows,cols", [(16, 128), (48, 1152), (16 * 149, 256), (16 * 300, 384), (64, 12288)])
@pytest.mark.parametrize("M", [2, 3, 4])
def test_tokens_do_not_depend_on_one_another(cuda, rows, cols, M):
    from insignia_b200 import ops

    rng = np.random.default_rng(rows + cols + M)
    w, s = rand_matrix(rng, rows, cols)
    x = (rng.standard_normal((M, cols)) * rng.uniform(0.01, 30, (M, 1))).astype(np.float32)
    packed = ops.repack(dev(w), dev(s))
    y = host(ops.gemv_packed(packed, dev(x)))
    for m in range(M):
        assert np.array_equal(host(ops.gemv_packed(packed, dev(x[m]))).reshape(-1), y[m]), m
        y64 = orc.gemv_mlx_f64(w, s, x[m])
        # the activation's two fp16 pieces keep 22 bits, the rest is the rounding of 32-bit sums: the bar of the one-token tests
        assert np.max(np.abs(y[m] - y64)) <= 4e-6 * np.abs(y64).max() + 1e-7
