"""The tcgen05 GEMM's seven digits per activation: groups whose largest element lies at either side of the extra bit, every digit's
edge values, and token counts at the edges of the groups of 16 and 32."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), ".."))
from oracle import oracle as orc  # noqa: E402
from tests.test_kernels_gpu import dev, host, rand_matrix  # noqa: E402

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

EDGE = 1 + 0x1F0000 / 2**23  # mantissas below it keep one bit more


@pytest.mark.parametrize("tokens", [9, 16, 17, 48, 49, 64, 65])
def test_digits_at_the_edges(cuda, tokens):
    from insignia_b200 import ops

    rows, cols = 160, 640  # a second tile of 32 rows; five k-blocks
    rng = np.random.default_rng(tokens)
    w, s = rand_matrix(rng, rows, cols)
    # each group of 32: its largest element at a chosen mantissa, the others anywhere below, many of them at multiples of powers of 13
    largest = np.array([1, np.nextafter(np.float32(EDGE), np.float32(0)), EDGE, np.nextafter(np.float32(2), np.float32(0)), 1.5], np.float32)
    groups = tokens * cols // 32
    top = largest[rng.integers(0, 5, groups)] * np.float32(2.0) ** rng.integers(-20, 20, groups).astype(np.float32)
    x = (rng.uniform(-1, 1, (groups, 32)) * top[:, None]).astype(np.float32)
    k = rng.integers(0, 7, (groups, 8))
    unit = 2.0 ** np.floor(np.log2(top))[:, None] / 2**23
    x[:, 8:16] = np.clip(rng.integers(-12, 13, (groups, 8)) * 13.0**k * unit, -top[:, None], top[:, None])
    x[:, 0] = top * rng.choice([-1, 1], groups)
    x = x.reshape(tokens, cols)
    y = host(ops.gemm_umma(ops.repack_umma(dev(w), dev(s)), dev(x)))
    weights = np.abs(host(ops.dequant_mlx(dev(w), dev(s))).astype(np.float64))
    room = np.repeat(top.reshape(tokens, cols // 32), 32, axis=1).astype(np.float64)
    for m in range(tokens):
        # an element is off by half a unit of at most 2^-23 of its group's largest power of two; the sums of 32-element groups (fp32,
        # truncated) and the seven combinations add an ulp of the sum of magnitudes each at the very most
        bound = weights @ room[m] * 2.0**-24 + weights @ np.abs(x[m].astype(np.float64)) * 2.0**-23 * 8
        assert np.all(np.abs(y[m] - orc.gemv_mlx_f64(w, s, x[m])) <= bound), m
