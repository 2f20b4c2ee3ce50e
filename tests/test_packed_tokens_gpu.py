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


# ten and eleven row tiles a CTA at 12288 columns on 148 SMs: 60 and 66 records a warp, on either side of the deeper chunks
@pytest.mark.parametrize("tiles", [10, 11])
def test_one_token_on_both_sides_of_the_chunk_depth(cuda, tiles):
    from insignia_b200 import ops

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rows, cols = 16 * tiles * sms, 12288
    gen = torch.Generator(device="cuda").manual_seed(tiles)
    w = torch.randint(-2**31, 2**31, (rows, cols // 8), generator=gen, device="cuda", dtype=torch.int64).to(torch.int32)
    s = torch.randint(118, 124, (rows, cols // 32), generator=gen, device="cuda", dtype=torch.uint8)
    packed = ops.repack(w, s)
    x = torch.randn(2, cols, generator=gen, device="cuda")
    y = host(ops.gemv_packed(packed, x))
    assert np.array_equal(host(ops.gemv_packed(packed, x[0])).reshape(-1), y[0])
    pick = np.r_[0:16, rows // 2:rows // 2 + 16, rows - 16:rows]
    y64 = orc.gemv_mlx_f64(host(w[pick]).view(np.uint32), host(s[pick]), host(x[0]))
    assert np.max(np.abs(y[0][pick] - y64)) <= 4e-6 * np.abs(y64).max() + 1e-7
