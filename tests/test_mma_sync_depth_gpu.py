"""The kernel on mma.sync on both sides of its deeper chunks (64 records a warp), which plain products of that size no longer reach: through the fused launch."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), ".."))
from oracle import oracle as orc  # noqa: E402
from tests.test_kernels_gpu import host  # noqa: E402

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# ten and eleven row tiles a CTA at 12288 columns: 60 and 66 records a warp
@pytest.mark.parametrize("tiles", [10, 11])
def test_one_token_on_both_sides_of_the_chunk_depth(cuda, tiles):
    from insignia_b200 import ops

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rows, cols = 16 * tiles * sms, 12288
    gen = torch.Generator(device="cuda").manual_seed(tiles)
    w = torch.randint(-2**31, 2**31, (rows, cols // 8), generator=gen, device="cuda", dtype=torch.int64).to(torch.int32)
    s = torch.randint(118, 124, (rows, cols // 32), generator=gen, device="cuda", dtype=torch.uint8)
    packed, x = ops.repack(w, s), torch.randn(2, cols, generator=gen, device="cuda")
    one, two = torch.empty(rows, device="cuda"), torch.empty(2, rows, device="cuda")
    ops.gemv_fused(x[0].clone(), [dict(packed=packed, out=one, rows=rows, epilogue="store")])
    ops.gemv_fused(x, [dict(packed=packed, out=two, rows=rows, epilogue="store")], cols=cols, tokens=2)
    assert np.array_equal(host(one), host(two)[0])
    pick = np.r_[0:16, rows // 2:rows // 2 + 16, rows - 16:rows]
    y64 = orc.gemv_mlx_f64(host(w[pick]).view(np.uint32), host(s[pick]), host(x[0]))
    assert np.max(np.abs(host(one)[pick] - y64)) <= 4e-6 * np.abs(y64).max() + 1e-7  # as for the smaller matrices
