"""Plain products on packed records around the size from which they run on tcgen05: the oracle's sums, a token's bits whatever travels along."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), ".."))
from oracle import oracle as orc  # noqa: E402
from tests.test_kernels_gpu import host  # noqa: E402

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# last tiles of 16 and 64 of 128 rows; one k-block (three of four CTAs have none), nine (an odd count for one), 96; the last and the first size of either kernel
@pytest.mark.parametrize("rows,cols", [(98304 + 16, 128), (10944, 1152), (3056, 4096), (3072, 4096), (3088, 4096), (1040, 12288), (12352, 4096)])
@pytest.mark.parametrize("tokens", [1, 2, 3, 5])
def test_products_on_packed_records(cuda, rows, cols, tokens):
    from insignia_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(rows + tokens)
    w = torch.randint(-2**31, 2**31, (rows, cols // 8), generator=gen, device="cuda", dtype=torch.int64).to(torch.int32)
    s = torch.randint(100, 140, (rows, cols // 32), generator=gen, device="cuda", dtype=torch.uint8)
    x = torch.randn(tokens, cols, generator=gen, device="cuda") * torch.logspace(-4, 3, tokens, device="cuda")[:, None]
    packed = ops.repack(w, s)
    y = host(ops.gemv_packed(packed, x))
    assert np.array_equal(host(ops.gemv_packed(packed, x)), y)
    pick = np.r_[0:128, rows // 2:rows // 2 + 32, rows - 32:rows]
    for m in range(tokens):
        assert np.array_equal(host(ops.gemv_packed(packed, x[m].clone())).reshape(-1), y[m]), m
        y64 = orc.gemv_mlx_f64(host(w[pick]).view(np.uint32), host(s[pick]), host(x[m]))
        assert np.max(np.abs(y[m][pick] - y64)) <= 4e-6 * np.abs(y64).max(), m  # 22 bits of the activation and 32-bit sums, as for the smaller matrices


def test_operands_off_sixteen_bytes_are_taken_as_before(cuda):
    from insignia_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(3)
    rows, cols = 3200, 4096
    w = torch.randint(-2**31, 2**31, (rows, cols // 8), generator=gen, device="cuda", dtype=torch.int64).to(torch.int32)
    s = torch.randint(118, 124, (rows, cols // 32), generator=gen, device="cuda", dtype=torch.uint8)
    x = torch.randn(cols, generator=gen, device="cuda")
    packed = ops.repack(w, s)
    room = torch.empty(packed.numel() + 16, dtype=torch.uint8, device="cuda")
    off = room[8:8 + packed.numel()]  # the kernel on mma.sync reads the records by four bytes
    off.copy_(packed)
    got, want = host(ops.gemv_packed(off, x, rows, cols)), host(ops.gemv_packed(packed, x))
    assert np.max(np.abs(got - want)) <= 4e-6 * np.abs(want).max()
