"""Plain products on packed records that are large enough for tcgen05, over the whole range of activations and weight scales: what the kernel on
mma.sync makes of the same records, and no further from float64."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), ".."))
from tests.test_kernels_gpu import host  # noqa: E402

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

ROWS, COLS = 3088, 4096  # 12.6 million weights; a last tile of 16 rows


def _case(tokens, scales, magnitude, seed=0):
    gen = torch.Generator(device="cuda").manual_seed(seed + tokens)
    w = torch.randint(-2**31, 2**31, (ROWS, COLS // 8), generator=gen, device="cuda", dtype=torch.int64).to(torch.int32)
    s = torch.randint(*scales, (ROWS, COLS // 32), generator=gen, device="cuda", dtype=torch.uint8)
    x = (torch.randn(tokens, COLS, generator=gen, device="cuda").double() * magnitude).float()
    return w, s, x


def _small(ops, packed, x):
    """The same product on mma.sync, which takes any size here."""
    out = torch.empty(x.shape[0], ROWS, device="cuda")
    ops.gemv_fused(x, [dict(packed=packed, out=out, rows=ROWS, epilogue="store")], cols=COLS, tokens=x.shape[0])
    return host(out)


def _exact(w, s, x):
    """In float64 throughout (the oracle's weights are fp32 and overflow at the upper end)."""
    code = np.array([0, 0.5, 1, 1.5, 2, 3, 4, 6, -0.0, -0.5, -1, -1.5, -2, -3, -4, -6])
    W = code[(host(w).view(np.uint32)[:, :, None] >> (4 * np.arange(8, dtype=np.uint32))) & 15].reshape(ROWS, COLS)
    return host(x).astype(np.float64) @ (W * np.repeat(np.exp2(host(s).astype(np.float64) - 127), 32, axis=1)).T


# scale bytes (without 0 and 255) and magnitudes of x: results between 1e-37 and 1e37
@pytest.mark.parametrize("scales,magnitude", [((1, 6), 1.0), ((1, 16), 1.0), ((1, 40), 30.0), ((16, 64), 1e-12), ((1, 8), 1e20), ((200, 215), 1e-9), ((235, 255), 1e-20), ((215, 225), 1e-33),
                                              ((118, 124), 1e-34), ((134, 140), 1e-37), ((150, 160), 1e-39), ((100, 240), 1e-10)])
@pytest.mark.parametrize("tokens", [1, 2, 3])
def test_small_and_large_scales(cuda, scales, magnitude, tokens):
    from insignia_b200 import ops

    w, s, x = _case(tokens, scales, magnitude)
    packed = ops.repack(w, s)
    got, want = host(ops.gemv_packed(packed, x)), _exact(w, s, x)
    top = np.abs(want).max(axis=1, keepdims=True)
    assert 1e-38 < top.min() and top.max() < 3e38
    # 22 bits of the activation and 32-bit sums; results that are subnormal themselves are rounded to 2^-149
    assert np.all(np.abs(got - want) <= 4e-6 * top + 2.0**-149)
    for m in range(tokens):
        assert np.array_equal(host(ops.gemv_packed(packed, x[m].clone())).reshape(-1), got[m])


@pytest.mark.parametrize("tokens", [1, 3, 4])
def test_rows_of_any_scale_beside_one_another(cuda, tokens):
    """Rows whose results lie far below the others', rows of zeros, a row that sums to zero, and a token of zeros."""
    from insignia_b200 import ops

    w, s, x = _case(tokens, (118, 124), 1.0)
    x[tokens - 1] = 0
    s[5], s[64:96], s[3087], s[1000] = 3, 20, 11, 250
    w[7], w[2000:2040], s[2010] = 0, 0, 1
    packed = ops.repack(w, s)
    got, want = host(ops.gemv_packed(packed, x)), _exact(w, s, x)
    top = np.abs(host(x)).astype(np.float64).max(axis=1, keepdims=True) * 6 * 64 * np.exp2(host(s).astype(np.float64).max(axis=1) - 127)  # of a row: about its largest sum
    over = np.abs(want) > np.finfo(np.float32).max
    assert over[:-1, 1000].all() and not np.isfinite(got[over]).any()
    assert np.all(np.abs(got - want)[~over] <= (4e-6 * top + 2.0**-149)[~over])
    assert np.all(got[tokens - 1] == 0) and np.all(got[:, 2000:2040] == 0)


@pytest.mark.parametrize("tokens", [1, 2, 4])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_a_non_finite_activation_makes_its_token_nan(cuda, tokens, value):
    from insignia_b200 import ops

    w, s, x = _case(tokens, (118, 124), 1.0)
    packed = ops.repack(w, s)
    clean = host(ops.gemv_packed(packed, x))
    for at in (0, 1037, COLS - 1):
        bad = x.clone()
        bad[tokens - 1, at] = value
        got = host(ops.gemv_packed(packed, bad))
        assert np.isnan(got[tokens - 1]).all() and np.array_equal(got[:-1], clean[:-1])
        assert np.array_equal(np.isnan(_small(ops, packed, bad)), np.isnan(got))


@pytest.mark.parametrize("tokens", [1, 3])
def test_scale_bytes_0_and_255_and_overflow_are_taken_as_by_the_other_kernel(cuda, tokens):
    from insignia_b200 import ops

    w, s, x = _case(tokens, (118, 124), 1.0)
    clean = host(ops.gemv_packed(ops.repack(w, s), x))
    s[9, 0] = s[130, 77] = s[3087, 127] = 255
    s[11, 3] = 0    # a group that counts nothing
    s[12], s[40] = 0, 0  # rows of nothing else
    s[14] = 254     # sums beyond the largest finite value
    packed = ops.repack(w, s)
    got, want = host(ops.gemv_packed(packed, x)), _small(ops, packed, x)
    # infinite or, where infinite terms differ in sign, NaN: which of the two follows from the order of the sums and the pieces they are made of
    assert np.array_equal(np.isfinite(got), np.isfinite(want))
    assert not np.isfinite(got[:, [9, 14, 130, 3087]]).any() and np.all(got[:, [12, 40]] == 0)
    rest = np.setdiff1d(np.arange(ROWS), [9, 11, 12, 14, 40, 130, 3087])
    assert np.array_equal(got[:, rest], clean[:, rest])
    assert np.all(np.abs(got[:, 11] - want[:, 11]) <= 4e-6 * np.abs(clean).max())
