"""Infinities, NaN and the largest finite values go through the tcgen05 products as fp32 arithmetic takes them: a token with one
gives NaN, the others of the launch are untouched."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), ".."))
from oracle import oracle as orc  # noqa: E402
from tests.test_kernels_gpu import bf16, dev, host, rand_matrix  # noqa: E402

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# up to eight tokens: the GEMV; more: the GEMM with 16 (up to 48) or 24 tokens a group
@pytest.mark.parametrize("tokens", [1, 2, 3, 8, 9, 16, 48, 49, 71])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_a_non_finite_activation_makes_its_token_nan(cuda, tokens, value):
    from insignia_b200 import ops

    rng = np.random.default_rng(tokens)
    rows, cols = 384, 1152
    P = ops.repack_umma(*(dev(a) for a in rand_matrix(rng, rows, cols)))
    x = rng.standard_normal((tokens, cols)).astype(np.float32)
    clean = host(ops.gemm_umma(P, dev(x)))
    for at in (0, 37, cols - 1):
        bad = x.copy()
        bad[tokens - 1, at] = value
        got = host(ops.gemm_umma(P, dev(bad)))
        assert np.isnan(got[tokens - 1]).all()
        assert np.array_equal(got[:-1], clean[:-1])


@pytest.mark.parametrize("tokens", [1, 3, 8])
def test_a_prepared_image_carries_nan(cuda, tokens):
    """A residual stream with a NaN, left as a digit image with sums of squares, and the product that takes the image."""
    from insignia_b200 import _lib, ops

    rng = np.random.default_rng(tokens)
    P, N = (ops.repack_umma(*(dev(a) for a in rand_matrix(rng, r, c))) for r, c in ((4096, 128), (256, 4096)))
    x, nw = dev(rng.standard_normal((tokens, 128)).astype(np.float32)), dev(bf16(rng, 4096))
    hidden = rng.standard_normal((tokens, 4096)).astype(np.float32)
    got = []
    for bad in (False, True):
        for rms in (False, True):
            h = hidden.copy()
            if bad:
                h[tokens - 1, 2049] = np.nan
            h, out = dev(h), torch.zeros(tokens, 256, device="cuda")
            image = torch.zeros(_lib.lib().insg_mxfp4_digit_image_bytes(4096, tokens), dtype=torch.uint8, device="cuda")
            sums, err = torch.zeros(tokens * 128, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
            kw = dict(layout=1, tokens=tokens, error_flag=err)
            ops.gemv_fused(x, [dict(packed=P, out=h, rows=4096, epilogue="residual", prep=image, prep_w=nw, prep_partials=sums)], cols=128, **kw)
            ops.gemv_fused(image, [dict(packed=N, out=out, rows=256, epilogue="store")], cols=4096, prologue="prepared",
                           **(dict(prep_partials=sums, prep_rms=True) if rms else {}), **kw)
            assert int(err.item()) == 0
            got.append(host(out))
    for clean, with_nan in zip(got[:2], got[2:]):
        assert np.isfinite(clean).all() and np.isnan(with_nan[-1]).all() and np.array_equal(clean[:-1], with_nan[:-1])


@pytest.mark.parametrize("tokens", [1, 8, 9, 49])
@pytest.mark.parametrize("scale", [1e32, 1e-33])
def test_groups_of_very_large_and_small_values(cuda, tokens, scale):
    from insignia_b200 import ops

    rng = np.random.default_rng(tokens)
    w, s = rand_matrix(rng, 256, 1152)
    x = (rng.standard_normal((tokens, 1152)) * scale).astype(np.float32)
    x[:, 64:96] *= 1e3  # one group far above the others
    got = host(ops.gemm_umma(ops.repack_umma(dev(w), dev(s)), dev(x))).astype(np.float64)
    for m in range(tokens):
        want = orc.gemv_mlx_f64(w, s, x[m])
        assert np.max(np.abs(got[m] - want)) <= 4e-6 * np.abs(want).max()
