"""Infinities, NaN and the largest finite values go through the tcgen05 products as fp32 arithmetic takes them: a token with one
gives NaN, the others of the launch are untouched."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), ".."))
from oracle import oracle as orc  # noqa: E402
from tests.fixtures import pair_tokens  # noqa: E402
from tests.test_kernels_gpu import bf16, dev, host, rand_matrix  # noqa: E402

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# up to eight tokens: the GEMV; more: the GEMM with 16 tokens a group, or with 32 on pairs of CTAs (with 17 in the last one)
@pytest.mark.parametrize("tokens", [1, 2, 3, 8, 9, 16, 48, 49, 71, "pairs"])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_a_non_finite_activation_makes_its_token_nan(cuda, tokens, value):
    from insignia_b200 import ops

    rows, cols = 384, 1152
    if tokens == "pairs":
        rows = 2432  # 19 tiles
        tokens = pair_tokens(rows, cols, last=17)
    rng = np.random.default_rng(tokens)
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


@pytest.mark.parametrize("tokens", [1, 8, 9, 49, "pairs"])
@pytest.mark.parametrize("scale", [1e32, 1e-33])
def test_groups_of_very_large_and_small_values(cuda, tokens, scale):
    from insignia_b200 import ops

    rows = 256
    if tokens == "pairs":
        rows = 2432
        tokens = pair_tokens(rows, 1152)
    rng = np.random.default_rng(tokens)
    w, s = rand_matrix(rng, rows, 1152)
    x = (rng.standard_normal((tokens, 1152)) * scale).astype(np.float32)
    x[:, 64:96] *= 1e3  # one group far above the others
    got = host(ops.gemm_umma(ops.repack_umma(dev(w), dev(s)), dev(x))).astype(np.float64)
    for m in range(tokens):
        want = orc.gemv_mlx_f64(w, s, x[m])
        assert np.max(np.abs(got[m] - want)) <= 4e-6 * np.abs(want).max()


def _chunk(ops, case, tokens, start, ctx, k, v, step):
    """The pass in calls of `step` tokens: `tokens` = the query tiles, 32 = the token-by-token form."""
    kc, vc, pos = case["kc"].clone(), case["vc"].clone(), torch.zeros(1, dtype=torch.int32, device="cuda")
    scratch, out = torch.zeros(32 * ops.gqa_scratch("cuda").numel(), dtype=torch.uint8, device="cuda"), []
    if step > 32:
        scratch = torch.zeros(step * ops.gqa_scratch("cuda").numel(), dtype=torch.uint8, device="cuda")
    for first in range(0, tokens, step):
        n = min(step, tokens - first)
        pos.fill_(start + first)
        out.append(host(ops.attention_chunk(case["q"][first:first + n].contiguous(), k[first:first + n].contiguous(), v[first:first + n].contiguous(), case["qw"],
                                            case["kw"], kc, vc, pos, ctx, scratch, n)))
    return np.concatenate(out).reshape(tokens, 16, 256)


# the value sits in the pass (tokens before it must not see it) or in the rows behind it; start 0: the first rows of an empty cache
@pytest.mark.parametrize("kv_bf16", [False, True])
@pytest.mark.parametrize("start", [0, 200])
@pytest.mark.parametrize("what,value", [("key", np.nan), ("value", np.nan), ("value", np.inf), ("value", 1e33), ("query", np.nan), ("none", 0.0)])
def test_prompt_attention_keeps_a_bad_row_to_the_tokens_that_see_it(cuda, kv_bf16, start, what, value):
    from insignia_b200 import ops

    rng = np.random.default_rng(start)
    tokens, at = 100, 41
    ctx, dt = start + tokens, torch.bfloat16 if kv_bf16 else torch.float32
    case = {n: torch.randn(ctx * 1024, device="cuda").to(dt) for n in ("kc", "vc")}
    case.update(qw=dev(bf16(rng, 256)), kw=dev(bf16(rng, 256)), q=dev(rng.standard_normal((tokens, 8192)).astype(np.float32)))
    k, v = (dev(rng.standard_normal((tokens, 1024)).astype(np.float32)) for _ in range(2))
    clean = _chunk(ops, case, tokens, start, ctx, k, v, tokens)
    if what == "query":
        case["q"][at, 512 * 5 + 3] = value  # query head 5
    else:
        {"key": k, "value": v, "none": v}[what][at, 256 * 1 + 7] += value  # kv head 1: query heads 4..7
    got, want = (_chunk(ops, case, tokens, start, ctx, k, v, step) for step in (tokens, 32))
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isinf(got), np.isinf(want))
    ok = np.isfinite(want)
    assert np.max(np.abs(got[ok] - want[ok]) / np.maximum(1, np.abs(want[ok]))) <= 1e-5  # two orders of fp32 sums
    assert np.max(np.abs(got[:at] - clean[:at])) <= 1e-5 and np.array_equal(got[:32], clean[:32])
    assert np.array_equal(np.delete(got, range(4, 8), 1), np.delete(clean, range(4, 8), 1))
