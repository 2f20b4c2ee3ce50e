"""The one-to-eight-token product's variants (two matrices, one residual segment, gated norm, nothing left prepared) on both sides of the sizes from which
they are taken: whole octets of k-blocks, one unit per cluster; with a ragged last tile."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), ".."))
from oracle import oracle as orc  # noqa: E402
from tests.test_kernels_gpu import bf16, dev, host, rand_matrix  # noqa: E402

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

TOKENS = [1, 2, 3, 5, 8]


def image_of(rng, tokens, cols):
    """A digit image as a residual launch leaves it, and the vectors it stands for."""
    from insignia_b200 import _lib, ops

    P, w = ops.repack_umma(*(dev(a) for a in rand_matrix(rng, cols, 128))), bf16(rng, cols)
    h = dev((rng.standard_normal((tokens, cols)) * rng.uniform(0.1, 30, (tokens, 1))).astype(np.float32))
    image = torch.zeros(_lib.lib().insg_mxfp4_digit_image_bytes(cols, tokens), dtype=torch.uint8, device="cuda")
    sums = torch.zeros(tokens * cols // 32, device="cuda")
    ops.gemv_fused(dev(rng.standard_normal((tokens, 128)).astype(np.float32)), [dict(packed=P, out=h, rows=cols, epilogue="residual", prep=image, prep_w=dev(w), prep_partials=sums)],
                   layout=1, tokens=tokens, cols=128)
    h = host(h)
    wf = (w.astype(np.uint32) << 16).view(np.float32)
    rms = np.sqrt((h.astype(np.float64) ** 2).mean(1, keepdims=True) + 1e-6)
    return image, sums, h * wf, h * wf.astype(np.float64) / rms


def close(got, want, bound):
    for m in range(len(want)):
        assert np.max(np.abs(got[m] - want[m])) <= bound * np.abs(want[m]).max(), m


def products(w, s, x):
    return np.stack([orc.gemv_mlx_f64(w, s, v.astype(np.float32)) for v in x])


# 1024 and 4096 columns: whole octets of k-blocks; 1152, 4224: not.  Three tiles, the last of 44 rows; more units than clusters (74 tiles)
@pytest.mark.parametrize("tokens", TOKENS)
@pytest.mark.parametrize("rows,cols", [(300, 1024), (300, 1152), (9472, 1024)])
def test_two_matrices(cuda, tokens, rows, cols):
    from insignia_b200 import ops

    rng = np.random.default_rng(rows + cols + tokens)
    image, sums, _, x = image_of(rng, tokens, cols)
    (wg, sg), (wu, su) = rand_matrix(rng, rows, cols), rand_matrix(rng, rows, cols)
    out, err = torch.zeros(tokens, rows, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    ops.gemv_fused(image, [dict(packed=ops.repack_umma(dev(wg), dev(sg)), packed2=ops.repack_umma(dev(wu), dev(su)), out=out, rows=rows, epilogue="swiglu")],
                   prologue="prepared", prep_partials=sums, prep_rms=True, layout=1, tokens=tokens, cols=cols, error_flag=err)
    g, u = products(wg, sg, x), products(wu, su, x)
    close(host(out), g / (1 + np.exp(-g)) * u, 1e-5)  # silu by fast exponentials
    assert int(err.item()) == 0


# one residual segment: three units; more units than clusters; an image past half an SM (streamed with three tokens and more); k-blocks that are no octets
@pytest.mark.parametrize("tokens", TOKENS)
@pytest.mark.parametrize("rows,cols", [(300, 1024), (300, 4096), (9472, 1024), (300, 12288), (300, 1152), (300, 11904)])
def test_one_residual_segment(cuda, tokens, rows, cols):
    from insignia_b200 import ops

    rng = np.random.default_rng(rows + cols + tokens)
    image, _, x, _ = image_of(rng, tokens, cols)
    w, s = rand_matrix(rng, rows, cols)
    res = rng.standard_normal((tokens, rows)).astype(np.float32)
    out, err = dev(res.copy()), torch.zeros(1, dtype=torch.int32, device="cuda")
    for _ in range(2):  # the second call adds to what the first one left
        ops.gemv_fused(image, [dict(packed=ops.repack_umma(dev(w), dev(s)), out=out, rows=rows, epilogue="residual")], prologue="prepared", layout=1, tokens=tokens,
                       cols=cols, error_flag=err)
    close(host(out), res + 2 * products(w, s, x), 4e-6)
    assert int(err.item()) == 0


@pytest.mark.parametrize("tokens", TOKENS)
@pytest.mark.parametrize("rows,cols", [(300, 1024), (9472, 1024), (300, 1152)])
@pytest.mark.parametrize("x_out", [False, True])
def test_gated_norm(cuda, tokens, rows, cols, x_out):
    from insignia_b200 import ops

    rng = np.random.default_rng(rows + cols + tokens)
    core, z = (rng.standard_normal((tokens, cols)).astype(np.float32) * 3 for _ in range(2))
    nw, (w, s) = bf16(rng, 128), rand_matrix(rng, rows, cols)
    res = rng.standard_normal((tokens, rows)).astype(np.float32)
    out, xo, err = dev(res.copy()), torch.zeros(tokens, cols, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    ops.gemv_fused(dev(core), [dict(packed=ops.repack_umma(dev(w), dev(s)), out=out, rows=rows, epilogue="residual")], prologue="gated_rmsnorm", aux=dev(z), norm_w=dev(nw),
                   layout=1, tokens=tokens, cols=cols, error_flag=err, **(dict(x_out=xo) if x_out else {}))
    x = np.stack([orc.rmsnorm_bf16(core[m].reshape(-1, 128), nw, gate=z[m].reshape(-1, 128)).reshape(-1) for m in range(tokens)])
    close(host(out), res + products(w, s, x), 1e-5)  # fast exponentials in the gate
    if x_out:
        close(host(xo), x, 1e-5)
    assert int(err.item()) == 0


@pytest.mark.parametrize("tokens", TOKENS)
@pytest.mark.parametrize("cols", [1024, 1152])
def test_projections_that_leave_nothing_prepared(cuda, tokens, cols):
    """qkv|z|a|b of independent sequences from a prepared input: conv + SiLU (two tiles, the second of 44 rows), store, decay, beta (32 rows each)."""
    from insignia_b200 import mxfp4, ops

    rng = np.random.default_rng(cols + tokens)
    image, sums, _, x = image_of(rng, tokens, cols)
    rows = (172, 300, 32, 32)
    mats = [rand_matrix(rng, r, cols, std=0.05) for r in rows]
    conv_w = mxfp4.f32_to_bf16_bits((0.5 * rng.standard_normal((rows[0], 4))).astype(np.float32))
    A_log, dt = rng.uniform(-1, 1, 32).astype(np.float32), mxfp4.f32_to_bf16_bits((0.5 * rng.standard_normal(32)).astype(np.float32))
    hist = (rng.standard_normal((tokens, rows[0] * 3)) * 0.3).astype(np.float32)
    state, out = dev(hist.copy()), [torch.zeros(tokens, r, device="cuda") for r in rows]
    seg = [dict(packed=ops.repack_umma(dev(w), dev(s)), out=o, rows=r) for (w, s), o, r in zip(mats, out, rows)]
    seg[0].update(epilogue="conv_silu", conv_state=state, conv_w=dev(conv_w), conv_token_stride=rows[0] * 3)
    seg[1].update(epilogue="store")
    seg[2].update(epilogue="decay", A_log=dev(A_log), dt_bias=dev(dt))
    seg[3].update(epilogue="beta")
    ops.gemv_fused(image, seg, prologue="prepared", prep_partials=sums, prep_rms=True, layout=1, tokens=tokens, cols=cols)
    q, z, a, b = (products(w, s, x) for w, s in mats)
    cw, dtf = ((v.astype(np.uint32) << 16).view(np.float32).astype(np.float64) for v in (conv_w, dt))
    h = hist.reshape(tokens, rows[0], 3).astype(np.float64)
    conv = (h * cw[:, :3]).sum(2) + q * cw[:, 3]
    soft = np.log1p(np.exp(a + dtf))
    for got, want in zip(out, (conv / (1 + np.exp(-conv)), z, -np.exp(A_log.astype(np.float64)) * soft, 1 / (1 + np.exp(-b)))):
        close(host(got), want, 1e-5)
    close(host(state), np.concatenate([h[:, :, 1:], q[:, :, None]], 2).reshape(tokens, -1), 4e-6)
