"""Products that hand their results on as digit images (layout 1, one to eight tokens) against the same chain in fp32 vectors."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), ".."))
from tests.test_kernels_gpu import bf16, dev, host, rand_matrix  # noqa: E402

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# inter: 128 = one k-block for four CTAs (three have none), 1152 = nine (ragged quarters), 3200 = 25
@pytest.mark.parametrize("tokens,inter", [(1, 1152), (2, 128), (3, 3200), (8, 1152)])
def test_prepared_chain_equals_fp32_chain(cuda, tokens, inter):
    """gate|up + SwiGLU -> down + residual -> RMSNorm'd product: the second and third take prepared inputs in one chain and
    convert for themselves in the other.  An image holds 25 bits of every value relative to its 32-element group, as the
    in-kernel conversion does, so the two differ by the rounding of one fp32 factor (2^-23) through three products."""
    from insignia_b200 import _lib, ops

    rng = np.random.default_rng(tokens * inter)
    P = {n: ops.repack_umma(*(dev(a) for a in rand_matrix(rng, r, c))) for n, r, c in
         (("g", inter, 4096), ("u", inter, 4096), ("d", 4096, inter), ("n", 256, 4096))}
    nw, nw2 = dev(bf16(rng, 4096)), dev(bf16(rng, 4096))
    hidden0 = (rng.standard_normal((tokens, 4096)) * rng.uniform(0.1, 30, (tokens, 1))).astype(np.float32)
    got = {}
    for prepared in (False, True):
        h, act, out = dev(hidden0.copy()), torch.zeros(tokens, inter, device="cuda"), torch.zeros(tokens, 256, device="cuda")
        image = [torch.zeros(_lib.lib().insg_mxfp4_digit_image_bytes(c, tokens), dtype=torch.uint8, device="cuda") for c in (inter, 4096)]
        sums, err = torch.zeros(tokens * 128, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
        kw = dict(layout=1, tokens=tokens, error_flag=err)
        for _ in range(2):
            a, b = (dict(prep=image[0]), dict(prep=image[1], prep_w=nw2, prep_partials=sums)) if prepared else ({}, {})
            ops.gemv_fused(h, [dict(packed=P["g"], packed2=P["u"], out=act, rows=inter, epilogue="swiglu", **a)], prologue="rmsnorm", norm_w=nw, cols=4096, **kw)
            ops.gemv_fused(image[0] if prepared else act, [dict(packed=P["d"], out=h, rows=4096, epilogue="residual", **b)],
                           prologue="prepared" if prepared else "plain", cols=inter, **kw)
            ops.gemv_fused(image[1] if prepared else h, [dict(packed=P["n"], out=out, rows=256, epilogue="store")], cols=4096,
                           **(dict(prologue="prepared", prep_partials=sums, prep_rms=True) if prepared else dict(prologue="rmsnorm", norm_w=nw2)), **kw)
        assert int(err.item()) == 0
        got[prepared] = [host(x) for x in (act, h, out)]
    for x, y in zip(*got.values()):
        for m in range(tokens):
            assert np.max(np.abs(x[m] - y[m])) <= 2e-6 * np.abs(x[m]).max(), m


def _project(ops, P, image_or_vector, n, **kw):
    out, err = torch.zeros(n, 256, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    ops.gemv_fused(image_or_vector, [dict(packed=P, out=out, rows=256, epilogue="store")], layout=1, tokens=n, cols=4096, error_flag=err, **kw)
    assert int(err.item()) == 0
    return host(out)


@pytest.mark.parametrize("sequences", [1, 2, 3, 5, 8])
def test_gated_deltanet_step_leaves_the_next_input(cuda, sequences):
    from insignia_b200 import _lib, ops

    rng = np.random.default_rng(10 + sequences)
    n, S = sequences, 32 * 128 * 128
    P = ops.repack_umma(*(dev(a) for a in rand_matrix(rng, 256, 4096)))
    qkv, z = (dev(rng.standard_normal((n, c)).astype(np.float32)) for c in (8192, 4096))
    g, beta = dev(-rng.uniform(0, 2, (n, 32)).astype(np.float32)), dev(rng.uniform(0, 1, (n, 32)).astype(np.float32))
    nw, state0 = dev(bf16(rng, 128)), dev((0.1 * rng.standard_normal((sequences, S))).astype(np.float32))
    flat = qkv.view(-1)
    want_state, state = state0.clone(), state0.clone()
    want = ops.deltanet_decode_batch(want_state, flat, flat[2048:], flat[4096:], g, beta, sequences, 8192)
    out = torch.zeros(n, 4096, device="cuda")
    image = torch.zeros(_lib.lib().insg_mxfp4_digit_image_bytes(4096, n), dtype=torch.uint8, device="cuda")
    p = lambda t: t.data_ptr()  # noqa: E731
    _lib.check(_lib.lib().insg_deltanet_decode_gated(p(state), S, p(flat), p(flat) + 4 * 2048, p(flat) + 4 * 4096, p(g), p(beta), p(out), sequences, 8192,
                                                     p(z), p(nw), p(image), 0, torch.cuda.current_stream().cuda_stream))
    # two fp32 sums over 128 terms of magnitude <= 1 in another order: 128 * 2^-24 of the largest
    assert torch.max(torch.abs(out - want)) <= 1e-5 * want.abs().max() and torch.max(torch.abs(state - want_state)) <= 1e-5 * want_state.abs().max()
    got = _project(ops, P, image, n, prologue="prepared")
    ref = _project(ops, P, out, n, prologue="gated_rmsnorm", aux=z, norm_w=nw)
    assert np.max(np.abs(got - ref)) <= 2e-6 * np.abs(ref).max()  # the order of one 128-term sum of squares, and 2^-24 of a group's largest


@pytest.mark.parametrize("sequences,elementwise,kv_bf16,ctx", [(1, False, False, 5), (1, True, True, 2100), (3, False, True, 130), (8, True, False, 300)])
def test_attention_step_leaves_the_next_input(cuda, sequences, elementwise, kv_bf16, ctx):
    import ctypes as C

    from insignia_b200 import _lib, ops

    rng = np.random.default_rng(sequences + ctx)
    n, dt = sequences, torch.bfloat16 if kv_bf16 else torch.float32
    P = ops.repack_umma(*(dev(a) for a in rand_matrix(rng, 256, 4096)))
    qraw, kraw, v = (dev(rng.standard_normal((n, c)).astype(np.float32)) for c in (8192, 1024, 1024))
    kc, vc = (torch.randn(n, ctx * 1024, device="cuda").to(dt) for _ in range(2))
    qw, kw, pos = dev(bf16(rng, 256)), dev(bf16(rng, 256)), torch.full((1,), ctx - 1, dtype=torch.int32, device="cuda")
    scratch = torch.zeros(n * ops.gqa_scratch("cuda").numel(), dtype=torch.uint8, device="cuda")
    want = ops.attention_batch(qraw, kraw, v, qw, kw, kc.clone(), vc.clone(), pos, ctx, scratch, n)
    out = torch.zeros(n, 4096, device="cuda")
    image = torch.zeros(_lib.lib().insg_mxfp4_digit_image_bytes(4096, n), dtype=torch.uint8, device="cuda")
    op = _lib.AttnOp()
    for name, t in dict(qraw=qraw, k_raw=kraw, v=v, q_norm_w=qw, k_norm_w=kw, k_cache=kc, v_cache=vc, out=out, position=pos, scratch=scratch, image=image).items():
        setattr(op, name, t.data_ptr())
    op.max_context, op.kv_dtype, op.fast_trig, op.scratch_bytes, op.gate_elementwise = ctx, int(kv_bf16), 1, scratch.numel(), int(elementwise)
    _lib.check(_lib.lib().insg_attention_batch(C.byref(op), n, kc.numel() // n * kc.element_size(), torch.cuda.current_stream().cuda_stream))
    assert torch.equal(out, want)
    got = _project(ops, P, image, n, prologue="prepared")
    ref = _project(ops, P, out, n, prologue="sigmoid_gate_qproj" if elementwise else "sigmoid_gate_head0", aux=qraw)
    assert np.array_equal(got, ref)  # the same gate, groups and digits wherever they are made
