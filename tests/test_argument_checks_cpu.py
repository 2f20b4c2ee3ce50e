"""Calls that a kernel could not serve are refused before anything is launched (checked without a GPU: a launch would fail
with another status)."""
import ctypes as C
import os
import sys

import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), ".."))

E_SHAPE, E_ARG = -1, -3
SOME = 1 << 20  # a pointer nobody follows


def attn_op(**kw):
    from insignia_b200 import _lib

    op = _lib.AttnOp()
    for f in ("qraw", "k_raw", "v", "q_norm_w", "k_norm_w", "k_cache", "v_cache", "out", "position", "scratch"):
        setattr(op, f, SOME)
    op.max_context, op.scratch_bytes = 4096, 1 << 40
    for k, v in kw.items():
        setattr(op, k, v)
    return op


@pytest.mark.parametrize("tokens", [9, 32, 33, 512])
def test_a_chunk_of_more_than_eight_tokens_has_no_image(tokens):
    from insignia_b200 import _lib

    assert _lib.lib().insg_attention_chunk(C.byref(attn_op(image=SOME)), tokens, SOME, 0, None) == E_SHAPE
    assert b"digit image" in _lib.lib().insg_last_error()


def gemv_op(tokens=1, rows=256, cols=4096, prologue="plain", **kw):
    from insignia_b200 import _lib, ops

    op = _lib.GemvOp()
    op.in_, op.cols, op.prologue, op.n_segments, op.layout, op.tokens = SOME, cols, ops.PRO[prologue], 1, 1, tokens
    op.seg[0].packed, op.seg[0].out, op.seg[0].rows = SOME, SOME, rows
    for k, v in kw.items():
        setattr(op, k, v)
    return op


@pytest.mark.parametrize("tokens", [1, 8])
def test_the_rms_factor_of_a_prepared_input_needs_its_sums(tokens):
    from insignia_b200 import _lib

    assert _lib.lib().insg_gemv_fused(C.byref(gemv_op(tokens, prologue="prepared", prep_rms=1)), None) == E_ARG
    assert b"sums" in _lib.lib().insg_last_error()


@pytest.mark.parametrize("tokens", [0, -1, 4097])
def test_a_product_takes_1_to_4096_tokens(tokens):
    from insignia_b200 import _lib

    assert _lib.lib().insg_mxfp4_gemm_umma(SOME, SOME, SOME, 256, 4096, tokens, SOME, 1 << 40, None) == E_SHAPE


@pytest.mark.parametrize("rows,cols", [(3_000_000, 128), (1_000_000, 12288)])
def test_three_tokens_of_very_many_rows_are_not_refused(rows, cols):
    """Their sums no longer fit one launch: they go as two and one.  Here the launch itself fails, for want of a device."""
    import torch

    from insignia_b200 import _lib

    if torch.cuda.is_available():
        pytest.skip("would launch")
    L = _lib.lib()
    assert [L.insg_mxfp4_gemv_packed(SOME, SOME, SOME, rows, cols, m, None) for m in (1, 2, 3)] == [-2] * 3  # INSG_E_CUDA


@pytest.mark.parametrize("entry", ["insg_deltanet_gated_step", "insg_deltanet_gated_step_apart"])
@pytest.mark.parametrize("change", [dict(layout=0), dict(tokens=2), dict(prologue="plain"), dict(cols=896), dict(cols=0), dict(rows=2048), dict(epilogue="residual"), dict(n_segments=2)])
def test_a_gated_step_takes_one_kind_of_product_on_every_route(entry, change):
    """The step reads 4096 gates of the product whichever way it goes: what does not make them is refused before the way is chosen."""
    from insignia_b200 import _lib, ops

    kw = dict(rows=4096, cols=1024, prologue="prepared")
    kw.update(change)
    epilogue = kw.pop("epilogue", "store")
    op, step = gemv_op(**kw), _lib.DeltaOp()
    op.seg[0].epilogue = ops.EPI[epilogue]
    for name, _ in step._fields_:
        setattr(step, name, SOME)
    assert getattr(_lib.lib(), entry)(C.byref(op), C.byref(step), None) == E_SHAPE
    step.norm_w = None
    assert getattr(_lib.lib(), entry)(C.byref(op), C.byref(step), None) == E_ARG


@pytest.mark.parametrize("change", [dict(layout=0), dict(prologue="plain"), dict(prologue="rmsnorm", norm_w=SOME), dict(tokens=9)])
def test_a_launch_that_does_not_hold_back_the_gated_step_is_refused(change):
    """pdl = 2 promises that the launch behind starts when this launch's own input is complete; other launches let it start at once."""
    from insignia_b200 import _lib

    op = gemv_op(**{**dict(prologue="prepared", pdl=2, umma_scratch=SOME, umma_scratch_bytes=1 << 40), **change})
    assert _lib.lib().insg_gemv_fused(C.byref(op), None) == E_ARG
    assert b"pdl = 2" in _lib.lib().insg_last_error()


@pytest.mark.parametrize("rows,cols", [(3_000_000, 128), (1_000_000, 12288)])
def test_nor_where_the_records_do_not_start_on_sixteen_bytes(rows, cols):
    """Such records stay on mma.sync whatever their number, whose sums of three tokens are the ones that go as two and one."""
    import torch

    from insignia_b200 import _lib

    if torch.cuda.is_available():
        pytest.skip("would launch")
    assert [_lib.lib().insg_mxfp4_gemv_packed(SOME + 8, SOME, SOME, rows, cols, m, None) for m in (1, 2, 3)] == [-2] * 3  # INSG_E_CUDA
