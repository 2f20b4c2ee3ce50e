"""The DeltaNet step made in the launch of the product that gates its output, against the product, the step and the gated norm as
operations of their own: the same bits."""
import ctypes as C
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), ".."))
from tests.test_kernels_gpu import bf16, dev, host, rand_matrix  # noqa: E402

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# cols: one, three and four stages of weights a CTA; pdl: beside an in-projection that lets it start early
@pytest.mark.parametrize("cols,pdl", [(1024, False), (3072, True), (4096, False), (4096, True)])
def test_step_beside_its_gate_has_the_bits_of_the_separate_operations(cuda, cols, pdl):
    from insignia_b200 import _lib, ops

    L, rng = _lib.lib(), np.random.default_rng(cols + pdl)
    p = lambda t: t.data_ptr()  # noqa: E731
    W = {n: ops.repack_umma(*(dev(a) for a in rand_matrix(rng, r, c))) for n, r, c in
         (("src", cols, 1024), ("qkv", 8192, cols), ("z", 4096, cols), ("a", 32, cols), ("b", 32, cols), ("out", 512, 4096))}
    x, nw, dn = dev(rng.standard_normal(1024).astype(np.float32)), dev(bf16(rng, cols)), dev(bf16(rng, 128))
    cw, A, dt = dev(bf16(rng, 8192 * 4)), dev(rng.uniform(-1, 1, 32).astype(np.float32)), dev(bf16(rng, 32))
    conv0, state0 = dev(rng.standard_normal((8192, 3)).astype(np.float32)), dev((0.1 * rng.standard_normal(32 * 128 * 128)).astype(np.float32))
    got = {}
    for beside in (False, True):
        hidden, z, qkv, a, b = (torch.zeros(n, device="cuda") for n in (cols, 4096, 8192, 32, 32))
        core, y, conv, state = torch.zeros(4096, device="cuda"), torch.zeros(512, device="cuda"), conv0.clone(), state0.clone()
        image, core_image = (torch.zeros(L.insg_mxfp4_digit_image_bytes(c, 1), dtype=torch.uint8, device="cuda") for c in (cols, 4096))
        sums, err = torch.zeros(cols // 32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
        kw = dict(layout=1, error_flag=err)
        prep = dict(prologue="prepared", prep_partials=sums, prep_rms=True, cols=cols, **kw)
        for _ in range(3):  # the state and the histories go on; the input changes
            ops.gemv_fused(x, [dict(packed=W["src"], out=hidden, rows=cols, epilogue="residual", prep=image, prep_w=nw, prep_partials=sums)], pdl=pdl, **kw)
            gates = [dict(packed=W["a"], out=a, rows=32, epilogue="decay", A_log=A, dt_bias=dt), dict(packed=W["b"], out=b, rows=32, epilogue="beta")]
            first = [dict(packed=W["qkv"], out=qkv, rows=8192, epilogue="conv_silu", conv_state=conv, conv_w=cw)]
            gate = [dict(packed=W["z"], out=z, rows=4096, epilogue="store")]
            if beside:
                ops.gemv_fused(image, first + gates, pdl=2 if pdl else 0, **prep)
                op, step = ops._gemv_op(image, gate, pdl=pdl, **prep), _lib.DeltaOp()
                for name, t in dict(state=state, q16=qkv, out32=core, g32=a, beta32=b, norm_w=dn, image=core_image).items():
                    setattr(step, name, p(t))
                step.k16, step.v32 = p(qkv) + 4 * 2048, p(qkv) + 4 * 4096
                _lib.check(L.insg_deltanet_gated_step(C.byref(op), C.byref(step), torch.cuda.current_stream().cuda_stream))
                ops.gemv_fused(core_image, [dict(packed=W["out"], out=y, rows=512, epilogue="residual")], prologue="prepared", cols=4096, pdl=pdl, **kw)
            else:
                ops.gemv_fused(image, first + gate + gates, **prep)
                core.copy_(ops.deltanet_decode(state, qkv, qkv[2048:], qkv[4096:], a, b))
                ops.gemv_fused(core, [dict(packed=W["out"], out=y, rows=512, epilogue="residual")], prologue="gated_rmsnorm", aux=z, norm_w=dn, cols=4096, **kw)
        assert int(err.item()) == 0
        got[beside] = [host(t) for t in (hidden, z, qkv, a, b, core, state, conv, y)]
    for one, other in zip(*got.values()):
        assert np.array_equal(one, other)


def test_step_beside_its_gate_refuses_other_products(cuda):
    from insignia_b200 import _lib, ops

    L, rng = _lib.lib(), np.random.default_rng(0)
    P = ops.repack_umma(*(dev(a) for a in rand_matrix(rng, 4096, 1024)))
    t, image = torch.zeros(32 * 128 * 128, device="cuda"), torch.zeros(L.insg_mxfp4_digit_image_bytes(4096, 2), dtype=torch.uint8, device="cuda")
    step = _lib.DeltaOp()
    for name, _ in step._fields_:
        setattr(step, name, t.data_ptr())
    stream = torch.cuda.current_stream().cuda_stream
    seg = dict(packed=P, out=t, rows=4096, epilogue="store")
    good = dict(prologue="prepared", layout=1, cols=1024)
    for change in (dict(layout=0), dict(tokens=2), dict(prologue="plain"), dict(cols=896)):
        op = ops._gemv_op(image, [seg], **{**good, **change})
        assert L.insg_deltanet_gated_step(C.byref(op), C.byref(step), stream) < 0, change
    for s in (dict(seg, rows=4096 - 128), dict(seg, epilogue="residual")):
        op = ops._gemv_op(image, [s], **good)
        assert L.insg_deltanet_gated_step(C.byref(op), C.byref(step), stream) < 0, s
    step.image = None
    op = ops._gemv_op(image, [seg], **good)
    assert L.insg_deltanet_gated_step(C.byref(op), C.byref(step), stream) < 0
