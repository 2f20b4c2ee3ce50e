"""The route a DeltaNet step beside its gate's product takes on a GPU that cannot hold the launch's clusters: the bits of the one launch."""
import ctypes as C
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), ".."))
from tests.test_kernels_gpu import bf16, dev, host, rand_matrix  # noqa: E402

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("cols,pdl", [(1024, False), (3072, True), (4096, False), (4096, True)])
def test_three_launches_have_the_bits_of_one(cuda, cols, pdl):
    from insignia_b200 import _lib, ops

    L, rng = _lib.lib(), np.random.default_rng(cols + pdl)
    W = {n: ops.repack_umma(*(dev(a) for a in rand_matrix(rng, r, c))) for n, r, c in (("src", cols, 1024), ("qkv", 8192, cols), ("z", 4096, cols), ("out", 512, 4096))}
    x, nw, dn, cw = dev(rng.standard_normal(1024).astype(np.float32)), dev(bf16(rng, cols)), dev(bf16(rng, 128)), dev(bf16(rng, 8192 * 4))
    a, b = dev(-rng.uniform(0.01, 2, 32).astype(np.float32)), dev(rng.uniform(0, 1, 32).astype(np.float32))
    conv0, state0 = dev(rng.standard_normal((8192, 3)).astype(np.float32)), dev((0.1 * rng.standard_normal(32 * 128 * 128)).astype(np.float32))
    got = []
    for entry in (L.insg_deltanet_gated_step, L.insg_deltanet_gated_step_apart):
        hidden, z, qkv, core, y = (torch.zeros(n, device="cuda") for n in (cols, 4096, 8192, 4096, 512))
        conv, state = conv0.clone(), state0.clone()
        image, core_image = (torch.zeros(L.insg_mxfp4_digit_image_bytes(c, 1), dtype=torch.uint8, device="cuda") for c in (cols, 4096))
        sums, err = torch.zeros(cols // 32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
        kw = dict(layout=1, error_flag=err)
        prep = dict(prologue="prepared", prep_partials=sums, prep_rms=True, cols=cols, **kw)
        for _ in range(3):  # the state and the history go on; the input changes
            ops.gemv_fused(x, [dict(packed=W["src"], out=hidden, rows=cols, epilogue="residual", prep=image, prep_w=nw, prep_partials=sums)], pdl=pdl, **kw)
            ops.gemv_fused(image, [dict(packed=W["qkv"], out=qkv, rows=8192, epilogue="conv_silu", conv_state=conv, conv_w=cw)], pdl=2 if pdl else 0, **prep)
            op, step = ops._gemv_op(image, [dict(packed=W["z"], out=z, rows=4096, epilogue="store")], pdl=pdl, **prep), _lib.DeltaOp()
            for name, t in dict(state=state, q16=qkv, out32=core, g32=a, beta32=b, norm_w=dn, image=core_image).items():
                setattr(step, name, t.data_ptr())
            step.k16, step.v32 = qkv.data_ptr() + 4 * 2048, qkv.data_ptr() + 4 * 4096
            _lib.check(entry(C.byref(op), C.byref(step), torch.cuda.current_stream().cuda_stream))
            ops.gemv_fused(core_image, [dict(packed=W["out"], out=y, rows=512, epilogue="residual")], prologue="prepared", cols=4096, pdl=pdl, **kw)
        assert int(err.item()) == 0
        got.append([host(t) for t in (z, core, state, core_image, y)])
    for one, other in zip(*got):
        assert np.array_equal(one, other)
