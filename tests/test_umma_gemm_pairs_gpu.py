"""Products of more than 48 tokens run on pairs of CTAs that multiply four row tiles with one set of digits."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), ".."))
from oracle import oracle as orc  # noqa: E402
from tests.test_kernels_gpu import dev, host, rand_matrix  # noqa: E402

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# rows: one to nine tiles (the last four of a pair of CTAs: one, two, three or all there), a ragged last tile; cols: one k-block, an odd
# number of them; tokens: the first count of the form, a full and a just begun group, sixteen groups
@pytest.mark.parametrize("rows,cols,M", [(100, 128, 49), (256, 384, 64), (384, 1152, 65), (500, 512, 96), (640, 4096, 49), (768, 256, 97), (1152, 12288, 64),
                                         (4096, 128, 512), (19008, 512, 100)])
def test_pairs_vs_oracle(cuda, rows, cols, M):
    from insignia_b200 import ops

    rng = np.random.default_rng(rows + cols + M)
    w, s = rand_matrix(rng, rows, cols)
    x = (rng.standard_normal((M, cols)) * rng.uniform(0.01, 30, (M, 1))).astype(np.float32)
    P, scratch = ops.repack_umma(dev(w), dev(s)), ops.umma_gemm_scratch(cols, M)
    y = host(ops.gemm_umma(P, dev(x), scratch=scratch))
    for m in (0, 15, 16, 31, 32, M // 2, M - 1):
        y64 = orc.gemv_mlx_f64(w, s, x[m])
        assert np.max(np.abs(y[m] - y64)) <= 4e-6 * np.abs(y64).max() + 1e-7, m
    assert np.array_equal(host(ops.gemm_umma(P, dev(x), scratch=scratch)), y)


# SwiGLU: a unit is the gate and up tiles of two times 128 rows; an odd number of row tiles leaves the second CTA without
@pytest.mark.parametrize("rows,M", [(128, 49), (300, 64), (640, 70)])
def test_pairs_swiglu(cuda, rows, M):
    from insignia_b200 import ops

    rng = np.random.default_rng(rows + M)
    mats = [rand_matrix(rng, rows, 1024) for _ in range(2)]
    x = rng.standard_normal((M, 1024)).astype(np.float32)
    g, u = (ops.repack_umma(dev(w), dev(s)) for w, s in mats)
    out = torch.zeros(M, rows, device="cuda")
    ops.gemv_fused(dev(x), [dict(packed=g, packed2=u, out=out, rows=rows, epilogue="swiglu")], layout=1, tokens=M, cols=1024,
                   umma_scratch=ops.umma_gemm_scratch(1024, M))
    for m in (0, 31, 32, M - 1):
        a, b = (orc.gemv_mlx_f64(w, s, x[m]) for w, s in mats)
        want = a / (1 + np.exp(-a)) * b
        assert np.max(np.abs(host(out)[m] - want)) <= 1e-5 * np.abs(want).max(), m
