"""Products with many stages or units run on pairs of CTAs that multiply four row tiles with one set of digits, those with few in groups of 16 tokens."""
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


# Beyond 44 stages of 16 tokens an SM (148 SMs: 6512 pairs of tiles x groups of 16 x k-blocks), or 2.5 units, two CTAs share a group of 32.  One, two, three
# and five tiles with long sums and many groups; 101 to 104 tiles (the last four one to all there, the very last ragged), odd k-blocks, a full and
# a just begun last group; then below the line: 16 tokens a group beyond 48 tokens
@pytest.mark.parametrize("rows,cols,M", [(100, 12288, 1200), (256, 12288, 1090), (384, 12288, 600), (640, 12288, 400), (128 * 101, 4224, 49), (128 * 102, 4096, 64),
                                         (128 * 103 - 28, 4224, 65), (128 * 104, 4096, 96), (128 * 150, 2176, 100),
                                         (100, 128, 49), (640, 4096, 61), (1152, 1152, 97), (4096, 128, 512)])
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
@pytest.mark.parametrize("rows,cols,M", [(128, 12288, 1100), (300, 4096, 1100), (640, 4096, 700), (640, 1024, 70)])
def test_pairs_swiglu(cuda, rows, cols, M):
    from insignia_b200 import ops

    rng = np.random.default_rng(rows + M)
    mats = [rand_matrix(rng, rows, cols) for _ in range(2)]
    x = rng.standard_normal((M, cols)).astype(np.float32)
    g, u = (ops.repack_umma(dev(w), dev(s)) for w, s in mats)
    out = torch.zeros(M, rows, device="cuda")
    ops.gemv_fused(dev(x), [dict(packed=g, packed2=u, out=out, rows=rows, epilogue="swiglu")], layout=1, tokens=M, cols=cols,
                   umma_scratch=ops.umma_gemm_scratch(cols, M))
    for m in (0, 31, 32, M - 1):
        a, b = (orc.gemv_mlx_f64(w, s, x[m]) for w, s in mats)
        want = a / (1 + np.exp(-a)) * b
        assert np.max(np.abs(host(out)[m] - want)) <= 1e-5 * np.abs(want).max(), m


# On both sides of the line, where the stages draw it and where the units do (few k-blocks)
@pytest.mark.parametrize("rows,cols", [(2048, 4096), (1152, 2304), (4096, 1024), (12352, 256), (640, 128)])
def test_either_side_of_the_line(cuda, rows, cols):
    from insignia_b200 import ops

    rng = np.random.default_rng(rows + cols)
    w, s = rand_matrix(rng, rows, cols)
    P, line = ops.repack_umma(dev(w), dev(s)), pair_tokens(rows, cols)
    x = (rng.standard_normal((line, cols)) * rng.uniform(0.01, 30, (line, 1))).astype(np.float32)
    for M in (line - 1, line):
        y = host(ops.gemm_umma(P, dev(x[:M])))
        for m in (0, 17, M - 1):
            y64 = orc.gemv_mlx_f64(w, s, x[m])
            assert np.max(np.abs(y[m] - y64)) <= 4e-6 * np.abs(y64).max() + 1e-7, (M, m)


# Five tiles: the last unit is a single one, multiplied by both CTAs; seven of SwiGLU: the last unit leaves the second CTA without a result
@pytest.mark.parametrize("rows,cols,swiglu", [(640, 12288, False), (4096, 4096, False), (256, 4096, False), (128 * 37, 512, False), (896, 4096, True)])
def test_pairs_have_the_same_bits_whoever_arrives_last(cuda, rows, cols, swiglu):
    """What one CTA of a pair hands the other (copied stages, emptied accumulators), and whichever pair finds or adds the other parts of a unit,
    shows in no bit.  Other work on the GPU moves the arrivals."""
    from insignia_b200 import ops

    M = pair_tokens(rows, cols, swiglu)
    rng = np.random.default_rng(rows + M)
    mats = [rand_matrix(rng, rows, cols) for _ in range(1 + swiglu)]
    x = (rng.standard_normal((M, cols)) * 2).astype(np.float32)
    packed = [ops.repack_umma(dev(w), dev(s)) for w, s in mats]
    seg = dict(packed=packed[0], rows=rows, epilogue="store")
    if swiglu:
        seg.update(packed2=packed[1], epilogue="swiglu")
    xd, scratch, calls = dev(x), ops.umma_gemm_scratch(cols, M), 60
    outs = torch.zeros(calls, M, rows, device="cuda")
    side, junk = torch.cuda.Stream(), torch.randn(1 << 22, device="cuda")
    torch.cuda.synchronize()
    for i in range(calls):
        with torch.cuda.stream(side):
            for _ in range(i % 4):
                junk[: 1 << (12 + i % 11)].mul_(1.0)
        ops.gemv_fused(xd, [dict(seg, out=outs[i])], layout=1, tokens=M, cols=cols, umma_scratch=scratch, pdl=i % 2 == 1)
    torch.cuda.synchronize()
    assert bool((outs == outs[0]).all())
    for m in (0, 15, 16, M // 2, M - 1):
        y64 = [orc.gemv_mlx_f64(w, s, x[m]) for w, s in mats]
        want = y64[0] / (1 + np.exp(-y64[0])) * y64[1] if swiglu else y64[0]
        assert np.max(np.abs(host(outs[0, m]) - want)) <= (2e-5 if swiglu else 4e-6) * np.abs(want).max(), m


def test_pairs_fused_inproj(cuda):
    """in_proj(qkv|z|a|b) of a long pass on pairs: RMSNorm per token, conv + SiLU with the history carried through the tokens, store, decay, beta; segments
    of three, two, one and one tiles (the last two of 32 rows) in units of four."""
    from insignia_b200 import mxfp4, ops

    rng = np.random.default_rng(41)
    nq, nz, cols = 384, 256, 4096
    T = pair_tokens(nq + nz + 128 + 128, cols, last=9)
    (wq, sq), (wz, sz) = rand_matrix(rng, nq, cols), rand_matrix(rng, nz, cols)
    (wa, sa), (wb, sb) = rand_matrix(rng, 32, cols, std=0.05), rand_matrix(rng, 32, cols, std=0.05)
    conv_w = mxfp4.f32_to_bf16_bits((0.5 * rng.standard_normal((nq, 4))).astype(np.float32))
    A_log, dt = rng.uniform(-1, 1, 32).astype(np.float32), mxfp4.f32_to_bf16_bits((0.5 * rng.standard_normal(32)).astype(np.float32))
    nw = bf16(rng, cols)
    P = [ops.repack_umma(dev(w), dev(s)) for w, s in ((wq, sq), (wz, sz), (wa, sa), (wb, sb))]
    state0 = (rng.standard_normal(nq * 3) * 0.3).astype(np.float32)
    conv_state, err = dev(state0.copy()), torch.zeros(1, dtype=torch.int32, device="cuda")
    out = [torch.zeros(T, r, device="cuda") for r in (nq, nz, 32, 32)]
    hidden = (rng.standard_normal((T, cols)) * 3).astype(np.float32)
    ops.gemv_fused(dev(hidden), [
        dict(packed=P[0], out=out[0], rows=nq, epilogue="conv_silu", conv_state=conv_state, conv_w=dev(conv_w)),
        dict(packed=P[1], out=out[1], rows=nz, epilogue="store"),
        dict(packed=P[2], out=out[2], rows=32, epilogue="decay", A_log=dev(A_log), dt_bias=dev(dt)),
        dict(packed=P[3], out=out[3], rows=32, epilogue="beta")], prologue="rmsnorm", norm_w=dev(nw), layout=1, error_flag=err, tokens=T, cols=cols,
        umma_scratch=ops.umma_gemm_scratch(cols, T))
    gq, gz, ga, gb = (host(o) for o in out)
    ref_state = state0.copy()
    for m in range(T):
        n = orc.rmsnorm_bf16(hidden[m], nw)
        q = orc.gemv_mlx(wq, sq, n)
        orc.causal_conv4_silu(q, ref_state, conv_w)
        assert np.max(np.abs(gq[m] - q)) <= 2e-5 * max(1.0, np.abs(q).max()), m
        if m % 16 in (0, 15) or m == T - 1:
            a, b = orc.gemv_mlx(wa, sa, n), orc.gemv_mlx(wb, sb, n)
            orc.deltanet_parameters(a, b, A_log, dt)
            assert np.max(np.abs(gz[m] - orc.gemv_mlx(wz, sz, n))) <= 2e-5, m
            assert np.max(np.abs(ga[m] - a)) <= 2e-5 * max(1.0, np.abs(a).max()) and np.max(np.abs(gb[m] - b)) <= 2e-6, m
    assert np.max(np.abs(host(conv_state) - ref_state)) <= 2e-5 * np.abs(ref_state).max()
    assert int(err.item()) == 0


@pytest.mark.parametrize("prologue", ["gated_rmsnorm", "sigmoid_gate", "sigmoid_gate_head0", "sigmoid_gate_qproj"])
def test_pairs_residual_behind_each_gate(cuda, prologue):
    """The out and o projections of a long pass on pairs against the same tokens in calls of 16 (the other form, which the oracle tests): two orders of
    fp32 sums, each within 4e-7 of the largest."""
    from insignia_b200 import ops

    rng = np.random.default_rng(len(prologue))
    rows, cols = 1000, 4096
    T = pair_tokens(rows, cols, last=1)
    P = ops.repack_umma(*(dev(a) for a in rand_matrix(rng, rows, cols)))
    x = dev(rng.standard_normal((T, cols)).astype(np.float32))
    aux = dev(rng.standard_normal((T, cols if prologue in ("gated_rmsnorm", "sigmoid_gate") else 2 * cols)).astype(np.float32))
    res, nw = rng.standard_normal((T, rows)).astype(np.float32), dev(bf16(rng, 128))
    kw = dict(prologue=prologue, layout=1, cols=cols, umma_scratch=ops.umma_gemm_scratch(cols, T), **(dict(norm_w=nw) if prologue == "gated_rmsnorm" else {}))
    got, want = dev(res.copy()), dev(res.copy())
    ops.gemv_fused(x, [dict(packed=P, out=got, rows=rows, epilogue="residual")], aux=aux, tokens=T, **kw)
    for m in range(0, T, 16):
        n = min(16, T - m)
        ops.gemv_fused(x[m:m + n], [dict(packed=P, out=want[m:m + n], rows=rows, epilogue="residual")], aux=aux[m:m + n], tokens=n, **kw)
    got, want = host(got), host(want)
    assert np.max(np.abs(got - want)) <= 8e-7 * np.abs(want).max()
    assert np.max(np.abs(want - res)) > 0.1
