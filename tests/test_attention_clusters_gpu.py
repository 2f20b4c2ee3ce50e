"""The decode attention at the row counts where its cut over CTAs and clusters changes, against a float64 softmax."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), ".."))
from tests.test_kernels_gpu import bf16, dev, host  # noqa: E402

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# rows: around the first cluster's end (48 rows x 8 CTAs), all eight clusters, the tensor-core loop from
# 2048 rows on; three and five sequences past 2048 rows of cache take clusters of four, eight on a short one pairs of them
@pytest.mark.parametrize("kv_bf16,sequences,rows,ctx", [
    (False, 1, 384, 400), (False, 1, 385, 400), (False, 1, 3073, 3100), (False, 2, 1537, 1600), (False, 3, 2100, 2200), (False, 3, 5, 2200),
    (False, 5, 577, 2200), (True, 1, 384, 400), (True, 1, 385, 400), (True, 1, 2047, 2100), (True, 1, 2049, 2100), (True, 3, 2500, 2600), (True, 8, 2048, 2048),
    (False, 8, 500, 512)])
def test_decode_attention_cuts_vs_float64(cuda, kv_bf16, sequences, rows, ctx):
    from insignia_b200 import ops

    rng = np.random.default_rng(rows + sequences)
    dt = torch.bfloat16 if kv_bf16 else torch.float32
    kc, vc = (torch.randn(sequences, ctx * 1024, device="cuda").to(dt) for _ in range(2))
    qw, kw = bf16(rng, 256), bf16(rng, 256)
    qraw, kraw, v = (dev(rng.standard_normal((sequences, n)).astype(np.float32)) for n in (8192, 1024, 1024))
    pos = torch.full((1,), rows - 1, dtype=torch.int32, device="cuda")
    scratch = torch.zeros(sequences * ops.gqa_scratch("cuda").numel(), dtype=torch.uint8, device="cuda")
    got = [host(ops.attention_batch(qraw, kraw, v, dev(qw), dev(kw), kc, vc, pos, ctx, scratch, sequences, fast_trig=False)) for _ in range(2)]
    assert np.array_equal(got[0], got[1])  # the scratch is left ready, and the order of arrival does not matter
    assert int(scratch.view(sequences, -1)[:, :64].to(torch.int32).sum().item()) == 0
    q = host(qraw).astype(np.float64).reshape(sequences, 16, 512)[:, :, :256]
    w = (qw.astype(np.uint32) << 16).view(np.float32).astype(np.float64)
    q = q / np.sqrt((q * q).mean(-1, keepdims=True) + 1e-6) * w
    ang = (rows - 1) * 1e7 ** (-2.0 * np.arange(32) / 64)
    lo, hi = q[..., :32].copy(), q[..., 32:64].copy()
    q[..., :32], q[..., 32:64] = lo * np.cos(ang) - hi * np.sin(ang), hi * np.cos(ang) + lo * np.sin(ang)
    K, V = (host(c.float()).astype(np.float64).reshape(sequences, ctx, 4, 256)[:, :rows] for c in (kc, vc))
    for s in {0, sequences - 1}:
        for h in range(16):
            x = K[s, :, h >> 2] @ q[s, h] / 16
            p = np.exp(x - x.max())
            want = (p / p.sum()) @ V[s, :, h >> 2]
            # fp32 sums over 256 dims and `rows` weights, the rotation angle good to rows * 2^-24; with the bf16 cache the query
            # and the weights go in as two bf16 pieces (2^-16 of each)
            assert np.max(np.abs(got[0].reshape(sequences, 16, 256)[s, h] - want)) <= (2e-4 if kv_bf16 else 5e-5), (s, h)


@pytest.mark.parametrize("kv_bf16", [False, True])
@pytest.mark.parametrize("sequences,rows", [(8, 1), (8, 128), (8, 129), (7, 384)])
def test_pairs_of_clusters_equal_one(cuda, kv_bf16, sequences, rows):
    """Seven sequences or more on short caches run two clusters of four each where a single step runs one of eight."""
    from insignia_b200 import ops

    rng = np.random.default_rng(rows)
    ctx, dt = 400, torch.bfloat16 if kv_bf16 else torch.float32
    kc, vc = (torch.randn(sequences, ctx * 1024, device="cuda").to(dt) for _ in range(2))
    qw, kw = dev(bf16(rng, 256)), dev(bf16(rng, 256))
    qraw, kraw, v = (dev(rng.standard_normal((sequences, n)).astype(np.float32)) for n in (8192, 1024, 1024))
    pos = torch.full((1,), rows - 1, dtype=torch.int32, device="cuda")
    scratch = torch.zeros(sequences * ops.gqa_scratch("cuda").numel(), dtype=torch.uint8, device="cuda")
    got = host(ops.attention_batch(qraw, kraw, v, qw, kw, kc.clone(), vc.clone(), pos, ctx, scratch, sequences))
    want = [host(ops.attention_step(qraw[s], kraw[s], v[s], qw, kw, kc[s], vc[s], pos, ctx, scratch)) for s in range(sequences)]
    assert np.array_equal(got, np.stack(want))
