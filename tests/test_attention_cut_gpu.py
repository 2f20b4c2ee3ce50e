"""Decode attention on both sides of the row counts where the cut over CTAs and clusters changes, against float64."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), ".."))
from tests.test_kernels_gpu import host  # noqa: E402

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# blocks of 32 rows a CTA; one cluster of eight up to 512 rows (fp32) or 768 (bf16, and batches); clusters of a block a CTA up to 1024 rows of the fp32
# cache, of two blocks beyond; from 2048 rows of capacity clusters of four with bf16
@pytest.mark.parametrize("rows,bf16", [(r, False) for r in (1, 31, 32, 33, 256, 257, 511, 512, 513, 1024, 1025, 2047, 2049)] + [(r, True) for r in (33, 768, 769, 1537, 2047)])
@pytest.mark.parametrize("capacity", ["rows", "more"])
def test_rows_around_the_cuts(cuda, rows, bf16, capacity):
    from insignia_b200 import ops

    rng = np.random.default_rng(rows)
    ctx, dt = rows if capacity == "rows" else 3000, torch.bfloat16 if bf16 else torch.float32
    q = torch.from_numpy(rng.standard_normal((16, 256)).astype(np.float32)).cuda()
    k, v = (torch.from_numpy(rng.standard_normal((ctx, 4, 256)).astype(np.float32)).cuda().to(dt) for _ in range(2))
    kd, vd = k[:rows].double(), v[:rows].double()
    s = torch.einsum("hgd,thd->hgt", q.double().view(4, 4, 256), kd) / 16
    want = host(torch.einsum("hgt,thd->hgd", torch.softmax(s, 2), vd).reshape(-1))
    # 32-bit sums; the tensor-core loop (bf16, 2048 rows and more) keeps 16 bits of the query and the weights
    bound = (1e-4 if bf16 and rows >= 2048 else 2e-6) * np.abs(want).max()
    if capacity == "rows":
        assert np.max(np.abs(host(ops.gqa_decode(q.view(-1), k, v, rows)) - want)) <= bound
    # the fused step: unit norms and position 0 of the rotation leave query and key as they are up to the norm
    pos = torch.full((1,), rows - 1, dtype=torch.int32, device="cuda")
    unit = torch.ones(256, device="cuda").to(torch.bfloat16).view(torch.int16)
    raw = torch.cat([q, torch.zeros_like(q)], 1).reshape(1, -1).contiguous()
    knew, vnew = (torch.from_numpy(rng.standard_normal((1, 1024)).astype(np.float32)).cuda() for _ in range(2))
    got = {}
    for n in (1, 2):  # one sequence, and two that share the device
        kc, vc = (t.reshape(1, -1).repeat(n, 1) for t in (k, v))
        scratch = torch.zeros(n * ops.gqa_scratch("cuda").numel(), dtype=torch.uint8, device="cuda")
        out = ops.attention_batch(raw.repeat(n, 1), knew.repeat(n, 1), vnew.repeat(n, 1), unit, unit, kc, vc, pos, ctx, scratch, n)
        got[n] = host(out).reshape(n, 4096)
        newk, newv = (t[0].view(ctx, 4, 256)[:rows].double() for t in (kc, vc))
    qd = q.double()
    qn = (qd * torch.rsqrt((qd * qd).mean(1, keepdim=True) + 1e-6)).float().double()
    if rows > 1:
        half = torch.arange(32, device="cuda", dtype=torch.float64)
        ang = (rows - 1) * 10000000.0 ** (-2 * half / 64)
        a, b = qn[:, :32].clone(), qn[:, 32:64].clone()
        qn[:, :32], qn[:, 32:64] = a * torch.cos(ang) - b * torch.sin(ang), b * torch.cos(ang) + a * torch.sin(ang)
    s = torch.einsum("hgd,thd->hgt", qn.view(4, 4, 256), newk) / 16
    want = host(torch.einsum("hgt,thd->hgd", torch.softmax(s, 2), newv).reshape(-1))
    # An fp32 angle of up to 2048 is off by up to 1.2e-4; a score of a query and a key of norm 16 moves by 16 * 16 * 1.2e-4 / 16 = 2e-3 at most, a weight
    # by as much of itself.
    for n in (1, 2):
        for i in range(n):
            assert np.max(np.abs(got[n][i] - want)) <= 3e-3 * np.abs(want).max(), n
    if ctx < 2048 and not bf16 and rows <= 512:  # the same cut: the same bits
        assert np.array_equal(got[1][0], got[2][0]) and np.array_equal(got[2][0], got[2][1])
