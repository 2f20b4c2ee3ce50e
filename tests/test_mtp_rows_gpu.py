"""The MTP block's input, its bf16 projection and its cache rows for several tokens at once, against the forms for one."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), ".."))
from tests.test_full_model_gpu import full_ckpt  # noqa: E402,F401
from tests.test_kernels_gpu import bf16, dev, host  # noqa: E402

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# row counts around a warp's two or four rows, columns around a step's vectors and the part of x in shared memory, tokens around eight
@pytest.mark.parametrize("rows,cols,tokens", [(4096, 8192, 8), (37, 8, 1), (37, 264, 2), (16, 2048, 7), (33, 2056, 9), (64, 520, 17), (16, 8712, 1), (16, 8712, 3)])
def test_bf16_projection_of_several_tokens(cuda, rows, cols, tokens):
    from insignia_b200 import ops

    rng = np.random.default_rng(rows + cols)
    w = (bf16(rng, rows * cols).reshape(rows, cols))
    x = rng.standard_normal((tokens, cols)).astype(np.float32)
    got = host(ops.bf16_gemv_tokens(dev(w), dev(x)))
    wf = (w.astype(np.uint32) << 16).view(np.float32).astype(np.float64)
    # fp32 sums of cols products in another order: cols / 32 steps of a lane and five of the warp, 2^-24 of the magnitudes each
    bound = (cols / 32 + 6) * 2.0 ** -24 * (np.abs(x).astype(np.float64) @ np.abs(wf).T)
    assert np.all(np.abs(got - x.astype(np.float64) @ wf.T) <= bound)
    one = np.stack([host(ops.bf16_gemv(dev(w), dev(x[m]))) for m in range(tokens)])
    assert np.array_equal(got, one)


@pytest.mark.parametrize("tokens", [1, 5])
def test_mtp_input_equals_its_parts(cuda, tokens):
    from insignia_b200 import ops, synth

    rng = np.random.default_rng(tokens)
    w, s = synth.quantize_rows_torch(torch.randn((64, 4096), device="cuda"))
    ids = torch.tensor([3, 63, 0, 64, -1][:tokens], dtype=torch.int32, device="cuda")  # the last two are outside the table
    hidden = dev(rng.standard_normal((tokens, 4096)).astype(np.float32))
    ne, nh = dev(bf16(rng, 4096)), dev(bf16(rng, 4096))
    got = host(ops.mtp_input(w, s, ids, hidden, ne, nh)).reshape(tokens, 2, 4096)
    emb = torch.stack([ops.get_row_mlx(w, s, int(i)) if 0 <= int(i) < 64 else torch.zeros(4096, device="cuda") for i in ids.tolist()])
    assert np.array_equal(got[:, 0], host(ops.rmsnorm_bf16(emb, ne)).reshape(tokens, 4096))
    assert np.array_equal(got[:, 1], host(ops.rmsnorm_bf16(hidden, nh)).reshape(tokens, 4096))


@pytest.mark.parametrize("count", [2, 9, 21])
def test_prompt_in_passes_leaves_the_rows_of_single_steps(cuda, full_ckpt, count):
    """prime_speculative against forward_token and mtp_draft token by token: MTP cache rows, hidden state, next token."""
    from insignia_b200.engine import Engine

    def view(e, field):
        class A:
            __cuda_array_interface__ = {"data": (e.buffer(field), False), "shape": (64 * 1024,), "typestr": "<f4", "strides": None, "version": 3}
        return torch.as_tensor(A(), device="cuda").view(64, 1024)

    prompt = [int(t) for t in np.random.default_rng(count).integers(0, 248320, count)]
    with Engine(full_ckpt[1], max_context=64) as e:
        for i, t in enumerate(prompt):
            e.forward_token(t)
            h = e.read("hidden")
            if i + 1 < count:
                e.mtp_draft(prompt[i + 1])
        e.reset()
        want_k, want_v = host(view(e, "mtp_keys")).copy(), host(view(e, "mtp_values")).copy()
        view(e, "mtp_keys").zero_()
        view(e, "mtp_values").zero_()
        first = e.prime_speculative(prompt)
        got_k, got_v, got_h = host(view(e, "mtp_keys")), host(view(e, "mtp_values")), e.read("hidden")
        assert np.all(got_k[count - 1:] == 0) and np.all(got_v[count - 1:] == 0)
        # several tokens' products sum in another order: the bound of a prompt pass against single steps
        for got, want in ((got_k[: count - 1], want_k[: count - 1]), (got_v[: count - 1], want_v[: count - 1]), (got_h, h)):
            assert np.max(np.abs(got - want)) <= 1e-3 * np.abs(want).max()
        e.reset()
        e.forward_tokens(prompt)
        assert first == e.logits_argmax()
