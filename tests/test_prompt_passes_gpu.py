"""Prompts in passes over the weights: buffers that fit the context, whatever it is."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), ".."))
from tests.test_model_gpu import small_engine  # noqa: E402

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

STATE, CONV = 3 * 32 * 128 * 128, 3 * 8192 * 3


def fields(engine, count):
    return {f: engine.read(f, n) for f, n in (("hidden", 4096), ("delta_state", STATE), ("conv_state", CONV), ("kv_keys", count * 1024), ("kv_values", count * 1024))}


def test_an_engine_pays_for_passes_it_can_take(cuda, golden_ckpt):
    """No pass is longer than the context: 64 rows of it need 64 tokens' activations and digits (47 thousand floats and 46 KB a token at 12288
    columns), not those of the longest pass."""
    def taken(ctx):
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        with small_engine(golden_ckpt[1], max_context=ctx):
            return before - torch.cuda.mem_get_info()[0]

    taken(64)  # the library's own memory is there from the first engine on
    rows = 2 * 9 * 4096  # keys and values of a token, the MTP head's among them
    assert taken(1024) - taken(64) >= 960 * (rows + 190_000)


@pytest.mark.parametrize("ctx", [9, 16, 33, 77])
def test_a_prompt_fills_a_small_context(cuda, golden_ckpt, ctx):
    rng = np.random.default_rng(ctx)
    prompt = [int(t) for t in rng.integers(0, 64, ctx)]
    with small_engine(golden_ckpt[1], max_context=ctx) as a, small_engine(golden_ckpt[1], max_context=ctx) as b:
        a.forward_tokens(prompt)
        for t in prompt:
            b.forward_token(t)
        fa, fb = fields(a, ctx), fields(b, ctx)
        for f in fa:
            assert np.max(np.abs(fa[f] - fb[f])) <= 2e-4 * np.abs(fb[f]).max(), f
        assert a.logits_argmax() == b.logits_argmax()
