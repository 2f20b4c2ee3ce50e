"""Prompts in passes over the weights: buffers that fit the context, whatever it is, and what one long pass leaves for the next."""
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


# a pass of just over half the longest and the longest one less a token; the longest; a second pass of 1 and of 8 tokens (the GEMV's), of 9
# (the GEMM's fewest) and of 76; two full ones and a third of 12
@pytest.mark.parametrize("count", [513, 1023, 1024, 1025, 1032, 1033, 1100, 2060])
def test_prompts_of_more_than_a_pass(cuda, golden_ckpt, count):
    """Position, DeltaNet and convolution state, cached rows and the last hidden state after passes of up to 1024 tokens are the token loop's, and
    decoding goes on with the same tokens.  Both sum in fp32, in another order: the bound of shorter prompts."""
    rng = np.random.default_rng(count)
    prompt = [int(t) for t in rng.integers(0, 64, count)]
    with small_engine(golden_ckpt[1], max_context=count + 8) as a, small_engine(golden_ckpt[1], max_context=count + 8) as b:
        a.forward_tokens(prompt)
        for t in prompt:
            b.forward_token(t)
        assert a.position == b.position == count
        fa, fb = fields(a, count), fields(b, count)
        for f in fa:
            assert np.max(np.abs(fa[f] - fb[f])) <= 2e-4 * np.abs(fb[f]).max(), f
        ta, tb = a.logits_argmax(), b.logits_argmax()
        for _ in range(6):
            assert ta == tb
            ta, tb = a.decode_token(ta), b.decode_token(tb)
        # the same prompt in two calls, cut elsewhere
        a.reset()
        a.forward_tokens(prompt[:300])
        a.forward_tokens(prompt[300:])
        fa = fields(a, count)
        for f in fa:
            assert np.max(np.abs(fa[f] - fb[f])) <= 2e-4 * np.abs(fb[f]).max(), f


@pytest.fixture(scope="module")
def mtp_ckpt(tmp_path_factory):
    from insignia_b200 import synth

    d = tmp_path_factory.mktemp("mtp")
    synth.write_checkpoint(synth.SynthConfig(layers=(0, 1, 2, 3), vocab_rows=64, mtp=True, seed=9, norms="random"), str(d / "m.safetensors"), str(d / "m.idx"))
    return str(d / "m.idx")


@pytest.mark.parametrize("count", [1024, 1034])
def test_a_long_pass_leaves_the_rows_of_the_mtp_head(cuda, mtp_ckpt, count):
    """Every position's row but the last one's, also across two passes, as single steps and drafts leave them."""
    prompt = [int(t) for t in np.random.default_rng(count).integers(0, 64, count)]
    with small_engine(mtp_ckpt, max_context=count + 8) as a, small_engine(mtp_ckpt, max_context=count + 8) as b:
        first = a.prime_speculative(prompt)
        for i, t in enumerate(prompt):
            b.forward_token(t)
            h = b.read("hidden")
            if i + 1 < count:
                b.mtp_draft(prompt[i + 1])
        for f in ("mtp_keys", "mtp_values"):
            got, want = a.read(f, (count - 1) * 1024), b.read(f, (count - 1) * 1024)
            assert np.max(np.abs(got - want)) <= 1e-3 * np.abs(want).max(), f  # the bound of a short prompt's rows
        assert np.max(np.abs(a.read("hidden") - h)) <= 1e-3 * np.abs(h).max()
        a.reset()
        a.forward_tokens(prompt)
        assert first == a.logits_argmax()
