"""Full-size model (32 layers, vocab 248320, 699 tensors) against the compiled reference engine.

The checkpoint is synthetic (seeded N(0, 0.02) -> MXFP4, generated on the GPU and written to a
RAM-backed file); both engines read the same file.  Bars: greedy token ids identical; per-layer
hidden states cosine >= 0.9999 and max-abs-rel <= 2e-2 (measured: a few 1e-6).
"""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), ".."))
from oracle import ref_engine  # noqa: E402

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not ref_engine.available(), reason="compiled reference (oracle/_ref) not built")]

SEED = 0


@pytest.fixture(scope="module")
def full_ckpt(cuda):
    import bench

    return bench.ensure_checkpoint(SEED, True)


def cos(a, b):
    return float(a @ b / np.linalg.norm(a) / np.linalg.norm(b))


def test_model_file_inventory(full_ckpt):
    from insignia_b200.checkpoint_io import load_index

    info = load_index(full_ckpt[1])
    assert len(info["tensors"]) == 699  # src/test_model.cpp:4
    names = {t["name"]: t for t in info["tensors"]}
    q = names["language_model.model.layers.3.self_attn.q_proj.weight"]
    assert q["shape"] == (8192, 512) and q["dtype"] == 5  # src/test_qwen35.cu:5: 8192 x 4096


def test_first_token_layer_seams_vs_reference(cuda, full_ckpt):
    """src/dump_layers.cu:5: embed token 42, run the 32 layers one by one, compare every seam."""
    from insignia_b200.engine import Engine

    ref = ref_engine.RefEngine(full_ckpt[1], max_context=16)
    try:
        with Engine(full_ckpt[1], max_context=16, use_graph=False) as e:
            ref.embed(42), e.embed(42)
            assert np.array_equal(ref.read("hidden", 4096), e.read("hidden"))  # dequantised row: bit-exact
            worst = 0.0
            for l in range(32):
                ref.layer(l), e.layer(l)
                a, b = e.read("hidden"), ref.read("hidden", 4096)
                assert cos(a, b) >= 0.9999, l
                rel = float(np.max(np.abs(a - b)) / np.abs(b).max())
                assert rel <= 2e-2, l
                worst = max(worst, rel)
            assert worst <= 1e-4, worst
    finally:
        ref.close()


def test_greedy_tokens_identical_to_reference(cuda, full_ckpt):
    """Prompt ingested token by token (src/generate_ids.cu:4), then greedy decode: ids must be identical."""
    from insignia_b200.engine import Engine

    n_prompt, n_gen = 96, 160
    rng = np.random.default_rng(20240601)
    prompt = rng.integers(0, 248320, n_prompt)
    ref = ref_engine.RefEngine(full_ckpt[1], max_context=n_prompt + n_gen + 4)
    try:
        with Engine(full_ckpt[1], max_context=n_prompt + n_gen + 4) as e:
            for t in prompt:
                ref.forward_token(int(t)), e.forward_token(int(t))
            tr, te = ref.logits_argmax(), e.logits_argmax()
            assert tr == te
            lr, le = ref.read("logits", 248320), e.read("logits")
            assert cos(lr, le) >= 0.9999 and np.max(np.abs(lr - le)) <= 2e-2 * np.abs(lr).max()
            want, t = [], tr
            min_gap = 1e9
            for _ in range(n_gen):
                t = ref.decode_token(t)
                want.append(t)
                top2 = np.partition(ref.read("logits", 248320), -2)[-2:]
                min_gap = min(min_gap, float(top2[1] - top2[0]))
            got = e.generate(te, n_gen)
            assert got == want, (min_gap, [i for i, (a, b) in enumerate(zip(got, want)) if a != b][:3])
            assert e.position == ref.position == n_prompt + n_gen
            assert cos(e.read("hidden"), ref.read("hidden", 4096)) >= 0.9999
            print(f"smallest top-2 logit gap of the reference over {n_gen} steps: {min_gap:.3e}")
    finally:
        ref.close()


@pytest.fixture(scope="module")
def cfg3_reference(cuda, full_ckpt):
    """BASELINE configs[3] on the reference engine: a 512-token seeded uniform-random prompt fed token by token
    (src/generate_ids.cu:4), then 256 greedy tokens; also the smallest gap between its two largest logits on the way."""
    n_prompt, n_gen = 512, 256
    prompt = [int(t) for t in np.random.default_rng(3).integers(0, 248320, n_prompt)]
    ref = ref_engine.RefEngine(full_ckpt[1], max_context=n_prompt + n_gen + 4)
    try:
        for t in prompt:
            ref.forward_token(t)
        first = ref.logits_argmax()
        want, t, min_gap = [], first, 1e9
        for _ in range(n_gen):
            t = ref.decode_token(t)
            want.append(t)
            top2 = np.partition(ref.read("logits", 248320), -2)[-2:]
            min_gap = min(min_gap, float(top2[1] - top2[0]))
        hidden = ref.read("hidden", 4096)
    finally:
        ref.close()
    print(f"configs[3]: smallest top-2 logit gap of the reference over {n_gen} steps: {min_gap:.3e}")
    return prompt, first, want, min_gap, hidden


@pytest.mark.parametrize("persistent", [False, True])
def test_cfg3_512_prompt_256_generated_identical_to_reference(cuda, full_ckpt, cfg3_reference, persistent):
    """The north-star identity check at its full length: 512 + 256 tokens, every generated id equal to the reference's,
    through the graph of launches and through the persistent token kernel."""
    from insignia_b200.engine import Engine

    prompt, first, want, min_gap, ref_hidden = cfg3_reference
    with Engine(full_ckpt[1], max_context=len(prompt) + len(want) + 4, persistent=persistent) as e:
        for t in prompt:
            e.forward_token(t)
        assert e.logits_argmax() == first
        got = e.generate(first, len(want))
        assert got == want, (min_gap, [i for i, (a, b) in enumerate(zip(got, want)) if a != b][:3])
        assert e.position == len(prompt) + len(want)
        h = e.read("hidden")
        assert cos(h, ref_hidden) >= 0.9999 and np.max(np.abs(h - ref_hidden)) <= 2e-2 * np.abs(ref_hidden).max()


@pytest.mark.parametrize("drafts", ["mtp", "forced"])
def test_speculative_decode_identical_to_reference(cuda, full_ckpt, cfg3_reference, drafts):
    """Draft-1 / verify greedy decode against the reference's plain greedy ids over 512 + 256 tokens.  "mtp": the drafts
    come from the MTP head (on random weights nearly all are wrong: the roll-back path).  "forced": the caller supplies
    drafts, right ones and wrong ones in runs of three, so that accepted and rejected passes alternate."""
    from insignia_b200.engine import Engine

    prompt, first, want, min_gap, ref_hidden = cfg3_reference
    n = len(want)
    forced = None
    if drafts == "forced":
        forced = [want[i] if (i // 3) % 2 == 0 else (want[i] + 1) % 248320 for i in range(n)]
    with Engine(full_ckpt[1], max_context=len(prompt) + n + 8) as e:
        assert e.prime_speculative(prompt) == first
        got, accepted = e.generate_speculative(first, n - 5, forced_drafts=forced)
        assert got == want[: n - 5], (min_gap, [i for i, (a, b) in enumerate(zip(got, want)) if a != b][:3])
        assert e.position == len(prompt) + n - 5
        if forced is not None:
            assert 0.25 * n < accepted < 0.5 * n, accepted
        # plain greedy decode carries on from the speculative state
        assert e.generate(got[-1], 5) == want[n - 5:]
        h = e.read("hidden")
        assert cos(h, ref_hidden) >= 0.9999 and np.max(np.abs(h - ref_hidden)) <= 2e-2 * np.abs(ref_hidden).max()
        print(f"speculative ({drafts}): {accepted} drafts accepted over {n - 5} tokens")


def test_prompt_in_passes_of_four_then_greedy_tokens_identical_to_reference(cuda, full_ckpt):
    """The prompt through forward_tokens, then greedy decode: same ids as the reference fed token by token."""
    from insignia_b200.engine import Engine

    n_prompt, n_gen = 61, 48  # all 61 in one pass through the tcgen05 kernel
    rng = np.random.default_rng(77)
    prompt = [int(t) for t in rng.integers(0, 248320, n_prompt)]
    ref = ref_engine.RefEngine(full_ckpt[1], max_context=n_prompt + n_gen + 4)
    try:
        with Engine(full_ckpt[1], max_context=n_prompt + n_gen + 4) as e:
            for t in prompt:
                ref.forward_token(t)
            e.forward_tokens(prompt)
            tr, te = ref.logits_argmax(), e.logits_argmax()
            assert tr == te
            assert cos(e.read("hidden"), ref.read("hidden", 4096)) >= 0.9999
            want, t = [], tr
            for _ in range(n_gen):
                t = ref.decode_token(t)
                want.append(t)
            assert e.generate(te, n_gen) == want
            assert e.position == ref.position == n_prompt + n_gen
    finally:
        ref.close()


@pytest.mark.parametrize("sequences", [2, 8])
def test_batch_on_the_full_model_identical_to_reference(cuda, full_ckpt, sequences):
    """configs[4] on the full model: sequences decoded in lock step on one weight copy (2: mma.sync kernel, 8: tcgen05 kernel),
    each from its own prompt; every sequence's greedy ids equal the reference engine's for that prompt."""
    from insignia_b200.engine import Batch, Engine

    n_prompt, n_gen = 24, 40
    rng = np.random.default_rng(5)
    prompts = rng.integers(0, 248320, (sequences, n_prompt))
    want = []
    for s in range(min(sequences, 3)):  # the reference decodes at 54 tok/s: three sequences are checked against it
        ref = ref_engine.RefEngine(full_ckpt[1], max_context=n_prompt + n_gen + 4)  # a fresh engine: fresh recurrent state
        try:
            for t in prompts[s]:
                ref.forward_token(int(t))
            t = ref.logits_argmax()
            toks = [t]
            for _ in range(n_gen):
                t = ref.decode_token(t)
                toks.append(t)
            want.append(toks)
        finally:
            ref.close()
    with Engine(full_ckpt[1], max_context=8) as e, Batch(e, sequences, n_prompt + n_gen + 4) as b:
        for i in range(n_prompt - 1):
            b.forward_tokens(prompts[:, i])
        first = b.decode_tokens(prompts[:, -1])
        got = b.generate(first, n_gen)
        for s in range(len(want)):
            assert [first[s]] + list(got[:, s]) == want[s], s


def test_mtp_draft_matches_reference(cuda, full_ckpt):
    """src/test_mtp.cu:3: forward a token, take the arg-max, draft twice."""
    from insignia_b200.engine import Engine

    ref = ref_engine.RefEngine(full_ckpt[1], max_context=32)
    try:
        with Engine(full_ckpt[1], max_context=32) as e:
            for t in (248045, 17, 99999):
                ref.forward_token(t), e.forward_token(t)
            tr, te = ref.logits_argmax(), e.logits_argmax()
            assert tr == te
            for _ in range(2):
                dr, de = ref.mtp_draft(tr), e.mtp_draft(te)
                assert dr == de
                a, b = e.read("hidden"), ref.read("hidden", 4096)
                assert cos(a, b) >= 0.9999 and np.max(np.abs(a - b)) <= 2e-2 * np.abs(b).max()
            assert e.position == ref.position == 3
    finally:
        ref.close()


def test_kv_bf16_and_elementwise_gate_run_full_model(cuda, full_ckpt):
    """The additive modes (bf16 KV cache, element-wise output gate, accurate RoPE) on the full model: finite,
    and the bf16 cache stays within the layer bar of the fp32 cache over a short decode."""
    from insignia_b200.engine import Engine

    with Engine(full_ckpt[1], max_context=64, kv_bf16=True, accurate_trig=True) as a, \
            Engine(full_ckpt[1], max_context=64, accurate_trig=True) as b, \
            Engine(full_ckpt[1], max_context=64, gate_elementwise=True) as c:
        for t in (5, 4242, 100000, 7, 248319, 0, 31337, 2):
            a.forward_token(t), b.forward_token(t), c.forward_token(t)
        ha, hb, hc = a.read("hidden"), b.read("hidden"), c.read("hidden")
        assert np.all(np.isfinite(ha)) and np.all(np.isfinite(hc))
        assert cos(ha, hb) >= 0.9999 and np.max(np.abs(ha - hb)) <= 2e-2 * np.abs(hb).max()
        assert not np.array_equal(hb, hc)
