"""The work this engine does for its users, as cases that can be timed.

Engine cases run the full 32-layer model (synthetic MXFP4 weights of the architecture's shapes) the way a serving program
drives it: the engine, its weights and the batches are opened once per process and kept, every request starts from
``reset()``.  Operator cases call the kernel-level entry points of :mod:`insignia_b200.ops` on the shapes the layers have.
Inputs (prompts, activations, operator weights, caches, states) come from the case's seed.
"""
import os
import shutil
import tempfile

import numpy as np
import torch

from insignia_b200 import ops, synth
from insignia_b200.engine import Batch, Engine

HIDDEN, INTER, VOCAB, LAYERS = synth.HIDDEN, synth.INTER, synth.VOCAB, synth.LAYERS
ATTN_LAYERS, DELTA_LAYERS = 8, 24
STATE, CONV, KV_ROW = 32 * 128 * 128, 8192 * 3, 1024  # floats per layer; values per cached key (or value) row
CONTEXT = 2560                                        # rows of the engines' caches: the longest request below fits
BATCH_CONTEXT = 512

MLP_PARAMS = 3 * HIDDEN * INTER
DELTA_PARAMS = (8192 + 4096 + 64) * HIDDEN + 4096 * HIDDEN + MLP_PARAMS
ATTN_PARAMS = (8192 + 2048) * HIDDEN + 4096 * HIDDEN + MLP_PARAMS
BLOCK_PARAMS = DELTA_LAYERS * DELTA_PARAMS + ATTN_LAYERS * ATTN_PARAMS
HEAD_PARAMS = VOCAB * HIDDEN
MTP_PARAMS = ATTN_PARAMS + HEAD_PARAMS
MTP_FC_BYTES = 2 * HIDDEN * HIDDEN * 2
ROW_OF = {"o_proj": (4096, 4096), "down": (4096, 12288), "in_proj": (12352, 4096), "gate_up": (24576, 4096), "lm_head": (VOCAB, 4096)}


def listed():
    return [
        # smallest call: one token through one square projection (the output projection of a block); latency decides
        {"name": "matvec o_proj", "kind": "matvec", "matrix": "o_proj", "tokens": 1},
        # a ragged fused in-projection (qkv|z|a|b rows) for three tokens: a short draft being scored
        {"name": "matvec in_proj x3", "kind": "matvec", "matrix": "in_proj", "tokens": 3},
        # a few dozen tokens against the widest layer matrix, an odd count: the tail of a prompt, or a verify batch
        {"name": "matmul gate_up x61", "kind": "matmul", "matrix": "gate_up", "tokens": 61},
        # one query token against a long context in the bf16 cache
        {"name": "attention 32768 bf16", "kind": "attention", "context": 32768, "bf16": True, "sequences": 1},
        # eight sequences, ragged mid-size context, fp32 cache (the default): one fused step of a serving batch
        {"name": "attention 8 x 5000 f32", "kind": "attention", "context": 5000, "bf16": False, "sequences": 8},
        # the recurrent layer over a 64-token sequence
        {"name": "deltanet 64 steps", "kind": "deltanet", "tokens": 64},
        # interactive use: a short question, the answer fetched token by token through decode_token
        {"name": "chat 23 + 24", "kind": "step", "prompt": 23, "generated": 24, "bf16": False},
        # the standard request: a 512-token prompt and a greedy continuation fed back on the device
        {"name": "request 512 + 64", "kind": "request", "prompt": 512, "generated": 64, "bf16": False},
        # prompt processing alone: a long document, bf16 cache
        {"name": "prompt 2048 bf16", "kind": "request", "prompt": 2048, "generated": 0, "bf16": True},
        # serving batches on one weight copy: a full one and a small odd one, prompt tokens in lock step, then generation
        {"name": "batch 8", "kind": "batch", "sequences": 8, "prompt": 8, "generated": 32, "bf16": False},
        {"name": "batch 3", "kind": "batch", "sequences": 3, "prompt": 8, "generated": 32, "bf16": False},
        # speculative greedy decode: MTP drafts, two-token verify passes
        {"name": "speculative 16 + 24", "kind": "speculative", "prompt": 16, "generated": 24, "bf16": False},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["matvec", "matmul", "attention", "deltanet", "step", "request", "request", "batch", "batch", "speculative"])
    bf16 = rng.random() < 0.4
    if kind == "matvec":
        return {"kind": kind, "matrix": rng.choice(sorted(ROW_OF)), "tokens": rng.choice([1, 1, 2, 3, 4])}
    if kind == "matmul":
        return {"kind": kind, "matrix": rng.choice(["o_proj", "down", "in_proj", "gate_up"]), "tokens": _log(rng, 5, 256)}
    if kind == "attention":
        sequences = rng.choice([1, 1, 2, 3, 5, 8])
        return {"kind": kind, "context": _log(rng, 64, 32768 if sequences < 3 else 8192), "bf16": bf16, "sequences": sequences}
    if kind == "deltanet":
        return {"kind": kind, "tokens": _log(rng, 1, 256)}
    if kind == "step":
        return {"kind": kind, "prompt": _log(rng, 2, 400), "generated": _log(rng, 2, 40), "bf16": bf16}
    if kind == "request":
        prompt = _log(rng, 4, 2000)
        return {"kind": kind, "prompt": prompt, "generated": rng.randint(0, 64) if prompt < 700 else rng.randint(0, 8), "bf16": bf16}
    if kind == "batch":
        return {"kind": kind, "sequences": rng.randint(1, 8), "prompt": rng.randint(1, 12), "generated": rng.randint(4, 32), "bf16": bf16}
    return {"kind": kind, "prompt": rng.randint(2, 24), "generated": rng.randint(4, 32), "bf16": bf16}


# ---- what a process keeps: the checkpoint file, one engine per cache type, batches -----------------------------------------
_engines, _batches = {}, {}


def _checkpoint():
    for base in ("/dev/shm", tempfile.gettempdir()):
        d = os.path.join(base, "insignia_b200_model_%d" % os.getuid())
        idx = os.path.join(d, "model.idx")
        if os.path.exists(idx):
            return idx
        try:
            if shutil.disk_usage(base).free < 8 << 30:
                continue
            os.makedirs(d, mode=0o700, exist_ok=True)
        except OSError:
            continue
        own = os.path.join(d, "%d" % os.getpid())
        synth.write_checkpoint(synth.SynthConfig(seed=0, norms="random", backend="torch"), own + ".safetensors")
        os.replace(own + ".safetensors", os.path.join(d, "model.safetensors"))
        synth.write_index(os.path.join(d, "model.safetensors"), own + ".idx")
        os.replace(own + ".idx", idx)
        torch.cuda.empty_cache()
        return idx
    raise RuntimeError("no scratch directory with 8 GiB free")


def _engine(bf16):
    if bf16 not in _engines:
        _engines[bf16] = Engine(_checkpoint(), max_context=CONTEXT, kv_bf16=bf16)
    return _engines[bf16]


def _batch(sequences, bf16):
    if (sequences, bf16) not in _batches:
        _batches[sequences, bf16] = Batch(_engine(bf16), sequences, BATCH_CONTEXT)
    return _batches[sequences, bf16]


class _DeviceArray:
    def __init__(self, address, count, typestr):
        self.__cuda_array_interface__ = {"data": (address, False), "shape": (count,), "typestr": typestr, "strides": None, "version": 3}


def _buffer(engine, field, count, bf16=False):
    t = torch.as_tensor(_DeviceArray(engine.buffer(field), count, "<i2" if bf16 else "<f4"), device="cuda")
    return t.view(torch.bfloat16) if bf16 else t


def _prompt(rng, n):
    return [int(t) for t in rng.integers(0, VOCAB, n)]


def _weights(matrix, gen):
    """A seeded N(0, 0.02) matrix in the checkpoint's layout, quantised a slice of rows at a time."""
    rows, cols = ROW_OF[matrix]
    w = torch.empty((rows, cols // 8), dtype=torch.int32, device="cuda")
    s = torch.empty((rows, cols // 32), dtype=torch.uint8, device="cuda")
    for r0 in range(0, rows, 8192):
        r1 = min(rows, r0 + 8192)
        w[r0:r1], s[r0:r1] = synth.quantize_rows_torch(torch.randn((r1 - r0, cols), generator=gen, device="cuda") * 0.02)
    return w, s


def prepare(case, seed):
    kind = case["kind"]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    rng = np.random.default_rng(seed)

    def randn(*shape):
        return torch.randn(shape, generator=gen, device="cuda")

    st = {"kind": kind}
    if kind in ("matvec", "matmul"):
        w, s = _weights(case["matrix"], gen)
        st["x"] = randn(case["tokens"], w.shape[1] * 8)
        if kind == "matvec":
            st["packed"] = ops.repack(w, s)
        else:
            st["packed"] = ops.repack_umma(w, s)
            st["scratch"] = ops.umma_gemm_scratch(w.shape[1] * 8, case["tokens"])
    elif kind == "attention":
        n, ctx = case["sequences"], case["context"]
        dt = torch.bfloat16 if case["bf16"] else torch.float32
        st.update(n=n, ctx=ctx, k=randn(n, ctx * KV_ROW).to(dt), v=randn(n, ctx * KV_ROW).to(dt))
        if n == 1:
            st.update(q=randn(4096), k=st["k"][0], v=st["v"][0], scratch=ops.gqa_scratch("cuda", ctx))
        else:
            st.update(qraw=randn(n, 8192), kraw=randn(n, KV_ROW), vraw=randn(n, KV_ROW),
                      norm=(1 + 0.1 * randn(256)).to(torch.bfloat16).view(torch.int16),
                      position=torch.full((1,), ctx - 1, dtype=torch.int32, device="cuda"))
            st["scratch"] = torch.zeros(n * ops.gqa_scratch("cuda", ctx).numel(), dtype=torch.uint8, device="cuda")
    elif kind == "deltanet":
        n = case["tokens"]
        st.update(n=n, state=0.1 * randn(STATE), qkv=randn(n, 8192), g=-torch.nn.functional.softplus(randn(n, 32)),
                  beta=torch.sigmoid(randn(n, 32)))
        flat = st["qkv"].view(-1)
        st.update(q=flat, k=flat[2048:], v=flat[4096:])
    elif kind == "batch":
        b = _batch(case["sequences"], case["bf16"])
        st.update(batch=b, prompts=rng.integers(0, VOCAB, (case["prompt"], case["sequences"])), generated=case["generated"])
    else:
        e = _engine(case["bf16"])
        rows = case["prompt"] + case["generated"]
        caches = [_buffer(e, f, ATTN_LAYERS * CONTEXT * KV_ROW, case["bf16"]).view(ATTN_LAYERS, CONTEXT, KV_ROW)[:, :rows] for f in ("kv_keys", "kv_values")]
        st.update(engine=e, prompt=_prompt(rng, case["prompt"]), generated=case["generated"],
                  buffers={"hidden": _buffer(e, "hidden", HIDDEN), "delta_state": _buffer(e, "delta_state", DELTA_LAYERS * STATE),
                           "conv_state": _buffer(e, "conv_state", DELTA_LAYERS * CONV), "keys": caches[0], "values": caches[1]})
        if kind != "speculative":  # that mode leaves no row of logits: its results are tokens and state
            st["buffers"]["logits"] = _buffer(e, "logits", VOCAB)
    return st


def run(st):
    kind = st["kind"]
    if kind == "matvec":
        return ops.gemv_packed(st["packed"], st["x"])
    if kind == "matmul":
        return ops.gemm_umma(st["packed"], st["x"], scratch=st["scratch"])
    if kind == "attention":
        if st["n"] == 1:
            return ops.gqa_decode(st["q"], st["k"], st["v"], st["ctx"], scratch=st["scratch"])
        out = ops.attention_batch(st["qraw"], st["kraw"], st["vraw"], st["norm"], st["norm"], st["k"], st["v"], st["position"], st["ctx"],
                                  st["scratch"], st["n"])
        row = slice((st["ctx"] - 1) * KV_ROW, st["ctx"] * KV_ROW)
        return {"out": out, "key_row": st["k"][:, row], "value_row": st["v"][:, row]}
    if kind == "deltanet":
        return {"out": ops.deltanet_decode_tokens(st["state"], st["q"], st["k"], st["v"], st["g"], st["beta"], st["n"], 8192), "state": st["state"]}
    if kind == "batch":
        b = st["batch"]
        b.reset()
        for row in st["prompts"][:-1]:
            b.forward_tokens(row)
        first = b.decode_tokens(st["prompts"][-1])
        tokens = b.generate(first, st["generated"])
        return {"first": np.array(first), "tokens": tokens, "hidden": [b.read("hidden", s) for s in range(b.n)]}
    e = st["engine"]
    e.reset()
    out = dict(st["buffers"])
    if kind == "speculative":
        first = e.prime_speculative(st["prompt"])
        tokens, out["accepted"] = e.generate_speculative(first, st["generated"])
    else:
        e.forward_tokens(st["prompt"])
        first = e.logits_argmax()
        if kind == "request":
            tokens = e.generate(first, st["generated"])
        else:
            tokens, token = [], first
            for _ in range(st["generated"]):
                token = e.decode_token(token)
                tokens.append(token)
    out["tokens"] = np.array([first] + tokens)
    return out


def work(case):
    kind = case["kind"]
    if kind in ("matvec", "matmul"):
        (rows, cols), t = ROW_OF[case["matrix"]], case["tokens"]
        return {"bytes": rows * cols * 17 / 32 + 4 * t * (rows + cols), "flops": 2 * rows * cols * t}
    if kind == "attention":
        n, ctx, size = case["sequences"], case["context"], 2 if case["bf16"] else 4
        return {"bytes": n * (2 * ctx * KV_ROW * size + 2 * 4096 * 4), "flops": n * 4 * 4096 * ctx}
    if kind == "deltanet":
        return {"bytes": 2 * 4 * STATE + case["tokens"] * 4 * (8192 + 64 + 4096), "flops": case["tokens"] * STATE * 7}
    size = 2 if case["bf16"] else 4
    state = 2 * 4 * DELTA_LAYERS * (STATE + CONV)
    row = 2 * KV_ROW * size * ATTN_LAYERS
    p, g, n = case["prompt"], case["generated"], case.get("sequences", 1)
    if kind == "batch":  # prompt tokens and generated ones are the same step
        steps = p + g
        return {"bytes": steps * ((BLOCK_PARAMS + HEAD_PARAMS) * 17 / 32 + n * state) + n * row * steps * steps / 2,
                "flops": 2 * n * steps * (BLOCK_PARAMS + HEAD_PARAMS)}
    if kind == "speculative":  # one main step and one draft per token (random weights: the drafts do not hold)
        steps = p + g
        return {"bytes": steps * ((BLOCK_PARAMS + HEAD_PARAMS + ATTN_PARAMS) * 17 / 32 + MTP_FC_BYTES + state) + g * HEAD_PARAMS * 17 / 32
                + row * steps * steps / 2, "flops": 2 * steps * (BLOCK_PARAMS + HEAD_PARAMS + ATTN_PARAMS) + 2 * g * (BLOCK_PARAMS + 2 * HEAD_PARAMS)}
    prompt = BLOCK_PARAMS * 17 / 32 + HEAD_PARAMS * 17 / 32 + state + row * p
    token = (BLOCK_PARAMS + HEAD_PARAMS) * 17 / 32 + state
    return {"bytes": prompt + g * token + row * g * (p + g / 2),
            "flops": 2 * (BLOCK_PARAMS * (p + g) + HEAD_PARAMS * (1 + g)) + 4 * 4096 * ATTN_LAYERS * (p * p / 2 + g * (p + g / 2))}


def tolerance(case):
    kind = case["kind"]
    if kind in ("matvec", "matmul"):
        return {"rel": 1e-5}  # 32-bit sums of up to 12288 terms
    if kind == "attention":
        return {"rel": 1e-3 if case["bf16"] else 1e-5}
    if kind == "deltanet":
        return {"rel": 5e-5}  # a 32-bit recurrence over the tokens
    return {"rel": 2e-3 if case["bf16"] else 1e-4}  # 32 layers of 32-bit arithmetic; rows rounded to the cache's type; ids equal
