#!/usr/bin/env python3
"""Decode benchmark: batch-1 greedy tok/s of the 32-layer MXFP4 hybrid on N GPUs of one node.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl reference] [--config 3|4]

Workload (the default): the full 32-layer model (24 gated-DeltaNet + 8 gated-GQA layers,
hidden 4096, FFN 12288, vocab 248320), every linear weight MXFP4 quantised from seeded N(0, 0.02); a 512-token prompt of
seeded uniform-random ids, then greedy decode.  A "step" is one decoded token = one pass of the hot path.  Weights are
synthetic (the real checkpoint is not available offline) and are written to a RAM-backed file once, then loaded through
the same ModelFile -> TieredStorage path a real checkpoint takes.

* ``value``  tok/s with everything resident in HBM: blocks of K tokens generated back to back with the arg-max fed back
  on the device (Qwen35Decode::generate), CUDA events on the engine's stream.  The block is repeated (each time from
  the same context length) until about two seconds have been timed; the median block counts.
* ``e2e``    tok/s through the reference-facing call Qwen35Decode::decode_token(int) -> int: the token id goes
  host -> device and the result device -> host every step; same repetition rule.
* ``roofline``  the fused GEMV kernel: algorithmic weight bytes of its 152 launches per token / the time of those
  launches replayed alone (CUDA events), against the measured HBM copy bandwidth of MEASURED_PEAKS.json.
* ``cpu_baseline``  the CPU oracle port (oracle/, C + OpenMP) decoding a few tokens of the same model on the host cores;
  ``cpu_baseline_legs`` adds the DeltaNet-layer workload of configs[0] on the port and with pre-dequantised weights.
* ``config.tokens_match_reference``  the K tokens of the first timed block compared, outside the timed region, with
  what the reference's own engine (oracle/_ref, when built) generates from the same prompt.

N > 1 (torchrun): independent replicas, one per GPU, no collective on the data path; ``value`` is the sum over ranks
divided by the slowest rank's time (weak scaling).

``--impl reference`` runs the reference's own engine: its unmodified CUDA sources compiled for sm_100a under oracle/_ref
(see oracle/Makefile), driven through its public decode_token loop on the same checkpoint and prompt, on rank 0 alone.
If that library is absent it falls back to the CPU oracle port.

``--config 1`` times the MXFP4 matrix products alone (the model's three largest shapes at 1, 2, 4, 16 and 64
tokens; 1-4 tokens on packed records, 16 and 64 through the tcgen05 GEMM) and ``--config 2`` the attention
decode kernel over cached contexts of 1024, 8192 and 32768 tokens; both print one JSON line with a ``legs`` list and run on
one GPU.

``--config 5`` (under torchrun with N ranks, one per GPU): the exchange step of a tensor-parallel block -- the one-shot
all-reduce of fp32[4096] over NVLink peer memory beside torch.distributed's (NCCL) all-reduce of the same vector -- and one
MLP block sharded N ways (gate|up rows and down columns per rank, fused GEMV launches, one all-reduce) beside the same block
on one GPU.  Device times, max over ranks.

``--config 4``: ``--batch B`` sequences per GPU decoded in lock step on one weight copy
(2048-token prompts by default, ``--steps`` generated tokens), aggregate tok/s; with ``--speculative`` the batch-1
draft-1 / verify greedy loop with its acceptance rate.
"""
from __future__ import annotations

import argparse
import json
import os
import shutil
import statistics
import subprocess
import sys
import threading
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

import numpy as np  # noqa: E402

HIDDEN, VOCAB = 4096, 248320
WEIGHT_BYTES_PER_TOKEN = 4_217_924_096  # 24 DeltaNet + 8 attention layers + lm_head, 17 bytes / 32 weights
STATE_BYTES_PER_TOKEN = 24 * 2 * (32 * 128 * 128 * 4 + 8192 * 3 * 4)
# (DRAM bytes read + written) / algorithmic bytes of the GEMV kernel in its ncu capture on a 65536 x 4096 matrix
# (reads alone: 1.001); traffic grows in proportion to the rows, so the ratio scales to the mean launch
GEMV_TRAFFIC_RATIO = 1.024
MIN_TIMED_S = 2.0


def parse_args():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=256)
    ap.add_argument("--warmup", type=int, default=16)
    ap.add_argument("--impl", default="native", choices=["native", "reference"])
    ap.add_argument("--config", type=int, default=3, choices=[1, 2, 3, 4, 5])
    ap.add_argument("--shape", default=None, help="config 1: only this matrix, as ROWSxCOLS")
    ap.add_argument("--tokens", type=int, default=None, help="config 1: only this token count; config 2: only this context length")
    ap.add_argument("--sequences", type=int, default=8, help="config 2: sequences of the batched leg (1 = skip it)")
    ap.add_argument("--eager", action="store_true", help="configs 1 and 2: plain launches instead of one CUDA graph of the steps (for profiler captures)")
    ap.add_argument("--prompt", type=int, default=None, help="prompt tokens (default 512 for config 3, 2048 for config 4)")
    ap.add_argument("--seed", type=int, default=0)
    ap.add_argument("--kv-bf16", action="store_true", help="bf16 KV cache (the default is the reference's fp32 cache)")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-reference-check", action="store_true", help="skip comparing the generated tokens with the reference engine")
    ap.add_argument("--gemv", default="mma", choices=["mma", "tcgen05"], help="GEMV kernel family of the persistent kernel's engine (the graph of launches runs tcgen05)")
    ap.add_argument("--persistent", action="store_true", help="the persistent token kernel (one cooperative launch per token) instead of the graph of launches")
    ap.add_argument("--prefetch", type=int, default=-1, help="persistent kernel: weight records per warp kept prefetched into L2 (-1 = default)")
    ap.add_argument("--batch", type=int, default=1, help="config 4: sequences per GPU decoded in lock step (1..8)")
    ap.add_argument("--speculative", action="store_true", help="config 4: batch-1 draft-1 / verify greedy decode through the MTP head")
    args = ap.parse_args()
    if args.prompt is None:
        args.prompt = 512 if args.config == 3 else 2048
    return args


def workdir() -> str:
    for base in ("/dev/shm", "/tmp"):
        try:
            if shutil.disk_usage(base).free > (8 << 30):
                d = os.path.join(base, "insignia_b200_bench")
                os.makedirs(d, exist_ok=True)
                return d
        except OSError:
            pass
    raise RuntimeError("no scratch directory with 8 GiB free")


def ensure_checkpoint(seed: int, use_cuda: bool) -> tuple[str, str]:
    from insignia_b200 import synth

    d = workdir()
    st, idx = os.path.join(d, f"qwen35_synth_seed{seed}.safetensors"), os.path.join(d, f"qwen35_synth_seed{seed}.idx")
    if not (os.path.exists(st) and os.path.exists(idx)):
        tmp = st + ".tmp"
        cfg = synth.SynthConfig(seed=seed, norms="ones", backend="torch" if use_cuda else "numpy")
        synth.write_checkpoint(cfg, tmp)
        os.replace(tmp, st)
        from insignia_b200.checkpoint_io import write_index

        write_index(st, idx)
    return st, idx


class ClockSampler:
    """Samples SM clock and throttle reasons with nvidia-smi while a timed region runs."""

    Q = ("clocks.sm,clocks.max.sm,clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu: int):
        self.gpu, self.rows, self.proc = gpu, [], None

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--id={self.gpu}", f"--query-gpu={self.Q}", "--format=csv,noheader,nounits",
                                          "-lms", "100"], stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except OSError:
            self.proc = None
        return self

    def _read(self):
        for line in self.proc.stdout:
            self.rows.append([c.strip() for c in line.split(",")])

    def __exit__(self, *exc):
        if self.proc:
            self.proc.terminate()
            self.t.join(timeout=2)

    def summary(self) -> dict:
        sm = [float(r[0]) for r in self.rows if len(r) >= 6 and r[0].replace(".", "").isdigit()]
        mx = [float(r[1]) for r in self.rows if len(r) >= 6 and r[1].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({n for r in self.rows if len(r) >= 6 for n, v in zip(names, r[2:6]) if v.lower().startswith("active")})
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(mx) if mx else None, "reasons": reasons,
                "samples": len(sm)}


def measured_hbm_peak() -> tuple[float, str]:
    try:
        return float(json.load(open(os.path.join(ROOT, "MEASURED_PEAKS.json")))["hbm_gbs"]), "measured"
    except Exception:
        return 6650.0, "fallback"


def prompt_for_rank(seed: int, rank: int, n: int) -> np.ndarray:
    """Every replica decodes its own sequence; rank 0's prompt is the one the reference arm decodes."""
    return np.random.default_rng(seed + 1000 * rank).integers(0, VOCAB, n)


def max_over_ranks(ms: float, dist, device) -> float:
    """A step is as slow as the slowest replica: the device time, maximum over the ranks (bracketed by barriers)."""
    import torch

    t = torch.tensor([ms], device=device)
    if dist:
        dist.barrier()
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def job_throughput(world: int, units_per_rank: int, ms: float) -> float:
    """Whole-job throughput of `world` replicas that each processed `units_per_rank` units in `ms` (the maximum over ranks)."""
    return world * units_per_rank / (ms * 1e-3)


def workload_config(args, world: int) -> dict:
    """The keys both arms print, so that their ``config`` objects compare equal apart from the engine's own entries."""
    return {"workload": "configs[3]: 32-layer hybrid (24 DeltaNet + 8 GQA), MXFP4 weights, batch-1 greedy decode after a "
                        f"{args.prompt}-token prompt of seeded uniform-random ids", "prompt_tokens": args.prompt,
            "kv_cache": "bf16" if args.kv_bf16 else "f32", "weights": "seeded N(0,0.02) -> MXFP4, norms 1.0",
            "parallelism": f"replica x{world}" if world > 1 else "single GPU",
            "l2": "weights streamed per token (4.2 GB) exceed the 126 MB L2; no flush needed"}


def cpu_port_baseline(st_path: str, prompt: np.ndarray, budget_s: float = 20.0) -> dict:
    """Times the CPU oracle port on the first tokens of the same workload (all host threads)."""
    from insignia_b200.checkpoint_io import SafetensorsReader
    from oracle import oracle as orc

    m = orc.OracleModel(SafetensorsReader(st_path), max_context=64, gate="broadcast", fast_gemv=True)
    t0 = time.perf_counter()
    m.decode_token(int(prompt[0]))
    t1 = time.perf_counter() - t0
    n = int(max(1, min(8, budget_s / max(t1, 1e-3))))
    t0 = time.perf_counter()
    for i in range(n):
        m.decode_token(int(prompt[1 + i]))
    dt = time.perf_counter() - t0
    return {"value": n / dt, "unit": "tok/s", "cores": orc.num_threads(), "kind": "port",
            "sample": f"{n} greedy tokens of the full 32-layer model from position 1 (after one warm-up token); weights stay MXFP4 "
                      "and are dequantised inside every matrix-vector product"}


def cpu_legs(st_path: str) -> dict:
    """configs[0] on the host: a 64-token run of DeltaNet layer 0 (a) through the port, which dequantises inside every
    product, and (b) with the layer's matrices dequantised once to fp32 and NumPy (BLAS) matrix-vector products."""
    from insignia_b200 import mxfp4
    from insignia_b200.checkpoint_io import SafetensorsReader
    from oracle import oracle as orc

    t = SafetensorsReader(st_path)
    rng = np.random.default_rng(0)
    m = orc.OracleModel(t, max_context=80, gate="broadcast", fast_gemv=True, n_layers=1)
    m.forward_token(1, want_logits=False)
    t0 = time.perf_counter()
    for i in range(64):
        m.forward_token(int(rng.integers(0, VOCAB)), want_logits=False)
    port = 64 / (time.perf_counter() - t0)
    base = "language_model.model.layers.0."
    names = [base + "linear_attn." + n for n in ("in_proj_qkv", "in_proj_z", "in_proj_a", "in_proj_b", "out_proj")] + \
            [base + "mlp." + n for n in ("gate_proj", "up_proj", "down_proj")]
    t0 = time.perf_counter()
    dense = [mxfp4.dequantize(t.get(n + ".weight"), t.get(n + ".scales")) for n in names]
    dq_s = time.perf_counter() - t0
    xs = {w.shape[1]: rng.standard_normal(w.shape[1]).astype(np.float32) for w in dense}
    t0 = time.perf_counter()
    for _ in range(64):
        for w in dense:
            w @ xs[w.shape[1]]
    pre = 64 / (time.perf_counter() - t0)
    return {"cfg0_deltanet_layer_64_tokens_port": {"value": port, "unit": "tok/s", "cores": orc.num_threads(),
                                                   "how": "oracle port, MXFP4 dequantised inside every product"},
            "cfg0_deltanet_layer_64_tokens_predequantised": {"value": pre, "unit": "tok/s", "cores": os.cpu_count(),
                                                             "how": "the layer's eight matrices dequantised once to fp32 "
                                                                    f"({dq_s:.1f} s), then NumPy matrix-vector products only"}}


def reference_tokens(idx: str, prompt, first: int, count: int):
    """The reference engine's greedy continuation of the same prompt (None when oracle/_ref is not built)."""
    from oracle import ref_engine

    if not ref_engine.available():
        return None
    eng = ref_engine.RefEngine(idx, max_context=len(prompt) + count + 8, budget=16 << 30)
    try:
        for t in prompt:
            eng.forward_token(int(t))
        if eng.logits_argmax() != first:
            return []
        out, t = [], first
        for _ in range(count):
            t = eng.decode_token(t)
            out.append(t)
        return out
    finally:
        eng.close()


def run_native(args, rank, world, local_rank):
    import torch

    from insignia_b200.engine import Engine

    torch.cuda.set_device(local_rank)
    dist = None
    if world > 1:
        import torch.distributed as dist

        dist.init_process_group("nccl", device_id=torch.device("cuda", local_rank))
    if rank == 0:
        st, idx = ensure_checkpoint(args.seed, True)
    if dist:
        dist.barrier()
    st, idx = ensure_checkpoint(args.seed, True)
    if args.config == 4:
        return run_config4(args, rank, world, local_rank, dist, st, idx)

    K, W = args.steps, args.warmup
    ctx = args.prompt + W + K + 64
    eng = Engine(idx, max_context=ctx, budget_bytes=16 << 30, kv_bf16=args.kv_bf16, device=local_rank, gemv_tcgen05=args.gemv == "tcgen05",
                 persistent=args.persistent)
    if args.prefetch >= 0:
        eng.set_program_option("prefetch_records", args.prefetch)
    # every rank decodes its own sequence (replicas); rank 0's is the one the reference arm decodes
    prompt = prompt_for_rank(args.seed, rank, args.prompt)
    stream = torch.cuda.ExternalStream(eng.stream, device=local_rank)
    # the prompt goes in by forward_tokens (not part of the metric; reported as "prefill")
    PRE = 40 if args.prompt >= 80 else min(8, args.prompt - 1)
    eng.forward_tokens([int(t) for t in prompt[:PRE]])  # loads and repacks every weight, in both layouts
    torch.cuda.synchronize()
    pa, pb = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    pa.record(stream)
    eng.forward_tokens([int(t) for t in prompt[PRE:]])
    pb.record(stream)
    torch.cuda.synchronize()
    prefill_ms = pa.elapsed_time(pb)
    first = eng.logits_argmax()

    def timed(fn):
        if dist:
            dist.barrier()
        torch.cuda.synchronize()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        out = fn()
        b.record(stream)
        torch.cuda.synchronize()
        return max_over_ranks(a.elapsed_time(b), dist, "cuda"), out

    warm = eng.generate(first, W) if W > 0 else []
    tok = warm[-1] if warm else first
    start_pos = eng.position

    def e2e_block():
        t = tok
        for _ in range(K):
            t = eng.decode_token(t)
        return t

    # Blocks of exactly K steps, each from the same context length (the position is rewound; rows beyond it are simply
    # overwritten), repeated until about MIN_TIMED_S have been timed per arm: more repeats, the median counts.  Every rank
    # runs the same number of blocks (the count is agreed through the max-reduced times).
    blocks, e2e_blocks, launches, first_block = [], [], 0, None
    with ClockSampler(local_rank) as clocks:
        while True:
            eng.position = start_pos
            l0 = eng.launch_count
            ms, toks = timed(lambda: eng.generate(tok, K))
            launches = eng.launch_count - l0
            if first_block is None:
                first_block = toks
            blocks.append(ms)
            if sum(blocks) >= MIN_TIMED_S * 1e3 or len(blocks) >= 64:
                break
        while True:
            eng.position = start_pos
            ms, _ = timed(e2e_block)
            e2e_blocks.append(ms)
            if sum(e2e_blocks) >= MIN_TIMED_S * 1e3 or len(e2e_blocks) >= 64:
                break
    ms, ms_e2e = statistics.median(blocks), statistics.median(e2e_blocks)
    final_ctx = start_pos + K
    # the dominant kernel in its own flow: the token's fused-GEMV launches alone, replayed between two events
    eng.position = start_pos
    chain = eng.profile_gemv_chain(replays=8)
    gemv = {"bytes": chain["bytes"], "ms": chain["ms_per_token"], "launches": chain["launches"]}
    peak, peak_kind = measured_hbm_peak()
    gemv_gbs = gemv["bytes"] / (gemv["ms"] * 1e-3) / 1e9
    kv_bytes = 8 * 1024 * 2 * (2 if args.kv_bf16 else 4) * (start_pos + K // 2)
    token_bytes = WEIGHT_BYTES_PER_TOKEN + STATE_BYTES_PER_TOKEN + kv_bytes
    value = job_throughput(world, K, ms)
    cfg = workload_config(args, world)
    mma_sync = args.persistent and args.gemv == "mma"  # the launch chain runs its products on tcgen05 whatever --gemv says
    cfg.update({"context_at_end": final_ctx, "engine": {"gemv": "mma.sync" if mma_sync else "tcgen05", "token_step": "persistent kernel" if args.persistent else
                                                        "CUDA graph of 162 launches with programmatic dependent launch"},
                "timed_blocks": {"value": len(blocks), "e2e": len(e2e_blocks), "rule": f"blocks of K steps until >= {MIN_TIMED_S} s, median block"}})
    out = {
        "metric": "9B MXFP4 hybrid decode tok/s (bs1)", "value": value, "unit": "tok/s", "n_gpus": world, "steps": K, "warmup": W,
        "ms_per_step": ms / K, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
        "data": "synthetic", "impl": "native", "config": cfg,
        "e2e": {"value": job_throughput(world, K, ms_e2e), "unit": "tok/s", "h2d_bytes_per_step": 8, "d2h_bytes_per_step": 8},
        "gpu_launches": int(launches),
        "token_hbm": {"algorithmic_bytes_per_token": token_bytes, "achieved_gbs": token_bytes / (ms / K * 1e-3) / 1e9,
                      "frac_of_measured_peak": token_bytes / (ms / K * 1e-3) / 1e9 / peak,
                      "frac_of_8tbs": token_bytes / (ms / K * 1e-3) / 1e9 / 8000.0},
        "roofline": {"bound": "hbm", "kernel": "gemv_fused_kernel" if mma_sync else "umma_gemv_kernel", "achieved": gemv_gbs, "peak": peak, "unit": "GB/s",
                     "frac": gemv_gbs / peak, "traffic": gemv["bytes"] / gemv["launches"] * GEMV_TRAFFIC_RATIO,
                     "peak_source": f"{peak_kind} (MEASURED_PEAKS.json hbm_gbs, burst copy)",
                     "bytes_per_launch": gemv["bytes"] / gemv["launches"], "us_per_launch": gemv["ms"] * 1e3 / gemv["launches"],
                     "launches_per_token": gemv["launches"],
                     "timing": "CUDA events around 8 replays of only this kernel's launches of one token (dependent-launch overlap "
                               "on, weights exceed L2)"},
        "clocks": clocks.summary(),
        "prefill": {"value": world * (args.prompt - PRE) / (prefill_ms * 1e-3), "unit": "tok/s", "tokens": args.prompt - PRE,
                    "how": "forward_tokens: passes of up to 1024 tokens through the tcgen05 kernel (16 or 32 tokens per kind::mxf4 "
                           "instruction), the DeltaNet recurrence of a pass in one launch per layer, the attention of a pass in "
                           "two launches per layer; outside the timed metric"},
    }
    if rank == 0 and world == 1:
        if not args.no_reference_check:
            eng.close()  # the reference engine needs its own 10 GB
            eng = None
            ref = reference_tokens(idx, prompt, first, W + K)
            cfg["tokens_match_reference"] = None if ref is None else bool(len(ref) == W + K and ref[:W] == list(warm) and ref[W:] == list(first_block))
        if not args.no_cpu_baseline:
            out["cpu_baseline"] = cpu_port_baseline(st, prompt)
            out["cpu_baseline_legs"] = cpu_legs(st)
    if eng is not None:
        eng.close()
    if rank == 0:
        print(json.dumps(out), flush=True)
    if dist:
        dist.barrier()
        dist.destroy_process_group()


def _event_us(fn, steps, warmup, eager=False):
    """Mean device time of one call: `steps` calls captured into one CUDA graph (so that the host's launch rate is not what
    is measured), the graph replayed three times between CUDA events on the capturing stream; the fastest replay counts."""
    import torch

    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        for _ in range(warmup):
            fn()
        side.synchronize()
        if eager:  # launch by launch: includes the host's launch rate
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(side)
            for _ in range(steps):
                fn()
            b.record(side)
            side.synchronize()
            return a.elapsed_time(b) * 1e3 / steps
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            for _ in range(steps):
                fn()
        graph.replay()
        side.synchronize()
        best = None
        for _ in range(3):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(side)
            graph.replay()
            b.record(side)
            side.synchronize()
            ms = a.elapsed_time(b)
            best = ms if best is None else min(best, ms)
    return best * 1e3 / steps


def run_kernel_configs(args):
    """the matrix product and the attention decode kernels alone, CUDA events on the launching
    (current) stream, operands rotated over copies that together exceed the L2 so that every launch streams from HBM."""
    import torch

    from insignia_b200 import mxfp4, ops

    torch.cuda.set_device(0)
    peak, src = measured_hbm_peak()
    K, W = (args.steps if args.steps != 256 else 20), max(3, min(args.warmup, 5))
    rng = np.random.default_rng(args.seed)
    legs = []
    with ClockSampler(0) as clocks:
        if args.config == 1:
            shapes = [(24576, 4096), (4096, 12288), (248320, 4096)]
            if args.shape:
                shapes = [tuple(int(v) for v in args.shape.lower().split("x"))]
            for rows, cols in shapes:
                base = (rng.standard_normal((min(rows, 4096), cols)) * 0.02).astype(np.float32)
                w, s = mxfp4.quantize_rows(base)
                reps = -(-rows // base.shape[0])
                dw = torch.from_numpy(np.tile(w, (reps, 1))[:rows].view(np.int32)).cuda()
                ds = torch.from_numpy(np.tile(s, (reps, 1))[:rows]).cuda()
                nbytes = rows * cols * 17 // 32
                copies = max(2, -(-(160 << 20) // nbytes))
                for M in ([args.tokens] if args.tokens else [1, 2, 4, 16, 64]):
                    x = torch.randn(M, cols, device="cuda")
                    it = [0]
                    if M >= 16:
                        packs = [ops.repack_umma(dw, ds) for _ in range(copies)]
                        scratch = ops.umma_gemm_scratch(cols, M)
                        kernel = "umma_gemm_kernel (tcgen05 kind::mxf4)"

                        def fn():
                            it[0] += 1
                            ops.gemm_umma(packs[it[0] % copies], x, scratch=scratch)
                    else:
                        packs = [ops.repack(dw, ds) for _ in range(copies)]
                        kernel = "umma_gemv_kernel on packed records (tcgen05 kind::mxf4)"

                        def fn():
                            it[0] += 1
                            ops.gemv_packed(packs[it[0] % copies], x)
                    us = _event_us(fn, K, W, args.eager)
                    legs.append({"rows": rows, "cols": cols, "tokens": M, "kernel": kernel, "us": us, "tok_per_s": M / us * 1e6,
                                 "weight_gbs": nbytes / us * 1e-3, "frac_of_peak": nbytes / us * 1e-3 / peak})
                    del packs
            metric, unit = "MXFP4 matrix product, weight bytes streamed per second", "GB/s"
            head = max(legs, key=lambda l: l["frac_of_peak"])["weight_gbs"]
            work = "configs[1]: y[m] = W x[m], MXFP4 weights, fp32 activations, M tokens"
        else:
            for ctx in ([args.tokens] if args.tokens else [1024, 8192, 32768]):
                for dt in ((torch.bfloat16,) if args.kv_bf16 else (torch.float32, torch.bfloat16)):
                    n = max(2, -(-(160 << 20) // (2 * ctx * 1024 * (4 if dt == torch.float32 else 2))))
                    n = min(n, 40)
                    caches = [(torch.randn(ctx * 1024, device="cuda").to(dt), torch.randn(ctx * 1024, device="cuda").to(dt)) for _ in range(n)]
                    q = torch.randn(4096, device="cuda")
                    scratch = ops.gqa_scratch("cuda", ctx)
                    it = [0]

                    def fn():
                        it[0] += 1
                        k, v = caches[it[0] % n]
                        ops.gqa_decode(q, k, v, ctx, scratch=scratch)
                    us = _event_us(fn, K, W, args.eager)
                    nbytes = 2 * ctx * 1024 * (4 if dt == torch.float32 else 2)
                    if args.sequences <= 1:
                        legs.append({"context": ctx, "kv_cache": "f32" if dt == torch.float32 else "bf16", "sequences": 1, "us": us,
                                     "cache_gbs": nbytes / us * 1e-3, "frac_of_peak": nbytes / us * 1e-3 / peak})
                        del caches
                        continue
                    # several sequences, each with its own cache, in one launch of the fused step (norm, RoPE, cache write, attention)
                    B = args.sequences
                    n8 = max(2, min(6, -(-(160 << 20) // (B * nbytes))))
                    kc8 = [torch.randn(B, ctx * 1024, device="cuda").to(dt) for _ in range(n8)]
                    vc8 = [torch.randn(B, ctx * 1024, device="cuda").to(dt) for _ in range(n8)]
                    qraw, kraw, vraw = torch.randn(B, 8192, device="cuda"), torch.randn(B, 1024, device="cuda"), torch.randn(B, 1024, device="cuda")
                    nwq = torch.ones(256, dtype=torch.int16, device="cuda") * 0x3F80
                    posd = torch.full((1,), ctx - 1, dtype=torch.int32, device="cuda")
                    big = torch.zeros(B * scratch.numel(), dtype=torch.uint8, device="cuda")
                    it8 = [0]

                    def fn8():
                        it8[0] += 1
                        ops.attention_batch(qraw, kraw, vraw, nwq, nwq, kc8[it8[0] % n8], vc8[it8[0] % n8], posd, ctx, big, B)
                    us8 = _event_us(fn8, K, W, args.eager)
                    legs.append({"context": ctx, "kv_cache": "f32" if dt == torch.float32 else "bf16", "sequences": 1, "us": us,
                                 "cache_gbs": nbytes / us * 1e-3, "frac_of_peak": nbytes / us * 1e-3 / peak,
                                 "sequences_8_us": us8, "sequences_8_cache_gbs": B * nbytes / us8 * 1e-3,
                                 "sequences_8_frac_of_peak": B * nbytes / us8 * 1e-3 / peak,
                                 "note": "eight sequences: one launch of the fused step over eight caches"})
                    del kc8, vc8
                    del caches
            metric, unit = "GQA decode (16 query heads, 4 kv heads, head 256), cache bytes streamed per second", "GB/s"
            head = max(legs, key=lambda l: l["frac_of_peak"])["cache_gbs"]
            work = "configs[2]: one query token against a cached context"
    print(json.dumps({"metric": metric, "value": head, "unit": unit, "n_gpus": 1, "steps": K, "warmup": W, "higher_is_better": True,
                      "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic", "impl": "native",
                      "gpu_launches": K * len(legs), "clocks": clocks.summary(),
                      "config": {"workload": work, "peak_gbs": peak, "peak_source": src,
                                 "l2": "operands rotate over copies that together exceed the 126 MB L2"}, "legs": legs}), flush=True)


def tp_shards(rank: int, world: int, seed: int):
    """One MLP's matrices (4096 -> 12288 -> 4096, seeded, the same on every rank) and this rank's shards in the MLX layout:
    rows [r, r + 12288 / world) of gate and up, the matching columns of down."""
    from insignia_b200 import mxfp4

    rng = np.random.default_rng(seed)
    full = {n: mxfp4.quantize_rows((rng.standard_normal(shape) * 0.02).astype(np.float32))
            for n, shape in (("gate", (12288, 4096)), ("up", (12288, 4096)), ("down", (4096, 12288)))}
    per = 12288 // world
    r0, r1 = rank * per, (rank + 1) * per
    shard = {"gate": (full["gate"][0][r0:r1], full["gate"][1][r0:r1]), "up": (full["up"][0][r0:r1], full["up"][1][r0:r1]),
             "down": (np.ascontiguousarray(full["down"][0][:, r0 // 8:r1 // 8]), np.ascontiguousarray(full["down"][1][:, r0 // 32:r1 // 32]))}
    return full, shard, per


def run_tp_blocks(args, rank, world, local_rank):
    """config 5: the tensor-parallel exchange step and one sharded MLP block (see the module docstring)."""
    import torch

    from insignia_b200 import ops

    torch.cuda.set_device(local_rank)
    dist = None
    if world > 1:
        import torch.distributed as dist

        dist.init_process_group("nccl", device_id=torch.device("cuda", local_rank))
    K = args.steps if args.steps != 256 else 200
    dev = lambda a: torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).cuda()  # noqa: E731

    comm = ops.Comm(rank, world, 4096)
    comm.set_timeout(20_000_000)  # 20 ms: a rank out of step ends its waits quickly instead of stretching the run
    if dist:
        mine = torch.frombuffer(bytearray(comm.handle()), dtype=torch.uint8).cuda()
        every = [torch.empty_like(mine) for _ in range(world)]
        dist.all_gather(every, mine)
        comm.connect([h.cpu().numpy().tobytes() for h in every])
    else:
        comm.connect([comm.handle()])

    def graph_us(fn, steps):
        side = torch.cuda.Stream()
        with torch.cuda.stream(side):
            if dist:
                dist.barrier()  # the ranks reach the first exchange together (its waits are short)
            torch.cuda.synchronize()
            for _ in range(3):
                fn()
            side.synchronize()
            if comm.error():
                raise RuntimeError("a wait of the one-shot all-reduce ran out during warm-up (ranks out of step)")
            if dist:
                dist.barrier()
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=side):
                for _ in range(steps):
                    fn()
            g.replay()
            side.synchronize()
            best = None
            for _ in range(3):
                if dist:
                    dist.barrier()
                torch.cuda.synchronize()
                a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                a.record(side)
                g.replay()
                b.record(side)
                side.synchronize()
                ms = max_over_ranks(a.elapsed_time(b), dist, "cuda")
                best = ms if best is None else min(best, ms)
        return best * 1e3 / steps

    x = torch.randn(4096, device="cuda")
    with ClockSampler(local_rank) as clocks:
        oneshot_us = graph_us(lambda: comm.allreduce(x), K)
        nccl_us = None
        if dist:
            try:
                nccl_us = graph_us(lambda: dist.all_reduce(x), K)
            except Exception as e:  # a collective library that cannot be captured is timed launch by launch
                sys.stderr.write(f"[bench] NCCL all-reduce not captured in a graph ({e}); timing eager launches\n")
                torch.cuda.synchronize()
                a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                for _ in range(10):
                    dist.all_reduce(x)
                a.record()
                for _ in range(K):
                    dist.all_reduce(x)
                b.record()
                torch.cuda.synchronize()
                nccl_us = max_over_ranks(a.elapsed_time(b), dist, "cuda") * 1e3 / K

        full, shard, per = tp_shards(rank, world, args.seed)
        P = {n: ops.repack(dev(w), dev(s)) for n, (w, s) in shard.items()}
        hidden = torch.randn(4096, device="cuda", generator=torch.Generator(device="cuda").manual_seed(args.seed))
        nw = torch.ones(4096, dtype=torch.int16, device="cuda") * 0x3F80  # bf16 1.0
        act, y = torch.zeros(per, device="cuda"), torch.zeros(4096, device="cuda")

        def block():
            ops.gemv_fused(hidden, [dict(packed=P["gate"], packed2=P["up"], out=act, rows=per, epilogue="swiglu")], prologue="rmsnorm", norm_w=nw)
            ops.gemv_fused(act, [dict(packed=P["down"], out=y, rows=4096, epilogue="store")], cols=per)
            comm.allreduce(y)

        tp_us = graph_us(block, K)
        block()
        torch.cuda.synchronize()
        got = y.cpu().numpy()
        single_us, err = None, None
        if rank == 0:
            F = {n: ops.repack(dev(w), dev(s)) for n, (w, s) in full.items()}
            act1, y1 = torch.zeros(12288, device="cuda"), torch.zeros(4096, device="cuda")

            def block1():
                ops.gemv_fused(hidden, [dict(packed=F["gate"], packed2=F["up"], out=act1, rows=12288, epilogue="swiglu")], prologue="rmsnorm", norm_w=nw)
                ops.gemv_fused(act1, [dict(packed=F["down"], out=y1, rows=4096, epilogue="store")], cols=12288)

            if world == 1:
                single_us = tp_us
            block1()
            torch.cuda.synchronize()
            want = y1.cpu().numpy()
            err = float(np.max(np.abs(got - want)) / np.abs(want).max())
        if dist:
            dist.barrier()
        if rank == 0 and world > 1:  # the same block on one GPU, timed alone (the other ranks idle)
            side_fn = block1
            single_us = None
            s2 = torch.cuda.Stream()
            with torch.cuda.stream(s2):
                for _ in range(3):
                    side_fn()
                s2.synchronize()
                g = torch.cuda.CUDAGraph()
                with torch.cuda.graph(g, stream=s2):
                    for _ in range(K):
                        side_fn()
                g.replay()
                s2.synchronize()
                a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                a.record(s2)
                g.replay()
                b.record(s2)
                s2.synchronize()
                single_us = a.elapsed_time(b) * 1e3 / K
        if dist:
            dist.barrier()
    if rank == 0:
        print(json.dumps({"metric": "tensor-parallel exchange step: all-reduce of fp32[4096], device time", "value": oneshot_us, "unit": "us",
                          "n_gpus": world, "steps": K, "warmup": 3, "higher_is_better": False, "scaling": "strong", "vs_baseline": None,
                          "dtype": "f32", "data": "synthetic", "impl": "native", "gpu_launches": K * 4, "clocks": clocks.summary(),
                          "config": {"workload": "one-shot all-reduce over NVLink peer memory (one kernel per rank) and one MLP block "
                                                 "(4096 -> 12288 -> 4096, MXFP4) sharded over the ranks", "parallelism": f"tp{world}"},
                          "allreduce_us": {"oneshot": oneshot_us, "nccl": nccl_us},
                          "mlp_block_us": {"sharded": tp_us, "one_gpu": single_us, "max_rel_difference": err}}), flush=True)
    comm.close()
    if dist:
        dist.barrier()
        dist.destroy_process_group()


def run_config4(args, rank, world, local_rank, dist, st, idx):
    """``--batch`` sequences per GPU in lock step on one weight copy (the prompt goes through the same batch
    steps), or the batch-1 draft-1 / verify loop with ``--speculative``."""
    import torch

    from insignia_b200.engine import Batch, Engine

    K, W, B = args.steps, args.warmup, args.batch
    ctx = args.prompt + W + K + 16
    rng = np.random.default_rng(args.seed + 1000 * rank)
    eng = Engine(idx, max_context=ctx if args.speculative else 64, budget_bytes=24 << 30, kv_bf16=args.kv_bf16, device=local_rank)
    extra = {}

    def timed(stream, fn):
        if dist:
            dist.barrier()
        torch.cuda.synchronize()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        out = fn()
        b.record(stream)
        torch.cuda.synchronize()
        return max_over_ranks(a.elapsed_time(b), dist, "cuda"), out

    with ClockSampler(local_rank) as clocks:
        if args.speculative:
            prompt = [int(t) for t in rng.integers(0, VOCAB, args.prompt)]
            stream = torch.cuda.ExternalStream(eng.stream, device=local_rank)
            # the plain greedy continuation first: the right drafts for the upper-bound leg
            first = eng.prime_speculative(prompt)
            truth = eng.generate(first, W + K)

            def leg(forced):
                eng.reset()
                tok = eng.prime_speculative(prompt)
                if W > 0:
                    toks, _ = eng.generate_speculative(tok, W, forced_drafts=truth[:W] if forced else None)
                    tok = toks[-1]
                ms, (toks, acc) = timed(stream, lambda: eng.generate_speculative(tok, K, forced_drafts=truth[W:W + K] if forced else None))
                return ms, toks, acc

            ms_right, toks_right, acc_right = leg(True)
            ms, toks, accepted = leg(False)
            seqs, launches = 1, 0
            extra = {"draft_acceptance": accepted / max(1, K), "identical_to_plain_greedy": toks == truth[W:W + K] and toks_right == truth[W:W + K],
                     "all_drafts_right": {"value": job_throughput(world, K, ms_right), "unit": "tok/s", "accepted": acc_right,
                                          "how": "the same loop with the right drafts supplied by the caller: the bound a trained MTP head approaches"},
                     "note": "random-weight MTP head: its drafts are almost never accepted, so a step costs a draft plus a two-token verify "
                             "pass for one token"}
        else:
            bt = Batch(eng, B, ctx)
            stream = torch.cuda.ExternalStream(bt.stream, device=local_rank)
            prompts = rng.integers(0, VOCAB, (B, args.prompt))
            t0 = time.perf_counter()
            for i in range(args.prompt - 1):
                bt.forward_tokens(prompts[:, i])
            first = bt.decode_tokens(prompts[:, -1])
            torch.cuda.synchronize()
            extra["prompt_s"] = time.perf_counter() - t0
            if W > 0:
                first = list(bt.generate(first, W)[-1])
            l0 = bt.launch_count
            ms, _ = timed(stream, lambda: bt.generate(first, K))
            launches, seqs = bt.launch_count - l0, B
            bt.close()
    out = {"metric": "9B MXFP4 hybrid decode tok/s (batch, aggregate)", "value": job_throughput(world, seqs * K, ms), "unit": "tok/s",
           "n_gpus": world, "steps": K, "warmup": W, "ms_per_step": ms / K, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
           "dtype": "f32", "data": "synthetic", "impl": "native", "gpu_launches": int(launches), "clocks": clocks.summary(),
           "config": {"workload": f"configs[4]: {seqs} sequence(s) per GPU, {args.prompt}-token prompts of seeded uniform-random ids, "
                                  f"{K} generated tokens" + (", draft-1 / verify greedy decode through the MTP head" if args.speculative else
                                                             ", decoded in lock step on one weight copy"),
                      "sequences_per_gpu": seqs, "prompt_tokens": args.prompt, "kv_cache": "bf16" if args.kv_bf16 else "f32",
                      "parallelism": f"replica x{world}" if world > 1 else "single GPU", **extra}}
    eng.close()
    if rank == 0:
        print(json.dumps(out), flush=True)
    if dist:
        dist.barrier()
        dist.destroy_process_group()


def run_reference(args, rank, world, local_rank):
    if rank != 0:
        return  # the reference is single-GPU, single-sequence: rank 0 alone runs it
    K, W = args.steps, args.warmup
    prompt = prompt_for_rank(args.seed, 0, args.prompt)
    # n_gpus is what this arm used: one GPU, whatever the launch's world size
    base = {"metric": "9B MXFP4 hybrid decode tok/s (bs1)", "unit": "tok/s", "n_gpus": 1, "steps": K, "warmup": W,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
            "impl": "reference"}
    cfg = workload_config(args, 1)
    from oracle import ref_engine

    if ref_engine.available():
        import torch

        torch.cuda.set_device(local_rank)
        st, idx = ensure_checkpoint(args.seed, True)
        eng = ref_engine.RefEngine(idx, max_context=args.prompt + W + K + 64, budget=16 << 30)
        for t in prompt:
            eng.forward_token(int(t))
        tok = eng.logits_argmax()
        for _ in range(W):
            tok = eng.decode_token(tok)
        start_pos = eng.position
        blocks = []
        with ClockSampler(local_rank) as clocks:
            while True:
                eng.position = start_pos
                torch.cuda.synchronize()
                a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                a.record()
                t = tok
                for _ in range(K):
                    t = eng.decode_token(t)
                b.record()
                torch.cuda.synchronize()
                blocks.append(a.elapsed_time(b))
                if sum(blocks) >= MIN_TIMED_S * 1e3 or len(blocks) >= 64:
                    break
        ms = statistics.median(blocks)
        eng.close()
        v = K / (ms * 1e-3)
        cfg.update({"context_at_end": start_pos + K,
                    "engine": {"what": "the reference's CUDA sources, unmodified, compiled for sm_100a with its own flags (-O3 --use_fast_math), "
                                       "driven through Qwen35Decode::decode_token (src/decode.cu:23) on this GPU"},
                    "timed_blocks": {"value": len(blocks), "e2e": len(blocks), "rule": f"blocks of K steps until >= {MIN_TIMED_S} s, median block"}})
        base.update({"value": v, "ms_per_step": ms / K, "clocks": clocks.summary(), "config": cfg,
                     "cpu_baseline": {"value": v, "unit": "tok/s", "cores": 1, "kind": "reference", "runs_on": "gpu",
                                      "sample": f"{K} greedy tokens after a {args.prompt}-token prompt.  The reference has no multi-token CPU "
                                                "implementation: this is its own GPU engine, one host thread driving ~580 launches per token; "
                                                "the CPU figure of this path is the native arm's cpu_baseline (oracle port)"},
                     "e2e": {"value": v, "unit": "tok/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}})
    else:
        st, idx = ensure_checkpoint(args.seed, False)
        cb = cpu_port_baseline(st, prompt)
        cfg.update({"context_at_end": 0, "engine": {"what": "CPU oracle port (oracle/_ref not built)"}, "timed_blocks": {"value": 1, "e2e": 1, "rule": "bounded sample"}})
        base.update({"value": cb["value"], "ms_per_step": 1e3 / cb["value"], "cpu_baseline": cb, "config": cfg,
                     "e2e": {"value": cb["value"], "unit": "tok/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}})
    print(json.dumps(base), flush=True)


def main():
    args = parse_args()
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))
    if args.config in (1, 2):
        if rank == 0:
            run_kernel_configs(args)
    elif args.config == 5:
        run_tp_blocks(args, rank, world, local_rank)
    elif args.impl == "reference":
        run_reference(args, rank, world, local_rank)
    else:
        run_native(args, rank, world, local_rank)


if __name__ == "__main__":
    main()
