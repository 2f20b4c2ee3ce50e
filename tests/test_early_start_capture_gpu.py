"""Calls that start before the launch ahead of them has ended, captured into a graph behind whatever can stand ahead of them: a memset, a copy, a kernel
of another stream, several streams that meet.  The graph's results are those of the calls apart, also when it is replayed on new inputs."""
import functools
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), ".."))
from tests.test_kernels_gpu import bf16, dev, host, rand_matrix  # noqa: E402

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@functools.lru_cache(1)
def _calls(ops):
    """Name -> (inputs as host arrays from a generator, the call on device inputs)."""
    rng = np.random.default_rng(1)
    w, s = rand_matrix(rng, 3072, 4096)
    large, umma, small = ops.repack(dev(w), dev(s)), ops.repack_umma(dev(w), dev(s)), ops.repack(dev(w[:256]), dev(s[:256]))
    norm = dev(bf16(rng, 256))
    scratch = torch.zeros(8 * ops.gqa_scratch("cuda").numel(), dtype=torch.uint8, device="cuda")
    f32 = lambda *shape: (lambda g: g.standard_normal(shape).astype(np.float32))  # noqa: E731
    gem = ops.umma_gemm_scratch(4096, 61)

    def steps(n):
        def run(state, qkv, g, beta):
            st, flat = state.clone(), qkv.view(-1)
            return torch.cat([ops.deltanet_decode_tokens(st, flat, flat[2048:], flat[4096:], -g.abs(), beta.sigmoid(), n, 8192).view(-1), st])
        return [f32(32 * 128 * 128), f32(n, 8192), f32(n, 32), f32(n, 32)], run

    def batch(q, k, v, kc, vc):
        pos = torch.full((1,), 599, dtype=torch.int32, device="cuda")
        return ops.attention_batch(q, k, v, norm, norm, kc.clone(), vc.clone(), pos, 600, scratch, 2)

    return {
        "records": ([f32(3, 4096)], lambda x: ops.gemv_packed(large, x)),
        "mma.sync": ([f32(2, 4096)], lambda x: ops.gemv_packed(small, x)),
        "image": ([f32(2, 4096)], lambda x: ops.gemm_umma(umma, x, scratch=gem)),
        "gemm": ([f32(61, 4096)], lambda x: ops.gemm_umma(umma, x, scratch=gem)),
        "step": steps(1),
        "steps": steps(5),
        "attention": ([f32(4096), f32(5000 * 1024), f32(5000 * 1024)], lambda q, k, v: ops.gqa_decode(q, k, v, 5000, scratch=scratch)),
        "batch": ([f32(2, 8192), f32(2, 1024), f32(2, 1024), f32(2, 600 * 1024), f32(2, 600 * 1024)], batch),
    }


@pytest.mark.parametrize("ahead", ["memset", "copy", "kernel", "other stream", "streams that meet", "stream and memset"])
@pytest.mark.parametrize("name", ["records", "mma.sync", "image", "gemm", "step", "steps", "attention", "batch"])
def test_captured_behind_anything(cuda, name, ahead):
    from insignia_b200 import ops

    make, call = _calls(ops)[name]
    draws = [[m(np.random.default_rng(seed)) for m in make] for seed in (1, 2, 3)]
    source = [dev(a) for a in draws[0]]  # what the graph is replayed on
    want = []
    for d in draws:
        want.append(host(call(*[dev(a) for a in d])).copy())
        torch.cuda.synchronize()

    main, side = torch.cuda.Stream(), torch.cuda.Stream()
    main.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(main), torch.cuda.graph(graph, stream=main):
        inputs, other = [torch.empty_like(t) for t in source], torch.empty(1 << 22, device="cuda")
        if ahead in ("other stream", "streams that meet", "stream and memset"):
            side.wait_stream(main)
            with torch.cuda.stream(side):
                for t, a in zip(inputs, source):
                    torch.mul(a, 1.0, out=t)
                if ahead == "stream and memset":
                    other.zero_()
            if ahead == "streams that meet":
                torch.mul(other, 2.0, out=other)
            main.wait_stream(side)
            if ahead == "stream and memset":
                other[: 1 << 20].zero_()
        else:
            for t, a in zip(inputs, source):
                if ahead == "copy":
                    t.copy_(a)
                else:
                    torch.mul(a, 1.0, out=t)
            if ahead == "memset":
                other.zero_()
        out = call(*inputs)
        again = call(*inputs)  # and behind itself
    for d, y in zip(draws, want):
        for t, a in zip(source, d):
            t.copy_(dev(a))
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(host(out), y) and np.array_equal(host(again), y)
