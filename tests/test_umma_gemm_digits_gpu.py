"""The tcgen05 GEMM's seven digits per activation: groups whose largest element lies at either side of the extra bit, every digit's
edge values, and token counts at the edges of the groups of 16 (few tokens or little work) and of 32 (pairs of CTAs: "pairs", with so many tokens
in the last group)."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), ".."))
from oracle import oracle as orc  # noqa: E402
from tests.fixtures import pair_tokens  # noqa: E402
from tests.test_kernels_gpu import dev, host, rand_matrix  # noqa: E402

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

EDGE = 1 + 0x1F0000 / 2**23  # mantissas below it keep one bit more


@pytest.mark.parametrize("tokens,pairs", [(9, 0), (16, 0), (17, 0), (48, 0), (49, 0), (64, 0), (65, 0), ("pairs", 1), ("pairs", 16), ("pairs", 32)])
def test_digits_at_the_edges(cuda, tokens, pairs):
    from insignia_b200 import ops

    rows, cols = 2592 if pairs else 160, 640  # a last tile of 32 rows; five k-blocks
    if pairs:
        tokens = pair_tokens(rows, cols, last=pairs)
    rng = np.random.default_rng(tokens)
    w, s = rand_matrix(rng, rows, cols)
    # each group of 32: its largest element at a chosen mantissa, the others anywhere below, many of them at multiples of powers of 13
    largest = np.array([1, np.nextafter(np.float32(EDGE), np.float32(0)), EDGE, np.nextafter(np.float32(2), np.float32(0)), 1.5], np.float32)
    groups = tokens * cols // 32
    top = largest[rng.integers(0, 5, groups)] * np.float32(2.0) ** rng.integers(-20, 20, groups).astype(np.float32)
    x = (rng.uniform(-1, 1, (groups, 32)) * top[:, None]).astype(np.float32)
    k = rng.integers(0, 7, (groups, 8))
    unit = 2.0 ** np.floor(np.log2(top))[:, None] / 2**23
    x[:, 8:16] = np.clip(rng.integers(-12, 13, (groups, 8)) * 13.0**k * unit, -top[:, None], top[:, None])
    x[:, 0] = top * rng.choice([-1, 1], groups)
    x = x.reshape(tokens, cols)
    y = host(ops.gemm_umma(ops.repack_umma(dev(w), dev(s)), dev(x)))
    weights = np.abs(host(ops.dequant_mlx(dev(w), dev(s))).astype(np.float64))
    room = np.repeat(top.reshape(tokens, cols // 32), 32, axis=1).astype(np.float64)
    for m in range(tokens):
        # an element is off by half a unit of at most 2^-23 of its group's largest power of two; the sums of 32-element groups (fp32,
        # truncated) and the seven combinations add an ulp of the sum of magnitudes each at the very most
        bound = weights @ room[m] * 2.0**-24 + weights @ np.abs(x[m].astype(np.float64)) * 2.0**-23 * 8
        assert np.all(np.abs(y[m] - orc.gemv_mlx_f64(w, s, x[m])) <= bound), m


BASE = 13


def spread_values(rng, count, limit):
    """`count` integers up to `limit` in magnitude: every residue of each of the three digit pairs, the carries between them (a pair of digits that
    ends negative takes one from the next pair), every last digit."""
    n = np.stack([rng.permutation(np.arange(count) % BASE**2) for _ in range(3)])
    last = rng.permutation(np.arange(count) % 9) - 4
    v = n[0] + BASE**2 * n[1] + BASE**4 * n[2] + BASE**6 * last.astype(np.int64)
    return np.where(np.abs(v) <= limit, v, v % (2 * limit + 1) - limit)


@pytest.mark.parametrize("tokens,pairs", [(9, 0), (16, 0), (17, 0), (48, 0), (49, 0), (64, 0), (65, 0), ("pairs", 1), ("pairs", 17), ("pairs", 32)])
def test_every_digit_reaches_the_product(cuda, tokens, pairs):
    """Rows with a single weight of one: each product is one activation as its digits hold it, the nearest multiple of its group's unit, and
    nothing rounds on the way but the seventh digit's addition.  Bit for bit."""
    from insignia_b200 import mxfp4, ops

    cols, copies = 384, 11 if pairs else 1  # three k-blocks, three tiles of rows: an odd one; 33: a unit of a single tile behind eight of four
    if pairs:
        tokens = pair_tokens(copies * cols, cols, last=pairs)
    rng = np.random.default_rng(100 + tokens)
    eye = np.tile(np.eye(cols, dtype=np.float32), (copies, 1))
    w, s = mxfp4.quantize_rows(eye)
    assert np.array_equal(host(ops.dequant_mlx(dev(w), dev(s))), eye)
    largest = np.array([1, np.nextafter(np.float32(EDGE), np.float32(0)), EDGE, np.nextafter(np.float32(2), np.float32(0)), 1.5], np.float64)
    groups = tokens * cols // 32
    mantissa, exponent = largest[np.arange(groups) % 5], rng.integers(-20, 20, groups)
    unit = 2.0 ** (exponent - np.where(mantissa < EDGE, 24, 23))  # one bit more below the edge
    limit = (mantissa * 2.0**exponent / unit).astype(np.int64)
    v = np.stack([spread_values(rng, groups, 2**24 - 1) for _ in range(32)], axis=1)
    v = np.clip(v, -limit[:, None], limit[:, None])
    x = v * unit[:, None]
    x[:, 16:24] += rng.uniform(-0.5, 0.5, (groups, 8)) * unit[:, None]  # between two multiples
    x = np.clip(x, -(mantissa * 2.0**exponent)[:, None], (mantissa * 2.0**exponent)[:, None])
    top = rng.integers(0, 32, groups)
    x[np.arange(groups), top] = mantissa * 2.0**exponent * rng.choice([-1, 1], groups)
    x = x.astype(np.float32)
    want = (np.rint(x.astype(np.float64) / unit[:, None]) * unit[:, None]).astype(np.float32).reshape(tokens, cols)
    got = host(ops.gemm_umma(ops.repack_umma(dev(w), dev(s)), dev(x.reshape(tokens, cols))))
    assert np.array_equal(got, np.tile(want, (1, copies)))


@pytest.mark.parametrize("tokens,rows,cols", [(t, 256, c) for t in (16, 61) for c in (640, 4096, 12288)] + [("pairs", 1152, 4096), ("pairs", 384, 12288)])
def test_products_of_normal_vectors(cuda, tokens, rows, cols):
    """An activation is off by a uniform half unit, 2^-22 of sqrt(1/12) = 0.7e-7 for groups whose largest lies in [2, 4); signs are random,
    so the product is off by as much of its root mean square, and its fp32 sums and combinations by about as much again."""
    from insignia_b200 import ops

    if tokens == "pairs":
        tokens = pair_tokens(rows, cols)
    rng = np.random.default_rng(cols + tokens)
    w, s = rand_matrix(rng, rows, cols)
    x = rng.standard_normal((tokens, cols)).astype(np.float32)
    y = host(ops.gemm_umma(ops.repack_umma(dev(w), dev(s)), dev(x)))
    y64 = np.stack([orc.gemv_mlx_f64(w, s, x[m]) for m in range(tokens)])
    assert np.sqrt(np.mean((y - y64) ** 2) / np.mean(y64**2)) <= 2e-7
