"""Engines whose products normalise their own inputs leave the normalised residual stream in the workspace's `norm`."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), ".."))

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gemv_tcgen05", [False, True])
def test_norm_holds_the_heads_input_after_a_token(cuda, golden_ckpt, gemv_tcgen05):
    from insignia_b200.engine import Engine

    weights = []
    with Engine(golden_ckpt[1], n_layers=4, vocab=64, max_context=64, prepared_inputs=False, gemv_tcgen05=gemv_tcgen05) as e:
        for token in (3, 5, 9, 12):  # eager steps and replays of the captured graph
            e.decode_token(token)
            h = e.read("hidden").astype(np.float64)
            weights.append(e.read("norm") / (h / np.sqrt(np.mean(h * h) + 1e-6)))  # the final norm's weight, whatever the token
    for w in weights[1:]:
        assert np.max(np.abs(w - weights[0])) <= 1e-5 * np.abs(weights[0]).max()  # a few fp32 roundings
