"""The products of a token, replayed alone: those that a token runs."""
import pytest

from tests.test_model_gpu import small_engine

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def test_the_chain_has_a_tokens_products(cuda, golden_ckpt):
    with small_engine(golden_ckpt[1]) as e:
        e.decode_token(1)
        chain = e.profile_gemv_chain(replays=2)
        # four a layer and the head; the second and third DeltaNet layer, whose input comes prepared, make their gates apart from the in-projection
        assert chain["launches"] == 4 * 4 + 2 + 1, chain
        weights = 4 * 3 * 4096 * 12288 + 3 * (12352 + 4096) * 4096 + (8192 + 2048 + 4096) * 4096 + 64 * 4096
        assert chain["bytes"] == weights * 17 // 32
