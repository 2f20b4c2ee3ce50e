"""Down projections of three tokens and more fetch their prepared digits with the weights of each stage instead of as one image."""
import pytest

from tests.test_digit_image_gpu import test_prepared_chain_equals_fp32_chain as _chain

pytestmark = pytest.mark.gpu
pytest.importorskip("torch")


# 96 and 88 k-blocks: stages of two in every quarter (12 and 11); 95 and 93: quarters of odd lengths, which keep the image
@pytest.mark.parametrize("tokens,inter", [(3, 12288), (4, 93 * 128), (5, 95 * 128), (6, 88 * 128), (8, 12288)])
def test_streamed_digits_equal_the_fp32_chain(cuda, tokens, inter):
    _chain(cuda, tokens, inter)
