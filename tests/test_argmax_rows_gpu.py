"""The arg-max of logit rows (a cluster of eight CTAs per row) against numpy's first maximum."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), ".."))

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


# n: fewer entries than CTAs (some slices are empty), one each, one more, around a CTA's threads, the vocabulary
@pytest.mark.parametrize("n", [1, 7, 8, 9, 513, 4097, 248320])
@pytest.mark.parametrize("count", [1, 2, 8])
def test_argmax_rows(cuda, n, count):
    from insignia_b200 import _lib

    rng = np.random.default_rng(n + count)
    stride = n + 5  # what lies past a row's n entries is larger than all of them and must not count
    per = (n + 7) // 8
    for trial in range(8):  # the winner in each CTA's slice in turn
        x = rng.standard_normal((count, stride)).astype(np.float32)
        x[:, n:] = 100
        for r in range(count):
            at = min(n - 1, ((trial + r) % 8) * per + int(rng.integers(0, per)))
            x[r, at] = 50
            x[r, min(n - 1, at + per):n:max(1, per)] = 50  # the same value in later slices: the lowest index wins
        d, out = torch.from_numpy(x).cuda(), torch.full((count,), -1, dtype=torch.int32, device="cuda")
        _lib.check(_lib.lib().insg_argmax_rows(d.data_ptr(), stride, n, count, out.data_ptr(), torch.cuda.current_stream().cuda_stream))
        assert out.cpu().tolist() == np.argmax(x[:, :n], axis=1).tolist()
