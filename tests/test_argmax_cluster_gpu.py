"""The greedy pick with one CTA and with a cluster of eight (65536 logits and more)."""
import numpy as np
import pytest
import torch

from tests.gpu_util import ptr, stream

pytestmark = pytest.mark.gpu


# around the line between the two forms, a last piece of every size, rows that start off a 16-byte boundary
@pytest.mark.parametrize("vocab", [1, 65535, 65536, 65537, 98304, 151936, 248320, 248327])
@pytest.mark.parametrize("shift", [0, 1])
def test_argmax_advance(lib, vocab, shift):
    rng = np.random.default_rng(vocab + shift)
    x = torch.from_numpy(rng.integers(-8, 8, vocab + 8).astype(np.float16)).cuda()[shift:]      # many equal maxima
    one = lambda v: torch.full((1,), v, dtype=torch.int64, device="cuda")
    tok, pos, length, count, history = one(-1), one(5), one(6), one(0), torch.zeros(8, dtype=torch.int64, device="cuda")
    spots = [vocab - 1, vocab // 2, 0]
    want = []
    for i in spots:                          # each maximum lies below the one before: the lowest index wins
        x[i] = 100.0
        want.append(i)
        assert lib.launch_argmax_advance(ptr(x), vocab, ptr(tok), ptr(pos), ptr(length), ptr(history), ptr(count), 8, stream()) == 0
    x[:vocab] = float("nan")
    x[vocab // 3] = -3.0                     # NaN is never the largest
    want.append(vocab // 3)
    assert lib.launch_argmax_advance(ptr(x), vocab, ptr(tok), ptr(pos), ptr(length), ptr(history), ptr(count), 8, stream()) == 0
    torch.cuda.synchronize()
    assert history[:4].tolist() == want and tok.item() == want[-1]
    assert (pos.item(), length.item(), count.item()) == (9, 10, 4)
