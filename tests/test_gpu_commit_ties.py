"""The quantiser's codes where (value - minimum) / scale lies on or next to a tie, where the range is empty, and next to
the clamp: there the product with the reciprocal may not stand in for the division. Byte-equal to the oracle."""
import importlib

import numpy as np
import pytest

torch = pytest.importorskip("torch")


@pytest.mark.gpu
@pytest.mark.parametrize("seed,step,lo", [(0, 0.5, 0.0), (1, 0.5, -7.5), (2, 0.25, 3.0), (3, 1.5, -100.0), (4, 2.0 ** -14, 0.0), (5, 1000.0, -15000.0)])
def test_codes_on_ties(orc, pkg, seed, step, lo):
    api = importlib.import_module(pkg.__name__ + ".api")
    g = np.random.default_rng(seed)
    nb = 5                                                        # 15 steps of 2 between the extremes: odd multiples of `step` are ties
    k = g.integers(0, 31, (2, nb, 32, 4, 128))
    k[..., 0] = 0; k[..., 1] = 30                                 # V: both extremes in every token
    k[0][:, 0] = 0; k[0][:, 1] = 30                               # K: in every channel
    x = (lo + step * k).astype(np.float16)
    bits = x.view(np.uint16)
    near = g.random(x.shape) < 0.3                                # a third of the values one fp16 step beside the tie
    bits[near & (k > 0) & (k < 30)] += 1
    x[:, nb - 1] = lo                                             # an empty range
    want = np.zeros((4, nb, orc.REC_BYTES), np.uint8)
    orc.kv_commit(x[0], x[1], want, nb, 0)
    cache = torch.zeros((4, nb, orc.REC_BYTES), dtype=torch.uint8, device="cuda")
    api.kv_commit(torch.from_numpy(x[0]).cuda(), torch.from_numpy(x[1]).cuda(), cache, nb, 0)
    torch.cuda.synchronize()
    assert np.array_equal(cache.cpu().numpy(), want)
