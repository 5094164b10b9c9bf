"""Biased attention of a context pass over many tiles of the cache, for every number of 64-column chunks of a key, up to the cache's last row."""
import numpy as np
import pytest

from tests.conftest import rel_err
from tests.test_finuvik_kernels_gpu import TOL, Attn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,G,dk,dv", [(2, 1, 64, 64), (4, 2, 128, 128), (2, 2, 144, 48), (3, 1, 192, 256), (2, 1, 208, 128), (1, 1, 256, 16)])
def test_many_tiles(cuda, ob, H, G, dk, dv):
    hist, counts = [0, 449, 575, 63], [700, 130, 129, 1]
    t = Attn(cuda, ob, "bf16", H, G, dk, dv, [h + c for h, c in zip(hist, counts)], 704, seed=dk + dv)
    q = t.queries(counts)
    got = t.context(hist, q)
    at = 0
    for b, (h, n) in enumerate(zip(hist, counts)):
        pick = np.unique(np.r_[0, n // 2, max(n - 2, 0), n - 1, np.arange(0, n, 31)])
        # the bound of the shorter sequences: an error of 2^-9 in a weight or a value whatever their number
        assert rel_err(got[at + pick], t.reference(b, q[b][pick], h + pick)) < TOL["bf16"], b
        at += n
