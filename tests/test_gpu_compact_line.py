"""Row lists of masks around the line between listed and walked chunks (32,768
rows, a quarter of them): one more and one fewer, spread and in one run."""
import numpy as np
import pytest
import torch

import falcondb_b200 as F
from falcondb_b200 import ops

pytestmark = pytest.mark.gpu

CHUNK = 32_768


@pytest.mark.parametrize("spread", [False, True])
@pytest.mark.parametrize("extra", [-1, 0, 1])
@pytest.mark.parametrize("n", [CHUNK, 3 * CHUNK + 4097])
def test_chunks_at_the_line(db, n, extra, spread):
    r = np.random.default_rng([n, extra + 1])
    m = np.zeros(n, dtype=bool)
    for c0 in range(0, n, CHUNK):
        rows = min(CHUNK, n - c0)
        take = min(rows, CHUNK // 4 + extra)
        m[c0 + (r.permutation(rows)[:take] if spread else rows - take + np.arange(take))] = True
    w = torch.from_numpy(F.validity_words(m).view(np.int64)).cuda()
    rows, cnt = ops.compact(db, w, n)
    assert int(cnt.item()) == m.sum()
    assert np.array_equal(rows[:int(m.sum())].cpu().numpy(), np.nonzero(m)[0])
