"""Row lists of masks whose last chunk (of 32,768 rows) has few of them, around the
half of its rows up to which it is listed."""
import numpy as np
import pytest
import torch

import falcondb_b200 as F
from falcondb_b200 import ops

pytestmark = pytest.mark.gpu

CHUNK = 32_768


@pytest.mark.parametrize("rows", [1, 63, 64, 3968, 10_000, CHUNK - 1, CHUNK, CHUNK + 3968])
@pytest.mark.parametrize("share", [0.3, 0.49, 0.51, 0.9, 1.0])
def test_a_part_chunk(db, rows, share):
    """Half of a last chunk's rows: its line."""
    m = np.random.default_rng([rows, int(share * 100)]).random(rows) < share
    w = torch.from_numpy(F.validity_words(m).view(np.int64)).cuda()
    got, cnt = ops.compact(db, w, rows)
    assert int(cnt.item()) == m.sum()
    assert np.array_equal(got[:int(m.sum())].cpu().numpy(), np.nonzero(m)[0])
