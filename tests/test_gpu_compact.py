"""Row lists of masks at the edges of a compaction chunk (512 words) and on both
sides of the density where a chunk is listed in shared memory first (2048 of its
32768 rows)."""
import numpy as np
import pytest
import torch

import falcondb_b200 as F
from falcondb_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 65, 32_767, 32_768, 32_769, 3 * 32_768 + 5])
@pytest.mark.parametrize("count", [0, 1, 2047, 2048, 2049, "half", "all"])
def test_compact_densities(db, n, count):
    r = np.random.default_rng(n)
    bits = np.zeros(n, bool)
    for a in range(0, n, 32_768):  # the same number of rows in every chunk
        m = min(32_768, n - a)
        k = {"half": m // 2, "all": m}.get(count, count)
        bits[a + r.permutation(m)[:k]] = True
    mask = torch.from_numpy(F.validity_words(bits).view(np.int64)).cuda()
    rows, cnt = ops.compact(db, mask, n)
    k = int(cnt.item())
    assert np.array_equal(rows[:k].cpu().numpy(), np.nonzero(bits)[0])
    # A shorter output takes the first rows and reports the rest as an error.
    if k > 1:
        short = torch.full((k + 64,), -7, dtype=torch.int32, device="cuda")
        F.check(F.lib().fdb_compact_mask(db.handle, mask.data_ptr(), n, short.data_ptr(), k // 2, cnt.data_ptr()))
        with pytest.raises(F.FalconError):
            db.synchronize()
        got = short.cpu().numpy()
        assert np.array_equal(got[:k // 2], np.nonzero(bits)[0][:k // 2]) and (got[k // 2:] == -7).all()
