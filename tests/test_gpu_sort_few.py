"""Sorts of few values by the radix passes, around the 65,536 rows up to which one CTA
scans a pass's counts, each after a sort of another size and kind.  All orders exact."""
import numpy as np
import pytest
import torch

from falcondb_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4097, 61_441, 65_535, 65_536, 65_537, 131_073, 420_001])
@pytest.mark.parametrize("values", [1, 12, 70_000])
def test_few_values(db, n, values):
    r = np.random.default_rng([n, values])
    v = r.integers(0, values, n) * 3 - 5
    u = r.random(n + 300_000)
    d, du = torch.from_numpy(v).cuda(), torch.from_numpy(u).cuda()
    for desc in (False, True):
        got = ops.sort(db, d, n, desc)[:n].cpu().numpy()
        assert np.array_equal(got, np.argsort(-v if desc else v, kind="stable"))
        m = len(u) if desc else n
        got = ops.sort(db, du, m, False)[:m].cpu().numpy()
        assert np.array_equal(got, np.argsort(u[:m], kind="stable"))
    _, first = np.unique(v, return_index=True)
    rows, cnt = ops.distinct(db, d, n)
    assert np.array_equal(rows[:int(cnt.item())].cpu().numpy(), np.sort(first))
