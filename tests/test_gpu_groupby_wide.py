"""GROUP BY of dense keys around the 2^22 key values from which the CTAs take tiles
half as large.  Keys, counts, MIN and MAX exactly, SUM (integers) exactly."""
import numpy as np
import pytest
import torch

import falcondb_b200 as F
from falcondb_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("domain", [(1 << 22) - 1, 1 << 22, (1 << 22) + 1])
def test_wide_domains(db, domain):
    r = np.random.default_rng(domain)
    n = 3_000_001
    key = r.integers(0, domain, n)
    key[:100_000] = r.integers(0, 50, 100_000)
    key[0], key[-1] = 0, domain - 1
    v = r.integers(-1000, 1000, n)
    out, ng = ops.group_by_i64(db, torch.from_numpy(key).cuda(), torch.from_numpy(v).cuda(), n)
    db.synchronize()
    rec = ops.to_records(out, F.GROUP_I64_DTYPE, int(ng.item()))
    uniq, inv, count = np.unique(key, return_inverse=True, return_counts=True)
    order = np.argsort(inv, kind="stable")
    start = np.concatenate([[0], np.cumsum(count)[:-1]])
    s = v[order]
    assert np.array_equal(rec["key"], uniq) and np.array_equal(rec["count"], count)  # in key order
    assert np.array_equal(rec["sum"], np.add.reduceat(s, start))
    assert np.array_equal(rec["min"], np.minimum.reduceat(s, start))
    assert np.array_equal(rec["max"], np.maximum.reduceat(s, start))
