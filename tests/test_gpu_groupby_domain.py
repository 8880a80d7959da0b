"""GROUP BY of dense keys around the 2048 values up to which a key's place in its
range is its slot in the CTA table: one to two tiles, with and without WHERE columns,
NULL keys and values and rows that the WHERE leaves out (lanes without a slot), keys
that repeat within a warp.  Keys, counts, MIN and MAX exactly, SUM within 1e-12
relative of the serial sum (all values are positive)."""
import numpy as np
import pytest
import torch

import falcondb_b200 as F
from falcondb_b200 import ops
from tests.test_gpu_groupby_merge import words
from tests.test_gpu_groupby_parts import reference

pytestmark = pytest.mark.gpu
I64MIN = np.iinfo(np.int64).min


@pytest.mark.parametrize("domain", [1, 2, 40, 2047, 2048, 2049])
@pytest.mark.parametrize("where", [0, 1, 2])
@pytest.mark.parametrize("nulls", [False, True])
@pytest.mark.parametrize("n", [1, 1023, 70_003])
@pytest.mark.parametrize("skewed", [False, True])
def test_dense_domains(db, domain, where, nulls, n, skewed):
    r = np.random.default_rng([domain, where, nulls, n, skewed])
    key = -1000 + (domain ** r.random(n) - 1 if skewed else r.integers(0, domain, n)).astype(np.int64)
    key[0] = -1000
    key[-1] = -1000 + domain - 1
    v, a, b = r.random(n) + 0.5, r.integers(0, 100, n), r.random(n)
    ones = np.ones(n, bool)
    kok, vok = (r.random(n) < 0.8, r.random(n) < 0.7) if nulls else (ones, ones)
    if nulls:
        key[r.random(n) < 0.05] = I64MIN
        kok[0] = kok[-1] = True
    keep = ones
    prog, cols = [], []
    if where:
        prog, cols = [ops.cmp(0, F.LT, 60)], [torch.from_numpy(a).cuda()]
        keep = a < 60
    if where == 2:
        prog, cols = prog + [ops.cmp(1, F.GT, 0.2), ops.AND()], cols + [torch.from_numpy(b).cuda()]
        keep = keep & (b > 0.2)
    dk, dv = torch.from_numpy(key).cuda(), torch.from_numpy(v).cuda()
    out, ng = ops.group_by_i64(db, (dk, words(kok)) if nulls else dk, (dv, words(vok)) if nulls else dv, n, prog, cols)
    db.synchronize()
    rec = ops.to_records(out, F.GROUP_I64_DTYPE, int(ng.item()))
    rec = np.sort(rec, order="key")
    want = reference(key[keep], v[keep], kok[keep], vok[keep])
    assert np.array_equal(rec["key"], want[0]) and np.array_equal(rec["count"], want[1])
    assert np.array_equal(rec["min"], want[3], equal_nan=True) and np.array_equal(rec["max"], want[4], equal_nan=True)
    assert (np.abs(rec["sum"] - want[2]) <= 1e-12 * np.abs(want[2])).all()
