"""Merging a warp's rows ahead of the CTA table, alone and batched: from one key
to none twice in a warp, NULL groups, NULL, NaN and infinite values, and counts
that leave warps and tiles part empty.  Keys, counts, MIN and MAX exactly, SUM
within 1e-12 relative of the serial sum (the finite values are positive)."""
import numpy as np
import pytest
import torch

import falcondb_b200 as F
from falcondb_b200 import ops
from tests.test_gpu_groupby_parts import MIX, reference

pytestmark = pytest.mark.gpu


def words(ok):
    return torch.from_numpy(F.validity_words(ok).view(np.int64)).cuda()


@pytest.mark.parametrize("batched", [False, True])
@pytest.mark.parametrize("n", [1, 31, 33, 4097, 300_007])
@pytest.mark.parametrize("kind", ["one", "two", "skewed", "spread", "null_keys", "special", "int"])
def test_merged_rows(db, batched, n, kind):
    r = np.random.default_rng([n, len(kind)])
    groups = {"one": 1, "two": 2, "spread": 5000}.get(kind, 40)
    key = np.minimum(r.integers(0, groups, n), r.integers(0, groups, n)) * MIX
    v = r.random(n) + 0.5
    kok = vok = np.ones(n, bool)
    if kind == "skewed":
        key[r.random(n) < 0.5] = 7
    elif kind == "null_keys":
        kok, vok = r.random(n) < 0.3, r.random(n) < 0.5
    elif kind == "special":
        for x, share in ((np.nan, 0.02), (np.inf, 0.01), (-0.0, 0.3)):
            v[r.random(n) < share] = x
    elif kind == "int":
        v = r.integers(1, 2**40, n)
    dk, dv = torch.from_numpy(key).cuda(), torch.from_numpy(v).cuda()
    cols = (dk, dv) if kind != "null_keys" else ((dk, words(kok)), (dv, words(vok)))
    if batched:
        b = ops.GroupByBatch(db, [(*cols, n)])
        b.run()
        db.synchronize()
        rec = np.sort(b.results(0), order="key")
        b.free()
    else:
        out, ng = ops.group_by_i64(db, *cols, n)
        db.synchronize()
        rec = np.sort(ops.to_records(out, F.GROUP_I64_DTYPE, int(ng.item())), order="key")
    want = reference(key, v.astype(np.float64), kok, vok)
    assert np.array_equal(rec["key"], want[0]) and np.array_equal(rec["count"], want[1])
    assert np.array_equal(rec["min"], want[3], equal_nan=True) and np.array_equal(rec["max"], want[4], equal_nan=True)
    fine = np.isfinite(want[2])
    assert np.array_equal(rec["sum"][~fine], want[2][~fine], equal_nan=True)
    assert (np.abs(rec["sum"][fine] - want[2][fine]) <= 1e-12 * np.abs(want[2][fine])).all()
