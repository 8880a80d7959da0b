"""Which GROUP BYs of scattered int64 keys the hash partitions take: their counts
are made only without a WHERE, and where a look at 512 keys finds many values and
no long runs.  Kernels launched, and every result against a numpy aggregation."""
import numpy as np
import pytest
import torch

import falcondb_b200 as F
from falcondb_b200 import ops
from tests.test_gpu_groupby_merge import words
from tests.test_gpu_groupby_parts import MIX, check
from tests.test_gpu_sort_spill import kernels, launched

pytestmark = pytest.mark.gpu


def column(kind, r):
    """Keys, and which are valid (None: all)."""
    if kind == "uniform":
        return r.integers(0, 60_000, 1_500_001) * MIX, None
    if kind == "nullable":  # NULLs store zeros
        ok = r.random(1_500_001) < 0.4
        return np.where(ok, r.integers(0, 60_000, len(ok)) * MIX, 0), ok
    if kind == "sparse":
        return r.integers(0, 60_000, 1_500_001) * 19 + 5, None
    if kind == "outlier":  # a range that one value spoils
        k = r.integers(0, 60_000, 1_500_001)
        k[777] = 2**50
        return k, None
    if kind == "short runs":
        return np.sort(r.integers(0, 150_000, 1_500_001) * MIX), None
    if kind == "few":
        return r.integers(0, 1000, 1_500_001) * MIX, None
    if kind == "skewed":
        return (400_000 ** r.random(1_500_001)).astype(np.int64) * MIX, None
    if kind == "long runs":
        return np.sort(r.integers(0, 40_000, 4_000_001) * MIX), None
    if kind == "all null":
        return r.integers(0, 60_000, 1_500_001) * MIX, np.zeros(1_500_001, bool)
    assert kind == "dense"
    return r.integers(0, 60_000, 1_500_001), None


# The estimate of the groups takes in what NULL rows store, so "all null" is taken too.
TAKEN = ["uniform", "nullable", "sparse", "outlier", "short runs", "all null"]
OTHERS = ["few", "skewed", "long runs", "dense"]


@pytest.mark.parametrize("kind", TAKEN + OTHERS)
def test_route(db, kind):
    r = np.random.default_rng(len(kind))
    key, kok = column(kind, r)
    v = r.random(len(key)) + 0.5
    check(db, key, v, kok)
    dk, dv = torch.from_numpy(key).cuda(), torch.from_numpy(v).cuda()
    if kok is not None:
        dk = (dk, words(kok))
    assert launched(kernels(lambda: ops.group_by_i64(db, dk, dv, len(v))), "gb_part_agg_kernel") == (kind in TAKEN)
    where = [ops.cmp(0, F.LT, 2.0)]  # every row
    assert not launched(kernels(lambda: ops.group_by_i64(db, dk, dv, len(v), where, [dv])), "gb_part_agg_kernel")


def test_an_unaligned_column(db):
    """Keys whose first lies 8 bytes past a 16-byte boundary."""
    r = np.random.default_rng(3)
    n = 1_300_002
    key, v = r.integers(0, 50_000, n) * MIX, r.random(n) + 0.5
    dk, dv = torch.from_numpy(key).cuda()[1:], torch.from_numpy(v).cuda()[1:]
    out, ng = ops.group_by_i64(db, dk, dv, n - 1)
    db.synchronize()
    rec = np.sort(ops.to_records(out, F.GROUP_I64_DTYPE, int(ng.item())), order="key")
    uniq, count = np.unique(key[1:], return_counts=True)
    assert np.array_equal(rec["key"], uniq) and np.array_equal(rec["count"], count)
    assert launched(kernels(lambda: ops.group_by_i64(db, dk, dv, n - 1)), "gb_part_agg_kernel")
