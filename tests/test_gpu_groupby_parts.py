"""GROUP BY scattered int64 keys on both sides of the lines where the hash
partitions take over (2^20 rows, 64 groups per partition, two tables' worth of
them, one partition's share of the rows), with NULL keys and values, against a
sorted numpy aggregation: keys, counts, MIN and MAX exactly, SUM within 1e-12
relative of the serial sum (all values positive)."""
import numpy as np
import pytest
import torch

import falcondb_b200 as F
from falcondb_b200 import ops

pytestmark = pytest.mark.gpu
MIX = np.int64(-7046029254386353131)


def reference(key, v, kok, vok):
    """Records by ascending key; NULL keys (and INT64_MIN) form the group INT64_MIN."""
    key = np.where(kok, key, np.iinfo(np.int64).min)
    uniq, inv, count = np.unique(key, return_inverse=True, return_counts=True)
    m = len(uniq)
    num = vok & ~np.isnan(v)
    total = np.bincount(inv[vok], weights=v[vok], minlength=m)
    low = np.full(m, np.inf)
    high = np.full(m, -np.inf)
    np.minimum.at(low, inv[num], v[num])
    np.maximum.at(high, inv[num], v[num])
    none = np.bincount(inv[num], minlength=m) == 0
    low[none] = high[none] = np.nan
    return uniq, count, total, low, high


def check(db, key, v, kok=None, vok=None):
    n = len(key)
    ones = np.ones(n, bool)
    dk, dv = torch.from_numpy(key).cuda(), torch.from_numpy(v).cuda()
    words = lambda ok: torch.from_numpy(F.validity_words(ok).view(np.int64)).cuda()  # noqa: E731
    out, ng = ops.group_by_i64(db, dk if kok is None else (dk, words(kok)), dv if vok is None else (dv, words(vok)), n)
    db.synchronize()
    rec = np.sort(ops.to_records(out, F.GROUP_I64_DTYPE, int(ng.item())), order="key")
    want = reference(key, v.astype(np.float64), ones if kok is None else kok, ones if vok is None else vok)
    assert np.array_equal(rec["key"], want[0]) and np.array_equal(rec["count"], want[1])
    assert np.array_equal(rec["min"], want[3], equal_nan=True) and np.array_equal(rec["max"], want[4], equal_nan=True)
    fine = np.isfinite(want[2])
    assert np.array_equal(rec["sum"][~fine], want[2][~fine], equal_nan=True)
    assert (np.abs(rec["sum"][fine] - want[2][fine]) <= 1e-12 * np.abs(want[2][fine])).all()


@pytest.mark.parametrize("n,groups", [((1 << 20) - 1, 100_000), (1 << 20, 100_000), (1_200_001, 20_000),
                                      (1_200_001, 40_000), (2_500_003, 1_300_000), (4_000_001, 2_400_000),
                                      (4_000_001, 3_900_000)])
def test_group_counts(db, n, groups):
    r = np.random.default_rng(groups)
    check(db, r.integers(0, groups, n) * MIX, r.random(n) + 0.5)


@pytest.mark.parametrize("nulls", ["keys", "values", "both"])
def test_nulls(db, nulls):
    n = 1_500_007
    r = np.random.default_rng(5)
    key, v = r.integers(0, 60_000, n) * MIX, r.random(n) + 0.5
    key[r.random(n) < 1e-3] = np.iinfo(np.int64).min  # reads as NULL
    kok = r.random(n) < 0.9 if nulls != "values" else None
    vok = (r.random(n) < 0.5) & (key % 7 != 0) if nulls != "keys" else None  # some groups hold no value
    check(db, key, v, kok, vok)


def test_special_values(db):
    """NaN with any bits, also those a NULL travels as, is a value: SUM is NaN,
    MIN / MAX pass over it; infinities take part."""
    n = 1_300_000
    r = np.random.default_rng(6)
    key, v = r.integers(0, 50_000, n) * MIX, r.random(n) + 0.5
    bits = v.view(np.uint64)
    bits[r.random(n) < 0.01] = 0x7FF4DEADBEEF0001
    bits[r.random(n) < 0.01] = 0xFFF8000000000000
    v[r.random(n) < 0.01] = np.inf
    check(db, key, v)


def test_int_values_and_skew(db):
    n = 1_400_000
    r = np.random.default_rng(7)
    key = r.integers(0, 50_000, n) * MIX
    check(db, key, r.integers(1, 10**12, n))
    key[r.random(n) < 0.1] = MIX  # one frequent key: its partition is far above its share
    check(db, key, r.integers(1, 10**6, n))


def test_within_a_small_budget():
    """A budget without room for the partitions: the hashed table, as before."""
    n = 2_000_000
    r = np.random.default_rng(8)
    with F.Database(0, mem_budget=130 << 20) as small:
        check(small, r.integers(0, 50_000, n) * MIX, r.random(n) + 0.5)
        small.synchronize()
        assert small.memory_stats()["in_use"] < 130 << 20


def test_capacity(db):
    n = 1_200_000
    r = np.random.default_rng(9)
    key, v = torch.from_numpy(r.integers(0, 50_000, n) * MIX).cuda(), torch.from_numpy(r.random(n)).cuda()
    ops.group_by_i64(db, key, v, n, capacity=40_000)
    with pytest.raises(F.FalconError):
        db.synchronize()
    out, ng = ops.group_by_i64(db, key, v, n)
    db.synchronize()
    assert int(ng.item()) == 50_000
