"""ORDER BY and DISTINCT at the edges of the sample sort's levels (one CTA up to
3968 pairs, one level of buckets up to 409,600, two above) over key
distributions that fill, crowd and overflow its buckets, against a stable numpy
sort of the order keys."""
import numpy as np
import pytest
import torch

import falcondb_b200 as F
from falcondb_b200 import ops

pytestmark = pytest.mark.gpu
SIZES = [1, 2, 33, 2048, 2049, 3968, 3969, 4096, 4097, 65_536, 409_600, 409_601, 819_201, 3_000_017]


def order_key(v):
    if v.dtype == np.float64:
        b = v.view(np.uint64)
        return np.where(b >> np.uint64(63), ~b, b | np.uint64(1 << 63))
    return v.view(np.uint64) ^ np.uint64(1 << 63)


def column(kind, n, r):
    if kind == "uniform":
        return r.random(n) * 100.0
    if kind == "spread":  # every exponent, both signs, and the values without one
        v = np.ldexp(r.random(n) + 0.5, r.integers(-1070, 1020, n)) * r.choice([-1.0, 1.0], n)
        v[r.random(n) < 1e-3] = np.nan
        v[r.random(n) < 1e-3] = -np.inf
        v[r.random(n) < 1e-3] = -0.0
        return v
    if kind == "ascending":
        return np.arange(n, dtype=np.int64) - n // 2
    if kind == "descending":
        return (2**33 - np.arange(n, dtype=np.int64)) * 3
    if kind == "wide":
        return r.integers(-2**63, 2**63 - 1, n, dtype=np.int64)
    if kind == "clustered":  # a few narrow clusters far apart: slots crowd
        return r.choice(np.array([-2**62, -5, 0, 2**31 - 300, 2**32, 2**61], dtype=np.int64), n) + r.integers(0, n + 1, n)
    if kind == "repeats":  # about 200 rows per key
        return r.integers(0, max(1, n // 200), n)
    if kind == "heavy":  # half the rows hold one key
        v = r.integers(0, 2**40, n)
        v[r.random(n) < 0.5] = 2**39
        return v
    assert kind == "equal"
    return np.full(n, 7, np.int64)


KINDS = ["uniform", "spread", "ascending", "descending", "wide", "clustered", "repeats", "heavy", "equal"]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("kind", KINDS)
def test_sort_levels(db, n, kind):
    r = np.random.default_rng([n, KINDS.index(kind)])
    v = column(kind, n, r)
    k = order_key(v)
    d = torch.from_numpy(v).cuda()
    for desc in (False, True):
        want = np.argsort(~k if desc else k, kind="stable")
        got = ops.sort(db, d, n, desc)[:n].cpu().numpy()
        assert np.array_equal(got, want), (kind, n, desc)
    u = np.where(np.isnan(v), np.nan, v + 0.0) if v.dtype == np.float64 else v
    keys = u.view(np.uint64).copy()
    if v.dtype == np.float64:
        keys[np.isnan(v)] = 1  # one NaN
    _, first = np.unique(keys, return_index=True)
    rows, cnt = ops.distinct(db, d, n)
    m = int(cnt.item())
    assert np.array_equal(rows[:m].cpu().numpy(), np.sort(first))


@pytest.mark.parametrize("n", [100, 5000, 1_000_003])
@pytest.mark.parametrize("share", [0.01, 0.999])
def test_sort_levels_with_nulls(db, n, share):
    r = np.random.default_rng(n)
    v, ok = r.random(n), r.random(n) < share
    w = torch.from_numpy(F.validity_words(ok).view(np.int64)).cuda()
    order = np.argsort(v, kind="stable")
    order, null = order[ok[order]], np.nonzero(~ok)[0]
    for nulls_last in (False, True):
        got = ops.sort(db, (torch.from_numpy(v).cuda(), w), n, False, nulls_last)[:n].cpu().numpy()
        assert np.array_equal(got, np.concatenate([order, null] if nulls_last else [null, order]))
    rows, cnt = ops.distinct(db, (torch.from_numpy(v).cuda(), w), n)
    want = np.sort(np.concatenate([np.nonzero(ok)[0], null[:1]]))
    assert np.array_equal(rows[:int(cnt.item())].cpu().numpy(), want)


def test_unsampled_heavy_keys_overflow(db):
    """Keys of 3000 rows among 20M are mostly missed by 16384 samples, and their
    leaves overflow: the radix passes must take over with the same answer."""
    n = 20_000_000
    r = np.random.default_rng(3)
    v = r.random(n)
    rows = r.permutation(n)[:30_000].reshape(10, 3000)
    for j, x in enumerate(rows):
        v[x] = 0.05 + j / 10
    got = ops.sort(db, torch.from_numpy(v).cuda(), n, False)[:n].cpu().numpy()
    assert np.array_equal(got, np.argsort(v, kind="stable"))


def test_sort_within_a_small_budget():
    """A context whose budget leaves no room for the sample sort's buckets sorts
    by radix passes, as before."""
    n = 2_000_000
    v = np.random.default_rng(4).random(n)
    with F.Database(0, mem_budget=200 << 20) as small:
        got = ops.sort(small, torch.from_numpy(v).cuda(), n, True)[:n].cpu().numpy()
        assert np.array_equal(got, np.argsort(-v, kind="stable"))
        small.synchronize()
        assert small.memory_stats()["in_use"] < 160 << 20


@pytest.mark.parametrize("n", [13_107_200, 13_107_201])
@pytest.mark.parametrize("kind", ["uniform", "spread"])
def test_sort_around_the_larger_sample(db, n, kind):
    """From 64 second-level buckets on the first level's map has twice the samples."""
    v = torch.from_numpy(column(kind, n, np.random.default_rng(n))).cuda()
    got = ops.sort(db, v, n, False, nulls_last=False).to(torch.int64) & 0xFFFFFFFF
    bits = v.view(torch.int64)
    key = torch.where(bits < 0, ~bits ^ torch.iinfo(torch.int64).min, bits)
    assert bool((got == torch.sort(key, stable=True).indices).all())
