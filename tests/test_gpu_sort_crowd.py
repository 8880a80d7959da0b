"""Sorts of at most one leaf whose keys crowd into few of its slots: the stable
counting sort (a range of keys below 2^36) and the bitonic network above it.
All orders are exact."""
import numpy as np
import pytest
import torch

from falcondb_b200 import ops

pytestmark = pytest.mark.gpu

SIZES = [40, 511, 512, 513, 2049, 3000, 3967, 3968]


def column(kind, n, r):
    if kind == "twelve":
        return r.integers(0, 12, n)
    if kind == "one":
        return np.full(n, -7)
    if kind == "around zero":  # both high halves of the key
        return r.integers(-5, 6, n)
    if kind == "hot":  # nine in ten rows of one value, the others spread
        return np.where(r.random(n) < 0.9, 3, r.integers(0, 1 << 20, n))
    if kind.startswith("range"):  # few values and both ends of [0, 2^bits)
        bits = int(kind.split()[1])
        v = (r.integers(0, 7, n) * (2**bits // 7)) ^ r.integers(0, 2, n)
        v[0], v[-1] = 0, 2**bits - 1
        return r.permutation(v)
    if kind == "ends":
        return np.where(r.random(n) < 0.5, np.iinfo(np.int64).min + 1, np.iinfo(np.int64).max)
    assert kind == "floats"
    return r.choice(np.array([-np.inf, -1.5, -0.0, 0.0, 0.25, 5.0, np.inf, np.nan]), n)


KINDS = ["twelve", "one", "around zero", "hot", "range 11", "range 12", "range 13", "range 24", "range 25", "range 36",
         "range 37", "range 62", "ends", "floats"]


def order_key(v):
    u = v.view(np.uint64)
    if v.dtype == np.float64:
        return np.where(u >> 63 == 1, ~u, u | np.uint64(1 << 63))
    return u ^ np.uint64(1 << 63)


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("kind", KINDS)
def test_crowded_keys(db, n, kind):
    v = column(kind, n, np.random.default_rng([n, KINDS.index(kind)]))
    d, k = torch.from_numpy(v).cuda(), order_key(v)
    for desc in (False, True):
        got = ops.sort(db, d, n, desc)[:n].cpu().numpy()
        assert np.array_equal(got, np.argsort(~k if desc else k, kind="stable")), desc
    u = np.where(np.isnan(v), 1e300, v + 0.0) if v.dtype == np.float64 else v
    _, first = np.unique(u, return_index=True)
    rows, cnt = ops.distinct(db, d, n)
    assert np.array_equal(rows[:int(cnt.item())].cpu().numpy(), np.sort(first))
