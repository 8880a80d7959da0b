"""Sample sorts some of whose leaves hold more pairs than their region: values of a
few thousand rows, or clusters of close ones, too small for the sample to see.
Their pairs are spilled and sorted apart; more of them than the spill list takes
(one in 16) leave the whole sort to the radix passes.  All orders are exact."""
import numpy as np
import pytest
import torch

import falcondb_b200 as F
from falcondb_b200 import ops

pytestmark = pytest.mark.gpu


def kernels(f):
    """The names of the kernels that f launches."""
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        f()
        torch.cuda.synchronize()
    return {e.name for e in prof.events()}


def launched(names, kernel):
    return any(kernel in x for x in names)


def clusters(n, count, size, close, seed):
    """Uniform values with `count` clusters of `size` rows: each one value, or
    distinct values too close for any step of a map."""
    r = np.random.default_rng(seed)
    v = r.random(n)
    at = r.permutation(n)[:count * size].reshape(count, size)
    for j, x in enumerate(at):
        v[x] = (j + 0.37) / count
        if close:
            v[x] += r.permutation(size) * 2.0**-52
    return v


def order_key(v):
    b = v.view(torch.int64)
    return torch.where(b < 0, ~b ^ torch.iinfo(torch.int64).min, b)


def check_order(db, v, desc):
    d = torch.from_numpy(v).cuda()
    k = order_key(d)
    want = torch.sort(~k if desc else k, stable=True).indices
    got = ops.sort(db, d, len(v), desc).to(torch.int64) & 0xFFFFFFFF
    assert bool((got == want).all())


# (rows, clusters, their rows): a leaf's region holds 3392 pairs in sorts of 20M
# rows and 3968 in sorts of 6M, so the last one's clusters may fit.
SPILLED = [(20_000_003, 5, 6000), (20_000_003, 60, 4000), (6_000_000, 1, 5000), (6_000_000, 20, 4500)]
CLUSTERS = SPILLED + [(6_000_000, 20, 3500)]


@pytest.mark.parametrize("n,count,size", CLUSTERS)
@pytest.mark.parametrize("close", [False, True])
@pytest.mark.parametrize("desc", [False, True])
def test_clusters(db, n, count, size, close, desc):
    check_order(db, clusters(n, count, size, close, [n, count]), desc)


@pytest.mark.parametrize("n,count,size", SPILLED)
def test_close_clusters_are_spilled(db, n, count, size):
    d = torch.from_numpy(clusters(n, count, size, True, [n, count])).cuda()
    names = kernels(lambda: ops.sort(db, d, n, False))
    assert launched(names, "msd_over_write_kernel")


@pytest.mark.parametrize("count,size", [(400, 4000), (250, 12_000)])
@pytest.mark.parametrize("close", [False, True])
def test_more_than_the_list_takes(db, count, size, close):
    n = 20_000_000
    v = clusters(n, count, size, close, count)
    d = torch.from_numpy(v).cuda()
    names = kernels(lambda: ops.sort(db, d, n, False))
    assert launched(names, "radix_scatter_kernel") and not launched(names, "msd_over_write_kernel")
    check_order(db, v, False)


@pytest.mark.parametrize("n,count,size", SPILLED)
@pytest.mark.parametrize("close", [False, True])
def test_distinct(db, n, count, size, close):
    v = clusters(n, count, size, close, [n, count, 7])
    r = np.random.default_rng(n)
    v[r.random(n) < 0.2] *= -1.0
    _, first = np.unique(v, return_index=True)
    rows, cnt = ops.distinct(db, torch.from_numpy(v).cuda(), n)
    assert np.array_equal(rows[:int(cnt.item())].cpu().numpy().view(np.uint32), np.sort(first))


def test_nulls_and_integers(db):
    """A row list before the sort, and INT64 keys with clusters at both ends of the range."""
    n = 8_000_000
    r = np.random.default_rng(11)
    v = r.integers(-2**62, 2**62, n)
    at = r.permutation(n)[:20_000].reshape(4, 5000)
    for j, x in enumerate((-2**63, -2**63 + 1, 2**63 - 1, 0)):
        v[at[j]] = x
    ok = r.random(n) < 0.95
    w = torch.from_numpy(F.validity_words(ok).view(np.int64)).cuda()
    order = np.argsort(v, kind="stable")
    got = ops.sort(db, (torch.from_numpy(v).cuda(), w), n, False, True).cpu().numpy().view(np.uint32)
    assert np.array_equal(got, np.concatenate([order[ok[order]], np.nonzero(~ok)[0]]))
