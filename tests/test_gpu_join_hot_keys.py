"""Join builds whose warps hold rows of one key: a single key, one that most rows
have, few keys, runs of a key across warp edges, with NULL keys, NULL payloads and
the key INT64_MIN among them.  Counts, sums and pairs are exact."""
import numpy as np
import pytest
import torch

import falcondb_b200 as F
from falcondb_b200 import ops

pytestmark = pytest.mark.gpu

INNER, LEFT = 0, 1
I64MIN = np.iinfo(np.int64).min


def keys_of(kind, n, r):
    if kind == "one":
        return np.full(n, 42)
    if kind == "most":
        return np.where(r.random(n) < 0.9, 42, r.integers(0, n, n) * 7919)
    if kind == "few":
        return r.integers(0, 5, n) * 7919
    if kind == "runs":
        return np.arange(n) // 45 * 7919
    k = r.integers(0, 40, n)
    k[r.random(n) < 0.3] = I64MIN
    return k


@pytest.mark.parametrize("n", [1, 31, 33, 1000, 70_001])
@pytest.mark.parametrize("kind", ["one", "most", "few", "runs", "min"])
@pytest.mark.parametrize("nulls", [False, True])
def test_hot_build_keys(db, n, kind, nulls):
    r = np.random.default_rng([n, len(kind)])
    k, p = keys_of(kind, n, r).astype(np.int64), r.integers(-10**12, 10**12, n)
    kv = r.random(n) < (0.9 if nulls else 2.0)
    pv = r.random(n) < (0.8 if nulls else 2.0)
    words = lambda ok: torch.from_numpy(F.validity_words(ok).view(np.int64)).cuda()
    col = lambda v, ok: (torch.from_numpy(v).cuda(), words(ok)) if nulls else torch.from_numpy(v).cuda()
    ht = ops.HashTable(db, col(k, kv), col(p, pv), n)
    probe = np.concatenate([np.unique(k), [42, 7, I64MIN, 7919 * 3]]).astype(np.int64)
    rows = {int(x): np.nonzero(kv & (k == x))[0] for x in np.unique(probe)}
    d = torch.from_numpy(probe).cuda()
    for jt in (INNER, LEFT):
        got = ops.to_records(ht.probe_agg(d, len(probe), jt), F.JOIN_AGG_DTYPE)[0]
        m = [rows[int(x)] for x in probe]
        assert got["count"] == sum(len(x) if jt == INNER else max(1, len(x)) for x in m)
        assert got["sum_payload"] == sum(int(p[x[pv[x]]].sum()) for x in m)
        assert got["payload_rows"] == sum(int(pv[x].sum()) for x in m)
    want = [(i, int(x)) for i, key in enumerate(probe) for x in rows[int(key)]]
    left, right, cnt = ht.probe_pairs(d, len(probe), INNER, len(want) + 8)
    c = int(cnt.item())
    assert sorted(zip(left[:c].tolist(), right[:c].tolist())) == want
    ht.free()
