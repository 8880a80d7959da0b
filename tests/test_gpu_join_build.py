"""The join build's two layouts (one row per key, and row lists when keys
repeat), hashed and dense, with NULL keys, NULL payloads and the key INT64_MIN,
against the oracle.  Counts, integer sums and row pairs are exact."""
import numpy as np
import pytest
import torch

import falcondb_b200 as F
from falcondb_b200 import ops
from oracle import oracle as O

pytestmark = pytest.mark.gpu
MIN = np.iinfo(np.int64).min


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("nulls", [False, True])
@pytest.mark.parametrize("kind", ["unique", "one_repeat", "min_repeats", "repeats", "one_key"])
@pytest.mark.parametrize("nb,step", [(1, 1), (255, 7919), (1025, 1), (150_001, 1), (150_001, 7919)])
def test_build_layouts(db, nb, step, kind, nulls):
    r = np.random.default_rng(nb + step)
    bk = r.permutation(nb).astype(np.int64) * step - 1000
    if kind == "one_repeat":
        bk[-1] = bk[0]
    elif kind == "min_repeats":
        bk[::max(1, nb // 3)] = MIN
    elif kind == "repeats":
        bk = bk[r.integers(0, max(1, nb // 5), nb)]
    elif kind == "one_key":
        bk[:] = bk[0]
    if kind != "min_repeats" and nb > 100:
        bk[nb // 2] = MIN
    pay = r.integers(-10**12, 10**12, nb)
    bv = pv = None
    if nulls:
        bv, pv = (F.validity_words(r.random(nb) > 0.2) for _ in range(2))
    pk = np.concatenate([r.choice(bk, 4000), r.integers(-2000, nb * step + 2000, 1000), [MIN, MIN + 1]]).astype(np.int64)
    key = (dev(bk), dev(bv.view(np.int64))) if nulls else dev(bk)
    val = (dev(pay), dev(pv.view(np.int64))) if nulls else dev(pay)
    h = ops.HashTable(db, key, val, nb)
    pval = np.zeros(len(pk))
    for jt in (F.JOIN_INNER, F.JOIN_LEFT, F.JOIN_SEMI, F.JOIN_ANTI):
        got = ops.to_records(h.probe_agg(dev(pk), len(pk), jt), F.JOIN_AGG_DTYPE, 1)[0]
        want = O.join_agg(bk, pay, pk, pval, jt, bvalid=bv, bpvalid=pv)
        assert got["count"] == want["count"], jt
        if jt <= 1:
            assert got["sum_payload"] == want["sum_payload"], jt
            assert got["payload_rows"] == want["payload_rows"], jt
    few = pk[-1202:] if kind != "one_key" else pk[-3:]
    want_l, want_r = O.join_pairs(bk, few, F.JOIN_LEFT, bvalid=bv)
    left, right, cnt = h.probe_pairs(dev(few), len(few), F.JOIN_LEFT, capacity=len(want_l) + 1)
    h.free()
    c = int(cnt.item())
    assert c == len(want_l)
    got = sorted(zip(left[:c].cpu().numpy().view(np.uint32).tolist(), right[:c].cpu().numpy().view(np.uint32).tolist()))
    assert got == sorted(zip(want_l.tolist(), want_r.tolist()))
