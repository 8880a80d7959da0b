"""Working memory that a call can do without is given back when the call ends:
what the memory budget admitted before a sample sort or a partitioned GROUP BY
it still admits after one."""
import numpy as np
import pytest
import torch

import falcondb_b200 as F
from falcondb_b200 import ops

pytestmark = pytest.mark.gpu

MIB = 1 << 20
SORT_ROWS = 1_200_000  # the sample sort takes about 75 MiB, the radix passes 32


def sorted_rows(db, n, seed=1):
    v = np.random.default_rng(seed).random(n)
    got = ops.sort(db, torch.from_numpy(v).cuda(), n, False)[:n].cpu().numpy()
    assert np.array_equal(got, np.argsort(v, kind="stable"))


def table(mib):
    return {"x": np.zeros(mib * MIB // 8)}


def test_nothing_is_held_after_a_sort_or_a_group_by():
    with F.Database(0, mem_budget=2048 * MIB) as db:
        held = db.memory_stats()["in_use"]
        sorted_rows(db, SORT_ROWS)
        db.synchronize()
        assert db.memory_stats()["in_use"] == held
        n = 8_000_000  # 128 MB of partitioned rows
        k = torch.randint(0, 500_000, (n,), dtype=torch.int64, device="cuda") * -7046029254386353131
        out, cnt = ops.group_by_i64(db, k, torch.ones(n, dtype=torch.float64, device="cuda"), n)
        g = ops.to_records(out, F.GROUP_I64_DTYPE, int(cnt.item()))
        assert len(g) == len(torch.unique(k)) and int(g["count"].sum()) == n
        db.synchronize()
        # The arena itself may have grown for the sizing pass, not for the rows.
        assert db.memory_stats()["in_use"] < held + 64 * MIB


def test_a_table_that_fitted_before_a_sort_fits_after_it():
    with F.Database(0, mem_budget=400 * MIB) as db:
        sorted_rows(db, SORT_ROWS)
        assert db.create_table("t", table(330)) == 330 * MIB // 8


def test_an_arena_that_fitted_before_a_sort_fits_after_it():
    with F.Database(0, mem_budget=400 * MIB) as db:
        sorted_rows(db, SORT_ROWS)
        db.create_table("t", table(255))
        sorted_rows(db, 5_500_000, 2)  # radix passes: 135 MiB of arena
        db.synchronize()
        assert db.memory_stats()["in_use"] < 400 * MIB


def test_nested_scratch_of_a_nullable_distinct():
    """DISTINCT takes its row mask, the NULL split and the sort from one spare arena."""
    n = 1_500_000
    r = np.random.default_rng(3)
    v, ok = r.random(n), r.random(n) < 0.9
    w = torch.from_numpy(F.validity_words(ok).view(np.int64)).cuda()
    with F.Database(0, mem_budget=1024 * MIB) as db:
        held = db.memory_stats()["in_use"]
        rows, cnt = ops.distinct(db, (torch.from_numpy(v).cuda(), w), n)
        want = np.sort(np.concatenate([np.nonzero(ok)[0], np.nonzero(~ok)[0][:1]]))
        assert np.array_equal(rows[:int(cnt.item())].cpu().numpy(), want)
        db.synchronize()
        assert db.memory_stats()["in_use"] == held
