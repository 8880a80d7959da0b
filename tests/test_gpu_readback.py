"""Query results around the size of the context's page-locked read-back buffer
(64 KB, 8192 values): a column below, at and above it, with its NULLs, and more
results in one wait than it keeps places for.  All are exact."""
import threading

import numpy as np
import pytest

import falcondb_b200 as F

pytestmark = pytest.mark.gpu


def table(n, seed):
    r = np.random.default_rng(seed)
    x = np.ma.masked_array(r.integers(-10**15, 10**15, n), mask=r.random(n) < 0.25)
    return {"id": np.arange(n, dtype=np.int64), "x": x}


@pytest.mark.parametrize("n", [1, 8000, 8191, 8192, 8193, 20_000])
def test_projected_columns(db, n):
    t = table(n, n)
    db.create_table("t", t)
    r = db.sql(f"SELECT x, id FROM t ORDER BY id LIMIT {n}")
    want = [None if m else int(v) for v, m in zip(np.ma.getdata(t["x"]), np.ma.getmaskarray(t["x"]))]
    assert [r.value(i, 0) for i in range(n)] == want
    assert list(r.column(1)) == list(range(n))


def test_two_databases_in_two_threads():
    """Each context reads back through its own buffer."""
    bad = []

    def run(seed):
        db = F.Database(0)
        t = table(5000, seed)
        db.create_table("t", t)
        for _ in range(20):
            if int(db.sql("SELECT SUM(x), COUNT(x) FROM t").column(1)[0]) != int(t["x"].count()):
                bad.append(("count", seed))
            if list(db.sql("SELECT id FROM t WHERE x IS NULL ORDER BY id LIMIT 100").column(0)) != list(
                    t["id"][np.ma.getmaskarray(t["x"])][:100]):
                bad.append(("rows", seed))
        del db

    th = [threading.Thread(target=run, args=(s,)) for s in (1, 2)]
    for x in th:
        x.start()
    for x in th:
        x.join()
    assert not bad
