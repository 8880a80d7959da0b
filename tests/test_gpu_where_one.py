"""Aggregates over NULL-free columns with no WHERE or one comparison: every operator
against the ends of the int64 range, zeros, infinities and NaN, over one to four
columns, whole and part tiles.  Counts, MIN, MAX and the (integer-valued) sums exactly."""
import numpy as np
import pytest
import torch

import falcondb_b200 as F
from falcondb_b200 import ops

pytestmark = pytest.mark.gpu
LO, HI = np.iinfo(np.int64).min, np.iinfo(np.int64).max
OPS = {F.EQ: np.equal, F.NE: np.not_equal, F.LT: np.less, F.LE: np.less_equal, F.GT: np.greater, F.GE: np.greater_equal}
AGGS = [F.AGG_COUNT, F.AGG_SUM, F.AGG_MIN, F.AGG_MAX]


def columns(n, r):
    edge = np.array([LO, LO + 1, -2**53, -1, 0, 1, 7, 2**53 + 1, HI - 1, HI])
    odd = np.array([-np.inf, -1.5, -0.0, 0.0, 2.0, np.inf, np.nan])
    return [r.choice(edge, n), r.choice(odd, n), r.integers(-1000, 1000, n), r.integers(-1000, 1000, n).astype(np.float64)]


def check(db, cols, dev, agg_col, prog, keep):
    n = len(cols[0])
    rec = ops.to_records(ops.aggregate(db, dev, n, prog, [(f, agg_col) for f in AGGS]), F.AGG_VALUE_DTYPE, 4)
    x = cols[agg_col][keep]
    assert rec[0]["i"] == len(x)
    num = x[~np.isnan(x)] if x.dtype == np.float64 else x
    if agg_col >= 2:
        assert rec[1]["f"] == float(x.sum())
    if len(num) == 0:
        assert not rec[2]["valid"] and not rec[3]["valid"]
    else:
        assert rec[2]["f"] == float(num.min()) and rec[3]["f"] == float(num.max())


@pytest.mark.parametrize("n", [1, 1024, 2049, 70_001])
@pytest.mark.parametrize("ncols", [3, 4])
def test_no_where(db, n, ncols):
    cols = columns(n, np.random.default_rng([n, ncols]))[:ncols]
    dev = [torch.from_numpy(c).cuda() for c in cols]
    for a in range(ncols):
        check(db, cols, dev, a, [], np.ones(n, bool))


@pytest.mark.parametrize("n", [1, 2049, 70_001])
@pytest.mark.parametrize("op", list(OPS))
@pytest.mark.parametrize("lit", [LO, LO + 1, -1, 0, 7, HI - 1, HI, np.nan, np.inf, -np.inf, -0.0, 2.0, -1.5])
def test_one_comparison(db, n, op, lit):
    cols = columns(n, np.random.default_rng([n, op]))
    dev = [torch.from_numpy(c).cuda() for c in cols]
    for c in (0, 1, 2):
        x = cols[c]
        # An int64 column widens to float64 against a float literal, as does an
        # int64 literal against a float64 column.
        exact = x.dtype == np.int64 and isinstance(lit, int)
        keep = OPS[op](x, np.int64(lit)) if exact else OPS[op](x.astype(np.float64), np.float64(lit))
        check(db, cols, dev, 2 if c != 2 else 3, [ops.cmp(c, op, lit)], keep)
        check(db, cols[:3], dev[:3], c, [ops.cmp(c, op, lit)], keep)
    # One column alone.
    keep = OPS[op](cols[2], np.int64(lit)) if isinstance(lit, int) else OPS[op](cols[2].astype(np.float64), lit)
    rec = ops.to_records(ops.aggregate(db, [dev[2]], n, [ops.cmp(0, op, lit)], [(F.AGG_SUM, 0)]), F.AGG_VALUE_DTYPE, 1)
    assert rec[0]["f"] == float(cols[2][keep].sum()) and rec[0]["n"] == keep.sum()
