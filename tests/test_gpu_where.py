"""WHERE programs over every term kind, column type and NULL form: the mask, the
count and the aggregates against a row-by-row numpy evaluation, at the edges of
tiles, warps and mask words, with aligned and shifted columns and validity."""
import ctypes as C

import numpy as np
import pytest
import torch

import falcondb_b200 as F
from falcondb_b200 import ops

pytestmark = pytest.mark.gpu
SIZES = [1, 31, 64, 255, 256, 257, 1023, 2049, 8192, 70_001]
NULL_CODE = 0xFFFFFFFF
CMP = {F.EQ: np.equal, F.NE: np.not_equal, F.LT: np.less, F.LE: np.less_equal, F.GT: np.greater,
       F.GE: np.greater_equal}


def make(n, seed, shift):
    """(host values, host validity or None, device column) of f64, i64 and
    UTF8 columns; `shift` rows into longer buffers (misaligned bases, and
    validity that starts inside a word)."""
    r = np.random.default_rng(seed)
    m = n + shift
    f = r.choice([0.0, -0.0, 1.5, 50.0, -3.0, np.nan, np.inf, -np.inf], m)
    i = r.integers(-4, 5, m)
    i[r.random(m) < 0.02] = np.iinfo(np.int64).min
    u = r.integers(0, 7, m).astype(np.uint32)
    u[r.random(m) < 0.1] = NULL_CODE
    out = []
    for k, (v, nullable) in enumerate([(f, True), (i, True), (u, True), (f[::-1].copy(), False)]):
        ok = r.random(m) < 0.8
        t = torch.from_numpy(v.view(np.int32) if v.dtype == np.uint32 else v).cuda()
        w = torch.from_numpy(F.validity_words(ok).view(np.int64)).cuda()
        raw = ops.dev_column(t)
        raw.values += shift * t.element_size()
        if nullable:
            raw.validity, raw.validity_offset = w.data_ptr(), shift
        col = F.DevColumn(raw, n)
        col.keep = (t, w)
        out.append((v[shift:], ok[shift:] if nullable else np.ones(n, bool), col))
    return out


def leaf(term, cols, passing):
    v, ok, _ = cols[term.col]
    utf8 = v.dtype == np.uint32
    null = ~ok | (v == NULL_CODE if utf8 else False)
    if term.kind == F.TERM_IS_NULL:
        return null
    if term.kind == F.TERM_IS_NOT_NULL:
        return ~null
    if term.kind == F.TERM_CODE_SET:
        return ~null & np.array([c < len(passing) and passing[c] for c in v])
    with np.errstate(invalid="ignore"):
        if v.dtype == np.float64:
            return ~null & CMP[term.op](v, term.lit_f if term.lit_type == F.FLOAT64 else float(term.lit_i))
        if utf8:
            return ~null & CMP[term.op](v.astype(np.int64), term.lit_i)
        if term.lit_type == F.FLOAT64:
            return ~null & CMP[term.op](v.astype(np.float64), term.lit_f)
        return ~null & CMP[term.op](v, term.lit_i)


def evaluate(prog, cols, passing):
    st = []
    for t in prog:
        if t.kind in (F.TERM_AND, F.TERM_OR):
            b, a = st.pop(), st.pop()
            st.append(a & b if t.kind == F.TERM_AND else a | b)
        else:
            st.append(leaf(t, cols, passing))
    return st[0] if st else np.ones(len(cols[0][0]), bool)


def programs(code_set):
    yield []
    for op in CMP:
        yield [ops.cmp(0, op, 1.5)]
        yield [ops.cmp(0, op, float("nan"))]
        yield [ops.cmp(0, op, 50)]
        yield [ops.cmp(1, op, 2), ops.cmp(1, op, -0.5), ops.OR()]
        yield [ops.cmp(2, op, 3), ops.is_not_null(0), ops.AND()]
    yield [ops.is_null(0), ops.is_null(1), ops.OR(), ops.is_null(2), ops.OR()]
    yield [ops.is_not_null(2), code_set, ops.AND()]
    yield [ops.is_null(3)]
    # Eight leaves pushed before the first operator: the deepest stack.
    deep = [ops.cmp(0, F.GE, 0.0), ops.cmp(1, F.LT, 3), code_set, ops.cmp(3, F.NE, 50.0), ops.is_not_null(0),
            ops.cmp(1, F.GT, -3.5), ops.is_null(2), ops.cmp(3, F.LE, 1.5)]
    yield deep + [ops.OR(), ops.AND(), ops.OR(), ops.AND(), ops.OR(), ops.AND(), ops.OR()]


@pytest.mark.parametrize("shift", [0, 1, 37])
@pytest.mark.parametrize("n", SIZES)
def test_where_forms(db, n, shift):
    passing = [True, False, True, True, False]
    term, keep = ops.code_set(2, passing, torch.device("cuda"))
    cols = make(n, n + shift, shift)
    dev = [c for _, _, c in cols]
    f, fok, _ = cols[0]
    i, iok, _ = cols[1]
    for prog in programs(term):
        want = evaluate(prog, cols, passing)
        got = ops.filter_mask(db, dev, n, prog).cpu().numpy().view(np.uint8)
        bits = np.unpackbits(got, bitorder="little")
        assert np.array_equal(bits[:n].astype(bool), want) and not bits[n:].any()
        assert int(ops.filter_count(db, dev, n, prog).item()) == want.sum()
        rec = ops.to_records(ops.aggregate(db, dev, n, prog, [(F.AGG_COUNT, 2), (F.AGG_MIN, 0), (F.AGG_SUM, 1),
                                                              (F.AGG_COUNT_STAR, 0)]), F.AGG_VALUE_DTYPE, 4)
        assert rec[0]["i"] == (want & cols[2][1]).sum() and rec[3]["i"] == want.sum()
        low = f[want & fok & ~np.isnan(f)]
        assert bool(rec[1]["valid"]) == bool(len(low)) and rec[1]["n"] == len(low)
        if len(low):
            assert rec[1]["f"] == low.min()
            if rec[1]["f"] == 0.0:  # -0.0 orders before +0.0
                assert np.signbit(rec[1]["f"]) == np.signbit(low[low == 0.0]).any()
        total = sum(int(x) for x in i[want & iok])
        assert rec[2]["n"] == (want & iok).sum() and rec[2]["f"] == float(total)
