"""Filter: predicate -> BOOL8 mask, mask -> compaction, the fused select,
and count_nonzero, against numpy on the same inputs (exact: masks,
kept rows and their order)."""
import numpy as np
import pytest

import eiger_b200 as gx
import oracle as O
from tests.helpers import to_dev, to_dev_raw

pytestmark = pytest.mark.gpu


def np_cmp(x, op, lo, hi):
    return {gx.CMP_LT: x < lo, gx.CMP_LE: x <= lo, gx.CMP_GT: x > lo, gx.CMP_GE: x >= lo, gx.CMP_EQ: x == lo,
            gx.CMP_NE: x != lo, gx.CMP_BETWEEN: (x >= lo) & (x < hi)}[op]


@pytest.mark.parametrize("n", [0, 1, 4095, 4096, 1 << 20])
def test_date_range_select_like_the_batched_pipeline(n):
    # The batched workload's filter: lo <= date < hi on an int32 date column.
    date = O.gen_values(n, np.int32, lo=0, hi=2557, seed=1)
    amount = O.gen_values(n, np.int64, lo=100, hi=10**7, seed=2)
    code = O.gen_values(n, np.int32, lo=0, hi=10**4, seed=3)
    cols = [to_dev(date), to_dev(amount), to_dev(code)]
    p = [gx.predicate(0, gx.CMP_BETWEEN, 500, 500 + 1023)]
    keep = (date >= 500) & (date < 1523)
    m = gx.select_to_bitmask(cols, p).cpu().numpy()
    assert np.array_equal(m.astype(bool), keep)
    t = gx.select(cols, p)
    d, a, c = t.numpy_columns()
    assert np.array_equal(d, date[keep]) and np.array_equal(a, amount[keep]) and np.array_equal(c, code[keep])
    t2 = gx.compact(cols, to_dev(keep.astype(np.uint8)).view(__import__("torch").bool))
    for x, y in zip(t2.numpy_columns(), (date[keep], amount[keep], code[keep])):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("combine", [gx.COMBINE_AND, gx.COMBINE_OR])
def test_every_comparison_on_every_type(combine):
    n = 100_003
    rng = np.random.default_rng(4)
    cols = {
        np.int8: rng.integers(-100, 100, n).astype(np.int8),
        np.uint16: rng.integers(0, 60000, n).astype(np.uint16),
        np.int32: rng.integers(-10**6, 10**6, n).astype(np.int32),
        np.uint64: rng.integers(0, 2**63, n, dtype=np.uint64) * np.uint64(2),
        np.float32: rng.normal(size=n).astype(np.float32),
        np.float64: rng.normal(size=n),
    }
    arrs = list(cols.values())
    lits = [(-3, 40), (1000, 50000), (-5000, 123456), (2**63 + 5, 2**64 - 10), (-0.25, 0.5), (0.1, 1.5)]
    for op in range(7):
        preds = []
        expect = np.ones(n, bool) if combine == gx.COMBINE_AND else np.zeros(n, bool)
        for j, (a, (lo, hi)) in enumerate(zip(arrs, lits)):
            preds.append(gx.predicate(j, op, lo, hi))
            e = np_cmp(a, op, a.dtype.type(lo), a.dtype.type(hi))
            expect = expect & e if combine == gx.COMBINE_AND else expect | e
        m = gx.select_to_bitmask([to_dev(a) for a in arrs], preds, combine).cpu().numpy().astype(bool)
        assert np.array_equal(m, expect), op
        t = gx.select([to_dev(a) for a in arrs], preds, combine)
        for got, a in zip(t.numpy_columns(), arrs):
            assert np.array_equal(got, a[expect])


def test_count_nonzero_and_validation():
    v = np.array([0, 1, -1, 0, 5], np.int64)
    assert gx.count_nonzero(to_dev(v)) == 3
    f = np.array([0.0, -0.0, np.nan, 2.0], np.float64)
    assert gx.count_nonzero(to_dev(f)) == 2  # NaN != 0, -0.0 == 0
    x = to_dev(np.arange(10, dtype=np.int32))
    with pytest.raises(gx.GxError):
        gx.select([x], [gx.predicate(3, gx.CMP_LT, 1)])  # column out of range
    with pytest.raises(gx.GxError):
        gx.select([x], [])  # no predicate


@pytest.mark.parametrize("dt", [np.int8, np.uint8, np.int16, np.uint16, np.int32, np.uint32, np.int64, np.uint64])
def test_integer_ranges_at_the_type_limits(dt):
    # Literals at, just inside and beyond the column type's limits: the ranges
    # that the comparisons become must neither wrap nor clip.
    inf = np.iinfo(dt)
    a = np.array([inf.min, inf.min + 1, 0, 1, inf.max - 1, inf.max] * 700, dt)[:4099]
    wide = [int(x) for x in a]
    lim = (0, 2**64 - 1) if inf.min == 0 else (-2**63, 2**63 - 1)
    lits = sorted({lim[0], lim[1], inf.min, inf.min + 1, inf.max, inf.max - 1, max(inf.min - 1, lim[0]),
                   min(inf.max + 1, lim[1]), 0, 1})
    cols = [to_dev_raw(a)]
    view = gx.ColumnView(cols[0].data_ptr(), len(a), gx._NP_TO_GX[np.dtype(dt)], 0)
    py = {gx.CMP_LT: lambda x, l, h: x < l, gx.CMP_LE: lambda x, l, h: x <= l, gx.CMP_GT: lambda x, l, h: x > l,
          gx.CMP_GE: lambda x, l, h: x >= l, gx.CMP_EQ: lambda x, l, h: x == l, gx.CMP_NE: lambda x, l, h: x != l,
          gx.CMP_BETWEEN: lambda x, l, h: l <= x < h}
    for op in range(7):
        for lo in lits:
            for hi in lits if op == gx.CMP_BETWEEN else [0]:
                m = gx.select_to_bitmask([view], [gx.predicate(0, op, lo, hi)]).cpu().numpy().astype(bool)
                assert np.array_equal(m, np.array([py[op](x, lo, hi) for x in wide])), (op, lo, hi)


@pytest.mark.parametrize("dt", [np.float32, np.float64])
def test_float_ranges_with_infinities_nan_and_zeros(dt):
    vals = [-np.inf, -1.5, -0.0, 0.0, 1e-40, 2.0, np.inf, np.nan]
    a = np.array(vals * 600, dt)[:4101]
    d = to_dev(a)
    for op in range(7):
        for lo in [-np.inf, -1.5, -0.0, 0.0, 0.1, 2.0, np.inf, np.nan]:
            for hi in [-np.inf, 0.0, 2.0, np.inf, np.nan] if op == gx.CMP_BETWEEN else [0.0]:
                e = np_cmp(a.astype(np.float64), op, lo, hi)
                p = gx.predicate(0, op)
                p.lo_f, p.hi_f = lo, hi
                assert np.array_equal(gx.select_to_bitmask([d], [p]).cpu().numpy().astype(bool), e), (op, lo, hi)
                got = gx.select([d], [p]).to_numpy(0)
                assert np.array_equal(got, a[e], equal_nan=True), (op, lo, hi)


@pytest.mark.parametrize("combine", [gx.COMBINE_AND, gx.COMBINE_OR])
@pytest.mark.parametrize("n", [1, 33, 511, 512, 513, 4097, 100_003])
@pytest.mark.parametrize("decided", [0.0, 0.9, 0.9999, 1.0])
def test_rows_decided_by_the_first_predicate(combine, n, decided):
    # Rows that the first predicate decides (false under AND, true under OR) are
    # not read by the later ones, whole warps of them or single rows.
    rng = np.random.default_rng(n)
    a = (rng.random(n) < decided).astype(np.int8)
    a[n // 2:] = a[n // 2:] if decided < 0.99 else 1  # long decided stretches
    b = rng.integers(0, 10, n).astype(np.uint16)
    c = np.where(rng.random(n) < 0.2, np.nan, rng.random(n)).astype(np.float32)
    cols = [to_dev(a), to_dev_raw(b), to_dev(c)]
    views = [gx.ColumnView(t.data_ptr(), n, gx._NP_TO_GX[x.dtype], 0) for t, x in zip(cols, (a, b, c))]
    first = gx.predicate(0, gx.CMP_EQ, 0 if combine == gx.COMBINE_AND else 1)
    preds = [first, gx.predicate(1, gx.CMP_NE, 4), gx.predicate(2, gx.CMP_LT, 0.5)]
    parts = [a == (0 if combine == gx.COMBINE_AND else 1), b != 4, c < 0.5]
    keep = np.logical_and.reduce(parts) if combine == gx.COMBINE_AND else np.logical_or.reduce(parts)
    assert np.array_equal(gx.select_to_bitmask(views, preds, combine).cpu().numpy().astype(bool), keep)
    for got, x in zip(gx.select(views, preds, combine).numpy_columns(), (a, b, c)):
        assert np.array_equal(got, x[keep], equal_nan=x.dtype.kind == "f")
