"""The aggregate of a handful of groups (each thread's own accumulators), the
dictionary encode that samples first, and batches that go straight to the
global table, against the one-pass global mode. Row counts at the edges of the
kernels' turns; groups at the edge of what the accumulators hold; NULL and
marker keys; columns with and without bitmaps; keys that no sample saw, in the
batch and in a later one; integers at the ends of their ranges. Integers are
equal; float64 sums within 1e-12 of the rows' total size; infinities and NaN
equal."""
import numpy as np
import pyarrow as pa
import pytest

from helpers import batch, concat

pytestmark = pytest.mark.gpu
MARKER = np.uint64(0x8080808080808080).astype(np.int64)


def run(kb, rt, batches, keys, aggs, mode):
    a = kb.HashAggregate(rt, kb.agg_spec(keys, aggs, mode=mode, expected_groups=16))
    for b in batches:
        a.push(b)
    a.finish()
    t = concat(a.result())
    cols = [t.column(i).to_pylist() for i in range(len(keys) if isinstance(keys, list) else 1)]
    order = sorted(range(t.num_rows), key=lambda i: tuple((c[i] is None, c[i] if c[i] is not None else 0) for c in cols))
    return t.take(pa.array(order))


def same(got, want, n):
    assert got.num_rows == want.num_rows
    for i in range(got.num_columns):
        g, w = got.column(i).combine_chunks(), want.column(i).combine_chunks()
        assert g.is_null().equals(w.is_null()), i
        if pa.types.is_floating(g.type):
            gn, wn = (x.fill_null(0).to_numpy(zero_copy_only=False) for x in (g, w))
            finite = np.isfinite(wn)
            assert np.array_equal(gn[~finite], wn[~finite], equal_nan=True), i
            assert np.all(np.abs(gn[finite] - wn[finite]) <= 1e-12 * n), i
        else:
            assert g.equals(w), i


def values(r, n, nulls, ncols):
    cols = {}
    for c in range(ncols):
        mask = r.random(n) < 0.05 if nulls else None
        kind = c % 4
        if kind == 0:
            v = r.integers(-2**63, 2**63 - 1, n, dtype=np.int64) >> (0 if c else 20)
        elif kind == 1:
            v = r.random(n) - 0.5
        elif kind == 2:
            v = r.integers(-2**31, 2**31 - 1, n).astype(np.int32)
        else:
            v = r.integers(-10**15, 10**15, n, dtype=np.int64)
        a = pa.array(v, mask=mask)
        if kind == 3:  # a decimal(18, 0)
            a = pa.array(v, mask=mask).cast(pa.decimal128(19, 0)).cast(pa.decimal128(18, 0))
        cols["c%d" % c] = a
    return cols


# groups 40 is past what the accumulators of four columns hold; 4096 * 148 * 5
# + 1 rows: one more than whole turns of the grid
@pytest.mark.parametrize("n", [(1 << 18), (1 << 18) + 129, 740 * 128 * 4 + 1])
@pytest.mark.parametrize("groups,ncols,nulls", [(1, 1, False), (6, 3, False), (6, 3, True), (7, 4, True), (3, 7, True), (40, 4, True)])
def test_few_groups(kb, rt, n, groups, ncols, nulls):
    r = np.random.default_rng(groups * 10 + ncols)
    k = r.integers(0, groups, n).astype(np.int64) * 1_000_003 - 5
    k[n // 2 + 1] = 77  # a key that the sample does not see, most likely
    k[n - 1] = MARKER
    mask = r.random(n) < 0.01 if nulls else None
    cols = {"k": pa.array(k, mask=mask), **values(r, n, nulls, ncols)}
    late = {"k": pa.array(r.integers(0, groups + 3, n).astype(np.int64) * 1_000_003 - 5), **values(r, n, nulls, ncols)}
    batches = [batch(**cols), batch(**late)]
    # sums of full-range int64 leave 64 bits: not asked for
    aggs = [("count_star", 0)]
    for c in range(ncols):
        aggs += [(f, 1 + c) for f in (("sum", "min", "max", "count") if c != 4 else ("min", "max", "count"))]
    same(run(kb, rt, batches, 0, aggs, kb.MODE_AUTO), run(kb, rt, batches, 0, aggs, kb.MODE_GLOBAL), 2 * n)


@pytest.mark.parametrize("n", [(1 << 18) + 5])
def test_few_groups_infinities(kb, rt, n):
    r = np.random.default_rng(3)
    k = r.integers(0, 5, n).astype(np.int32)
    v = r.random(n)
    v[np.flatnonzero(k == 0)[:2]] = np.inf
    v[np.flatnonzero(k == 1)[:2]] = [np.inf, -np.inf]
    v[np.flatnonzero(k == 2)[7]] = np.nan
    v[k == 3] = -0.0
    b = [batch(k=pa.array(k), v=pa.array(v))]
    aggs = [(f, 1) for f in ("sum", "min", "max", "avg", "count")]
    same(run(kb, rt, b, 0, aggs, kb.MODE_AUTO), run(kb, rt, b, 0, aggs, kb.MODE_GLOBAL), n)


@pytest.mark.parametrize("kind", ["ints", "strings", "nulls"])
@pytest.mark.parametrize("n", [20_000, 65_536, (1 << 18) + 3])
def test_dictionary_codes(kb, rt, kind, n):
    r = np.random.default_rng(n)

    def make(extra):
        a = r.integers(0, 3 + extra, n)
        b = r.integers(0, 2, n)
        a[n // 3 + 1] = 900 + extra  # not in the sample
        if kind == "strings":
            ka, kb_ = pa.array(np.array(["", "key"] + ["k%03d" % i for i in range(1000)])[a]), pa.array(b.astype(np.int32))
        else:
            m = r.random(n) < 0.1 if kind == "nulls" else None
            ka, kb_ = pa.array(a.astype(np.int32), mask=m), pa.array(b.astype(np.int64))
        return batch(a=ka, b=kb_, v=pa.array(r.integers(-9, 9, n).astype(np.int64)), w=pa.array(r.random(n)))
    batches = [make(0), make(0), make(4)]
    aggs = [("count_star", 0), ("sum", 2), ("min", 2), ("sum", 3), ("max", 3)]
    same(run(kb, rt, batches, [0, 1], aggs, kb.MODE_AUTO), run(kb, rt, batches, [0, 1], aggs, kb.MODE_GLOBAL), 3 * n)


@pytest.mark.parametrize("n", [1, 8192, 16_384, 16_385])
@pytest.mark.parametrize("groups", [1, 1000, 200_000])
def test_small_batches(kb, rt, n, groups):
    r = np.random.default_rng(n + groups)
    batches = [batch(k=pa.array(r.integers(0, groups, n)), v=pa.array(r.integers(-2**40, 2**40, n))) for _ in range(9)]
    t = pa.Table.from_batches(batches).group_by("k").aggregate([("v", "sum"), ("v", "min"), ("v", "count")]).sort_by("k")
    got = run(kb, rt, batches, 0, [("sum", 1), ("min", 1), ("count", 1)], kb.MODE_AUTO)
    for i, name in enumerate(["k", "v_sum", "v_min", "v_count"]):
        assert got.column(i).to_pylist() == t.column(name).to_pylist(), name
