"""The partitioned aggregate's fold kernel at the edges of its local table and
steps (512 rows), against the one-pass global mode, which shares none of its
kernels: no cold rows, a handful of keys to a partition, more keys in a
partition than the table holds (windows, the first batch and a later one),
many value columns (a small table), NULL and marker keys. Integers are equal;
float64 sums within 1e-12 relative."""
import numpy as np
import pyarrow as pa
import pytest

from helpers import batch, concat

pytestmark = pytest.mark.gpu
MARKER = np.uint64(0x8080808080808080).astype(np.int64)


def run(kb, rt, batches, aggs, mode, expected):
    a = kb.HashAggregate(rt, kb.agg_spec(0, aggs, mode=mode, expected_groups=expected))
    for b in batches:
        a.push(b)
    a.finish()
    t = concat(a.result())
    key = t.column(0).to_pylist()
    order = sorted(range(len(key)), key=lambda i: (key[i] is None, key[i] if key[i] is not None else 0))
    return t.take(pa.array(order))


@pytest.mark.parametrize("case", ["few", "mid", "many", "windows", "later", "wide"])
def test_fold_equals_one_pass(kb, rt, case):
    rng = np.random.default_rng(sum(map(ord, case)))
    n = (1 << 18) + 77
    groups = {"few": 3, "mid": 1500, "many": 120_000, "windows": 250_000, "later": 250_000, "wide": 60_000}[case]
    # expected_groups under the truth: fewer partitions, each with more keys than the table
    expected = {"many": 0, "wide": 0}.get(case, 10)
    ncols = 14 if case == "wide" else 3

    def make(seed, domain):
        r = np.random.default_rng(seed)
        k = r.integers(0, domain, n).astype(np.int64)
        if case in ("windows", "later"):  # the sample sees few of the keys
            k[:: max(1, n // 65536)] = 5
        k[11] = MARKER
        cols = {"k": pa.array(k, mask=r.random(n) < 0.001)}
        for c in range(ncols):
            mask = r.random(n) < 0.05
            if c % 3 == 0:
                cols["c%d" % c] = pa.array(r.integers(-2**62, 2**62, n, dtype=np.int64) // 4096, mask=mask)
            elif c % 3 == 1:
                cols["c%d" % c] = pa.array(r.random(n) - 0.5, mask=mask)
            else:
                cols["c%d" % c] = pa.array(r.integers(-2**31, 2**31 - 1, n).astype(np.int32), mask=mask)
        return batch(**cols)
    batches = [make(1, 1000 if case == "later" else groups)]
    if case == "later":
        batches.append(make(2, groups))
    aggs = [("count_star", 0)] + [(f, 1 + c) for c in range(ncols) for f in (("sum", "min", "max", "count") if ncols == 3 else ("sum", "min"))]
    got = run(kb, rt, batches, aggs, kb.MODE_AUTO, expected)
    want = run(kb, rt, batches, aggs, kb.MODE_GLOBAL, expected)
    assert got.num_rows == want.num_rows
    for i in range(got.num_columns):
        g, w = got.column(i).combine_chunks(), want.column(i).combine_chunks()
        assert g.is_null().equals(w.is_null()), i
        if pa.types.is_floating(g.type):
            gn, wn = g.fill_null(0).to_numpy(zero_copy_only=False), w.fill_null(0).to_numpy(zero_copy_only=False)
            # sums of values in [-0.5, 0.5): against the rows' total size
            assert np.all(np.abs(gn - wn) <= 1e-12 * np.maximum(1.0, np.abs(wn))), i
        else:
            assert g.equals(w), i
    del rng
