"""Edges of the partitioned aggregate's fold and split kernels that need a plan
the few-group kernel refuses (a decimal128 sum): a first batch whose sample
knows a handful of keys while every partition holds more than the local table
(windows, their keys looked up after), batches of known and new keys after it;
infinities and NaN in cold and in hot keys. Against the one-pass global mode:
integers equal, float64 sums within 1e-12 of the sum or of 1, the same infinities
and NaN."""
import numpy as np
import pyarrow as pa
import pytest

from test_agg_fold_gpu import run
from helpers import batch

pytestmark = pytest.mark.gpu
AGGS = [("count_star", 0), ("sum", 1), ("sum", 2), ("min", 2), ("max", 2), ("sum", 3), ("count", 2)]


def rows(rng, k, special):
    n = k.size
    f = rng.random(n) - 0.5
    if special:
        at = rng.integers(0, n, 60)
        f[at] = rng.choice([np.inf, -np.inf, np.nan, 1e308, -1e308, 5e-324, -0.0], 60)
    i = rng.integers(-2**62, 2**62, n)
    d = pa.array(rng.integers(-2**40, 2**40, n).astype(np.int32)).cast(pa.int64())
    d = d.cast(pa.decimal128(38, 0))
    return batch(k=pa.array(k), d=d, f=pa.array(f, mask=rng.random(n) < 0.05), i=pa.array(i // 4096))


@pytest.mark.parametrize("special", [False, True])
@pytest.mark.parametrize("case", ["windows", "windows twice", "hot"])
def test_fold_edges_equal_one_pass(kb, rt, case, special):
    rng = np.random.default_rng(len(case) + special)
    n = 1 << 18
    if case == "hot":
        k = np.where(rng.random(n) < 0.9, rng.integers(0, 20, n), rng.integers(0, 5000, n))
    else:  # the sample (every fourth row) sees key 5 and 40 others, the rest are 200,000 keys
        k = rng.integers(0, 200_000, n)
        k[::4] = np.where(rng.random(n // 4) < 0.6, 5, rng.integers(300_000, 300_040, n // 4))
    batches = [rows(rng, k, special)]
    if case == "windows twice":
        batches.append(rows(rng, rng.integers(100_000, 300_000, n), special))
    got = run(kb, rt, batches, AGGS, kb.MODE_AUTO, 10)
    want = run(kb, rt, batches, AGGS, kb.MODE_GLOBAL, 10)
    assert got.num_rows == want.num_rows and got.column(0).equals(want.column(0))
    for c in range(1, got.num_columns):
        if got.schema.field(c).type != pa.float64():
            assert got.column(c).equals(want.column(c)), got.schema.field(c).name
            continue
        a, b = (t.column(c).to_pandas().to_numpy() for t in (got, want))
        finite = np.isfinite(b.astype(float))
        assert np.array_equal(np.isnan(a.astype(float)), np.isnan(b.astype(float)))
        assert np.array_equal(a[~finite & ~np.isnan(b.astype(float))], b[~finite & ~np.isnan(b.astype(float))])
        assert np.all(np.abs(a[finite] - b[finite]) <= 1e-12 * np.abs(b[finite]) + 1e-12)
