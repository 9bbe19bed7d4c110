"""The hot keys of a large batch: none, one, as many as a bucket has places and
one more, as many as there is room for, more; even and very uneven counts. Sums
and counts against numpy, exact."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hot", [0, 1, 2, 31, 32, 33, 1000, 1024, 1100])
@pytest.mark.parametrize("even", [True, False])
def test_hot_keys(kb, rt, hot, even):
    rng = np.random.default_rng(hot + even)
    n = 4_000_003
    if even:
        k = rng.integers(0, max(hot, 1), n)
    else:  # key 0 has half the rows, the others fewer and fewer
        p = 0.999 ** np.arange(max(hot, 1))
        p[0] = p.sum()
        k = rng.choice(max(hot, 1), n, p=p / p.sum())
    cold = rng.random(n) < (0.02 if hot else 1.1)
    k[cold] = rng.integers(10**6, 10**6 + 200_000, int(cold.sum()))
    k = k * np.int64(0x1E3779B97F4A7C15)
    v = rng.integers(-99, 99, n)
    a = kb.HashAggregate(rt, kb.agg_spec(0, [("sum", 1), ("count_star", 0), ("min", 1)], expected_groups=201_000))
    a.push_device(kb.DeviceBatch([("k", torch.as_tensor(k, device="cuda"), None), ("v", torch.as_tensor(v, device="cuda"), None)]))
    a.finish()
    r = a.result_device()
    key, total, count, least = (c.cpu().numpy() for c in r.columns[:4])
    want, at = np.unique(k, return_inverse=True)
    order = np.argsort(key)
    assert np.array_equal(key[order], want)
    assert np.array_equal(total[order], np.bincount(at, v).astype(np.int64))
    assert np.array_equal(count[order], np.bincount(at))
    low = np.full(want.size, 99)
    np.minimum.at(low, at, v)
    assert np.array_equal(least[order], low)
