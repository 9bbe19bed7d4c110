"""Aggregates when memory is short: many small ones beside each other, batches
whose helpers do not fit. Exact."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def push(kb, a, k, v):
    a.push_device(kb.DeviceBatch([("k", torch.as_tensor(k, device="cuda"), None), ("v", torch.as_tensor(v, device="cuda"), None)]))


def groups_of(a):
    a.finish()
    r = a.result_device()
    order = np.argsort(r.columns[0].cpu().numpy())
    return [c.cpu().numpy()[order] for c in r.columns[:3]]


@pytest.mark.parametrize("budget", [0, 512 << 20])
def test_many_small_aggregates_live_together(kb, rt, budget):
    small = kb.Runtime.on_torch_stream(0, budget_bytes=budget, stream=rt.torch_stream)
    rng = np.random.default_rng(1)
    live = []
    for i in range(300):
        a = kb.HashAggregate(small, kb.agg_spec(0, [("sum", 1), ("count_star", 0)], expected_groups=100))
        k, v = rng.integers(0, 100, 1000), rng.integers(-9, 9, 1000)
        push(kb, a, k, v)
        live.append((a, k, v))
    assert small.used_bytes < (1 << 30) + (64 << 20)
    for a, k, v in live:
        key, total, count = groups_of(a)
        assert np.array_equal(key, np.unique(k))
        assert np.array_equal(total, np.bincount(k, v, minlength=100)[key].astype(np.int64))
        assert np.array_equal(count, np.bincount(k, minlength=100)[key])
        a.close()
    small.synchronize()
    assert small.used_bytes < 1 << 20
    small.close()
