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


@pytest.mark.parametrize("keys", [1, 2])
def test_push_that_finds_no_memory_may_be_made_again(kb, rt, keys):
    from test_join_memory_gpu import ballast, status
    budget = 512 << 20
    small = kb.Runtime.on_torch_stream(0, budget_bytes=budget, stream=rt.torch_stream)
    rng = np.random.default_rng(keys)
    n, groups = 300_001, 150_000  # more groups than the hint's table, and rows enough for the partitioned kernels
    k, v = rng.integers(0, groups, n), rng.integers(-99, 99, n)
    cols = [("k", torch.as_tensor(k, device="cuda"), None)]
    if keys == 2:
        cols = [("k0", (cols[0][1] // 400).to(torch.int32), None), ("k1", (cols[0][1] % 400).to(torch.int32), None)]
    cols.append(("v", torch.as_tensor(v, device="cuda"), None))
    batch = kb.DeviceBatch(cols)
    a = kb.HashAggregate(small, kb.agg_spec(0 if keys == 1 else (0, 1), [("sum", keys), ("count_star", 0)], expected_groups=10))
    failed = 0
    for free in [1 << 14] + [i << 21 for i in range(1, 100)]:
        b = ballast(kb, small, budget, free)
        st = status(kb, a.push_device, batch)
        if b is not None:
            b.close()
        if st == kb.OK:
            break
        assert st == kb.NEED_MEMORY
        failed += 1
    assert failed > 2 and st == kb.OK
    a.finish()
    r = a.result_device()
    c = [x.cpu().numpy() for x in r.columns]
    key = c[0] if keys == 1 else c[0].astype(np.int64) * 400 + c[1]
    order = np.argsort(key)
    assert np.array_equal(key[order], np.unique(k))
    assert np.array_equal(c[keys][order], np.bincount(k, v, minlength=groups)[key[order]].astype(np.int64))
    assert np.array_equal(c[keys + 1][order], np.bincount(k, minlength=groups)[key[order]])
    a.close()
    small.close()


def test_large_batch_of_hot_keys_takes_little_memory(kb, rt):
    """Nearly every row is of a key that the sample knows: under a budget the few others' partitions leave room for the table."""
    from test_join_memory_gpu import ballast
    budget = 512 << 20
    small = kb.Runtime.on_torch_stream(0, budget_bytes=budget, stream=rt.torch_stream)
    rng = np.random.default_rng(5)
    n = 1_700_003  # 54 MB as partition rows
    k, v = rng.integers(0, 100, n), rng.integers(-99, 99, n)
    k[::100] = rng.integers(100, 20_000, k[::100].size)
    a = kb.HashAggregate(small, kb.agg_spec(0, [("sum", 1), ("count_star", 0)], expected_groups=100))
    b = ballast(kb, small, budget, 130 << 20)
    push(kb, a, k, v)
    b.close()
    key, total, count = groups_of(a)
    assert np.array_equal(key, np.unique(k))
    assert np.array_equal(total, np.bincount(k, v)[key].astype(np.int64)) and np.array_equal(count, np.bincount(k)[key])
    a.close()
    small.close()


@pytest.mark.parametrize("expected", [10, 150_000])
def test_partitioned_batch_in_a_small_budget(kb, rt, expected):
    """The table holds the keys that there are, not a table's worth for every CTA beside."""
    budget = 56 << 20
    small = kb.Runtime.on_torch_stream(0, budget_bytes=budget, stream=rt.torch_stream)
    rng = np.random.default_rng(expected)
    n, groups = 300_001, 150_000
    a = kb.HashAggregate(small, kb.agg_spec(0, [("sum", 1), ("count_star", 0)], expected_groups=expected))
    ks, vs = [], []
    for i in range(2):  # the second batch's keys are half known
        k, v = rng.integers(0, groups, n) + i * groups // 2, rng.integers(-99, 99, n)
        push(kb, a, k, v)
        ks.append(k)
        vs.append(v)
    k, v = np.concatenate(ks), np.concatenate(vs)
    key, total, count = groups_of(a)
    assert np.array_equal(key, np.unique(k))
    assert np.array_equal(total, np.bincount(k, v)[key].astype(np.int64)) and np.array_equal(count, np.bincount(k)[key])
    a.close()
    small.close()


@pytest.mark.parametrize("keys", [1, 2])
def test_few_groups_without_room_to_list_the_rows(kb, rt, keys):
    from test_join_memory_gpu import ballast
    budget = 256 << 20
    small = kb.Runtime.on_torch_stream(0, budget_bytes=budget, stream=rt.torch_stream)
    rng = np.random.default_rng(keys)
    n = 8_000_003  # 32 MB to list them; 64 MB of codes for two columns
    k, v = rng.integers(0, 6, n), rng.integers(-99, 99, n)
    kt = torch.as_tensor(k, device="cuda")
    cols = [("k", kt, None)] if keys == 1 else [("k0", (kt // 2).to(torch.int32), None), ("k1", (kt % 2).to(torch.int32), None)]
    cols.append(("v", torch.as_tensor(v, device="cuda"), None))
    a = kb.HashAggregate(small, kb.agg_spec(0 if keys == 1 else (0, 1), [("sum", keys), ("count_star", 0)], expected_groups=6))
    b = ballast(kb, small, budget, (16 << 20) if keys == 1 else (110 << 20))
    a.push_device(kb.DeviceBatch(cols))
    b.close()
    a.finish()
    r = a.result_device()
    c = [x.cpu().numpy() for x in r.columns]
    key = c[0] if keys == 1 else c[0].astype(np.int64) * 2 + c[1]
    assert np.array_equal(np.sort(key), np.arange(6))
    assert np.array_equal(c[keys], np.bincount(k, v)[key].astype(np.int64)) and np.array_equal(c[keys + 1], np.bincount(k)[key])
    a.close()
    small.close()


def test_a_batch_left_half_taken_is_an_error(kb, rt):
    """Growth in the middle of a batch finds no memory: no later call gives sums with part of it, or part of it twice."""
    from test_join_memory_gpu import ballast, status
    budget = 64 << 20
    small = kb.Runtime.on_torch_stream(0, budget_bytes=budget, stream=rt.torch_stream)
    rng = np.random.default_rng(1)
    k, v = rng.integers(0, 4000, 5000), rng.integers(-9, 9, 5000)
    a = kb.HashAggregate(small, kb.agg_spec(0, [("sum", 1), ("count_star", 0)], expected_groups=10))
    push(kb, a, k[:10], v[:10])
    b = ballast(kb, small, budget, 128 << 10)
    assert status(kb, push, kb, a, k, v) == kb.NEED_MEMORY
    b.close()
    assert status(kb, push, kb, a, k, v) == kb.INTERNAL
    a.finish()
    assert status(kb, a.result_device) == kb.INTERNAL
    a.close()
    small.close()
