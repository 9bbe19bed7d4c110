"""Joins when the runtime's budget runs out: a call that fails for memory may be
made again, and what it was called on is as it was before. Exact."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
BUDGET = 64 << 20


def column(name, a):
    return (name, torch.as_tensor(a, device="cuda"), None)


def ballast(kb, rt, budget, free):
    """Takes a runtime's budget up to about `free` bytes: a join's arena with room for the rest."""
    rows = (budget - rt.used_bytes - free) // 8
    if rows < 2048:
        return None
    j = kb.HashJoin(rt, kb.join_spec("inner", build_rows_hint=int(rows)))
    j.build_push_device(kb.DeviceBatch([column("k", np.zeros(1, np.int64))]))
    return j


@pytest.fixture(scope="module")
def small(kb, rt):
    """A runtime of little memory, on the tests' stream."""
    r = kb.Runtime.on_torch_stream(0, budget_bytes=BUDGET, stream=rt.torch_stream)
    yield r
    r.synchronize()


def status(kb, call, *args):
    try:
        call(*args)
    except kb.KrvError as e:
        return e.status
    return kb.OK


@pytest.mark.parametrize("partitioned", [False, True])
def test_build_finish_may_be_called_again(kb, small, partitioned):
    rt = small
    n = 100_003
    k = np.random.default_rng(3).permutation(n).astype(np.int64) * 1_000_003
    j = kb.HashJoin(rt, kb.join_spec("inner", probe_out=[0], build_out=[1]), partitioned=partitioned)
    j.build_push_device(kb.DeviceBatch([column("k", k), column("v", np.arange(n))]))
    p = kb.DeviceBatch([column("k", k[::-1].copy())])
    for free in (1 << 16, 1 << 18, 1 << 19):  # the slots, a column or a partition's table do not fit
        b = ballast(kb, rt, BUDGET, free)
        assert status(kb, j.build_finish) == kb.NEED_MEMORY
        assert status(kb, j.probe_device, p) == kb.INVALID_ARGUMENT
        b.close()
    j.build_finish()
    got = [(r.columns[0].cpu().numpy(), r.columns[1].cpu().numpy()) for r in j.probe_device_all(p) if r.rows]
    key, v = (np.concatenate([g[i] for g in got]) for i in range(2))
    assert len(key) == n and np.array_equal(np.sort(v), np.arange(n)) and np.array_equal(k[v], key)
    assert j.counters()["build_keys"] == n
    j.close()
