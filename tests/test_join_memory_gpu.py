"""Joins when the runtime's budget runs out: a call that fails for memory may be
made again, and what it was called on is as it was before. Exact."""
import ctypes as C

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


@pytest.mark.parametrize("call", ["probe", "finish"])
def test_a_slice_that_cannot_be_handed_out_waits(kb, small, call):
    n = 1_000_003  # in slices whose bitmaps take more than ballast leaves
    k = np.arange(n)
    # probe: unmatched rows padded; finish: the full outer join's build rows that no row matched
    j = kb.HashJoin(small, kb.join_spec("full_outer", probe_out=[0], build_out=[1], max_output_rows=196_608))
    build, probe = (k + n, k[:10]) if call == "finish" else (k[:10] + n, k)
    j.build_push_device(kb.DeviceBatch([column("k", build), column("v", build * 3)]))
    j.build_finish()
    rows = []

    def take(call_again):
        arr, sch = kb.ArrowDeviceArray(), kb.ArrowSchema()
        st = call_again(C.byref(arr), C.byref(sch))
        if st != kb.NEED_MEMORY:
            r = kb.DeviceResult(arr, sch)
            null = np.unpackbits(r.valid[1 if call == "probe" else 0].cpu().numpy(), bitorder="little")[:r.rows] == 0
            rows.extend((r.columns[0] if call == "probe" else r.columns[1]).cpu().numpy()[null].tolist())
        return kb.check(st) if st != kb.NEED_MEMORY else st

    p, lib = kb.DeviceBatch([column("k", probe)]), kb.lib()
    st = take(lambda a, s: lib.krv_join_probe_device(j.h, C.byref(p.dev), C.byref(p.schema), a, s))
    failed = 0
    more = lambda a, s: (lib.krv_join_probe_device(j.h, None, None, a, s) if call == "probe"  # noqa: E731
                         else lib.krv_join_finish_device(j.h, a, s))
    if call == "finish":
        rows.clear()
        st = take(more)
    while st == kb.HAVE_MORE_OUTPUT:
        b = ballast(kb, small, BUDGET, 0)
        failed += take(more) == kb.NEED_MEMORY
        b.close()
        st = take(more)
    assert failed >= 3 and sorted(rows) == (k.tolist() if call == "probe" else (build * 3).tolist())
    j.close()


@pytest.mark.parametrize("dup,jt", [(1, "left_outer"), (1, "left_semi"), (2, "inner"), (2, "left_outer")])
@pytest.mark.parametrize("n", [1_000_003, 50_003])
def test_probe_with_room_for_little_but_its_output(kb, small, dup, jt, n):
    nb = 100_003
    k = np.random.default_rng(dup).permutation(nb).astype(np.int64) * 1_000_003
    pk = np.random.default_rng(n).permutation(np.resize(k, n))
    semi = jt == "left_semi"
    j = kb.HashJoin(small, kb.join_spec(jt, probe_out=[0, 1], build_out=[] if semi else [1]))
    j.build_push_device(kb.DeviceBatch([column("k", np.tile(k, dup)), column("v", np.arange(nb * dup))]))
    j.build_finish()
    p = kb.DeviceBatch([column("k", pk), column("r", np.arange(n))])
    out_rows = n * dup
    out = out_rows * (16 if semi else 24) + (out_rows // 8 if jt == "left_outer" else 0)
    b = ballast(kb, small, BUDGET, out + n // 8 + (96 << 10))  # less than the rows' lookups take
    r = j.probe_device(p)
    b.close()
    assert r.rows == out_rows
    row = r.columns[1].cpu().numpy()
    assert np.array_equal(np.sort(row), np.repeat(np.arange(n), dup))
    assert np.array_equal(r.columns[0].cpu().numpy(), pk[row])
    if not semi:
        v = r.columns[2].cpu().numpy()
        assert np.array_equal(k[v % nb], pk[row]) and np.unique(row * (nb * dup) + v).size == out_rows
    j.close()


@pytest.mark.parametrize("dup,jt", [(1, "inner"), (3, "inner"), (1, "left_semi"), (1, "left_anti")])
@pytest.mark.parametrize("n", [1_000_003, 40_003])
def test_probe_without_room_for_its_lookups(kb, small, dup, jt, n):
    """Few rows come out: the lookups are what does not fit, and they are made again a chunk at a time."""
    nb = 5_003
    k = np.arange(nb) * 1_000_003
    rng = np.random.default_rng(n + dup)
    hit = rng.random(n) < (0.99 if jt == "left_anti" else 0.01)
    pk = np.where(hit, k[rng.integers(0, nb, n)], -1 - np.arange(n))
    j = kb.HashJoin(small, kb.join_spec(jt, probe_out=[1], build_out=[1] if jt == "inner" else []))
    j.build_push_device(kb.DeviceBatch([column("k", np.tile(k, dup)), column("v", np.arange(nb * dup))]))
    j.build_finish()
    p = kb.DeviceBatch([column("k", pk), column("r", np.arange(n))])
    b = ballast(kb, small, BUDGET, n * 2 + (64 << 10))
    r = j.probe_device(p)
    b.close()
    out = np.flatnonzero(~hit if jt == "left_anti" else hit)
    assert np.array_equal(np.sort(r.columns[0].cpu().numpy()), np.repeat(out, dup))
    if jt == "inner":
        row, v = (c.cpu().numpy() for c in r.columns)
        assert np.array_equal(k[v % nb], pk[row]) and np.unique(row * (nb * dup) + v).size == out.size * dup
    j.close()


@pytest.mark.parametrize("jt", ["right_anti", "right_semi", "right_outer", "full_outer"])
def test_the_tail_comes_when_there_is_memory(kb, small, jt):
    n = 500_003
    k = np.arange(n)
    j = kb.HashJoin(small, kb.join_spec(jt, probe_out=[0], build_out=[1]))
    j.build_push_device(kb.DeviceBatch([column("k", k), column("v", k * 3)]))
    j.build_finish()
    j.probe_device(kb.DeviceBatch([column("k", k[:1000])]))
    b = ballast(kb, small, BUDGET, 1 << 20)
    assert status(kb, lambda: list(j.finish_device())) == kb.NEED_MEMORY
    b.close()
    v = np.concatenate([r.columns[-1].cpu().numpy() for r in j.finish_device() if r.rows])
    assert np.array_equal(np.sort(v), k[:1000] * 3 if jt == "right_semi" else k[1000:] * 3)
    j.close()
