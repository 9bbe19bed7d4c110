"""The partitioned join when memory runs out while it finishes: every call of
finish is made with less memory than it needs first, then with more until it
succeeds. No output row is lost or doubled: padded rows that wait in host
memory, deferred rows of resident partitions, spilled partitions, a partition
of one key joined by the fallback. Exact, against the unpartitioned join."""
import collections
import ctypes as C

import numpy as np
import pytest

from test_grace_gpu import dev, rows_of
from test_join_memory_gpu import BUDGET, ballast, small  # noqa: F401 (small: a fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("jt", ["left_outer", "inner"])
@pytest.mark.parametrize("case", ["waiting", "spilled", "heavy"])
def test_finish_loses_no_rows_to_memory(kb, small, jt, case):  # noqa: F811
    rt = small
    rng = np.random.default_rng(11)
    nb, n, domain = 40_001, 120_003, 80_000
    bk, pk = rng.integers(0, domain, nb), rng.integers(0, domain, n)
    if case == "heavy":
        bk[rng.random(nb) < 0.5] = 7
        pk[pk == 7] = 8
        pk[:3] = 7
    # waiting: the output of a call is more than its share, the tables stay; else most partitions spill
    device_budget = {"waiting": 6 << 20, "spilled": 600 << 10, "heavy": 600 << 10}[case]
    bcols = [("k", bk, rng.random(nb) > 0.02), ("v", np.arange(nb), None)]
    pcols = [("k", pk, rng.random(n) > 0.02), ("r", np.arange(n), None)]
    got = {}
    for partitioned in (False, True):
        spec = kb.join_spec(jt, probe_out=[0, 1], build_out=[1], radix_bits=3, max_output_rows=1 << 20)
        j = kb.HashJoin(rt, spec, partitioned=partitioned, device_budget=device_budget if partitioned else 0)
        for s in np.array_split(np.arange(nb), 3):
            j.build_push_device(dev(kb, [(c, a[s], None if v is None else v[s]) for c, a, v in bcols]))
        j.build_finish()
        rows, failed = [], 0
        for s in np.array_split(np.arange(n), 2):
            for r in j.probe_device_all(dev(kb, [(c, a[s], None if v is None else v[s]) for c, a, v in pcols])):
                rows += rows_of(r)
        st = kb.HAVE_MORE_OUTPUT
        while partitioned and st == kb.HAVE_MORE_OUTPUT:
            for free in [1 << 12, 1 << 14, 1 << 16] + [i << 17 for i in range(1, 40)] + [BUDGET]:
                b = ballast(kb, rt, BUDGET, free)
                try:
                    arr, sch = kb.ArrowDeviceArray(), kb.ArrowSchema()
                    st = kb.check(kb.lib().krv_join_finish_device(j.h, C.byref(arr), C.byref(sch)))
                    rows += rows_of(kb.DeviceResult(arr, sch))
                    break
                except kb.KrvError as e:
                    assert e.status == kb.NEED_MEMORY
                    failed += 1
                finally:
                    if b is not None:
                        b.close()
        got[partitioned] = collections.Counter(rows)
        if partitioned:
            assert failed > 0 and (j.spilled_partitions() == 0) == (case == "waiting")
        j.close()
    assert sum(got[True].values()) == sum(got[False].values())
    assert got[True] == got[False]


@pytest.mark.parametrize("jt", ["left_outer", "inner"])
@pytest.mark.parametrize("device_budget", [600 << 10, 24 << 20])
def test_a_batch_is_taken_whole_or_not_at_all(kb, small, jt, device_budget):  # noqa: F811
    """Batches of several slices, pushed and probed with too little memory first and then again."""
    rng = np.random.default_rng(3)
    nb, n, domain = 300_001, 400_003, 500_000
    bk, pk = rng.integers(0, domain, nb), rng.integers(0, domain, n)
    bcols = [("k", bk, rng.random(nb) > 0.02), ("v", np.arange(nb), None)]
    pcols = [("k", pk, rng.random(n) > 0.02), ("r", np.arange(n), None)]
    got = {}
    for partitioned in (False, True):
        spec = kb.join_spec(jt, probe_out=[1], build_out=[1], radix_bits=3, max_output_rows=1 << 20)
        j = kb.HashJoin(small, spec, partitioned=partitioned, device_budget=device_budget if partitioned else 0)
        build, probe = (dev(kb, cols) for cols in (bcols, pcols))
        failed = {}

        def insist(what, call):
            for free in [1 << 14] + [i << 17 for i in range(1, 300)] + [BUDGET]:
                b = ballast(kb, small, BUDGET, free) if partitioned else None
                try:
                    return call()
                except kb.KrvError as e:
                    assert e.status == kb.NEED_MEMORY
                    failed[what] = failed.get(what, 0) + 1
                finally:
                    if b is not None:
                        b.close()

        def column(r, i):
            c = r.columns[i].cpu().numpy()
            if r.valid[i] is None:
                return c
            return np.where(np.unpackbits(r.valid[i].cpu().numpy(), bitorder="little")[:r.rows] == 1, c, -1)
        insist("build", lambda: j.build_push_device(build))
        j.build_finish()
        pairs = []

        def probe_all():
            arr, sch = kb.ArrowDeviceArray(), kb.ArrowSchema()
            st = kb.check(kb.lib().krv_join_probe_device(j.h, C.byref(probe.dev), C.byref(probe.schema), C.byref(arr), C.byref(sch)))
            return st, kb.DeviceResult(arr, sch)
        st, first = insist("probe", probe_all)
        outs = [first]
        while st == kb.HAVE_MORE_OUTPUT:
            arr, sch = kb.ArrowDeviceArray(), kb.ArrowSchema()
            st = kb.check(kb.lib().krv_join_probe_device(j.h, None, None, C.byref(arr), C.byref(sch)))
            outs.append(kb.DeviceResult(arr, sch))
        outs += list(j.finish_device())
        for r in outs:
            if r.rows:
                pairs.append(column(r, 0) * (nb + 1) + column(r, 1) + 1)
        got[partitioned] = np.sort(np.concatenate(pairs))
        counters = j.counters()
        assert counters["build_rows"] == nb and counters["probe_rows"] == n
        if partitioned:
            assert failed["build"] > 1 and failed["probe"] > 1
        outs = first = r = None
        j.close()
    assert np.array_equal(got[True], got[False])
