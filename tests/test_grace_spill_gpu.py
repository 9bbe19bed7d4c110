"""The partitioned join's row movement against the unpartitioned join: build
rows scattered straight into the tables' arenas (grown without a size hint,
reserved with one), rows that leave for host memory side by side and come back
piece by piece, padded rows beside shared NULL columns. 4- and 8-byte columns,
projections without the key or without build columns, calls of several slices,
budgets under which nothing, some and most of the rows spill. Exact."""
import collections

import numpy as np
import pytest

from test_grace_gpu import dev, rows_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("probe_out,build_out", [([0, 1, 2], [1, 2]), ([2], []), ([1], [0, 1])])
@pytest.mark.parametrize("jt", ["left_outer", "inner"])
@pytest.mark.parametrize("budget,hint", [(0, 0), (8 << 20, 1), (8 << 20, 0), (2 << 20, 1), (400 << 10, 0)])
def test_partitioned_rows_move_intact(kb, rt, jt, budget, hint, probe_out, build_out):
    rng = np.random.default_rng(budget + hint)
    nb, n = 70_001, 200_003
    bk, bval = rng.integers(0, 140_000, nb), rng.random(nb) > 0.02
    pk, pval = rng.integers(0, 140_000, n), rng.random(n) > 0.02
    bcols = [("k", bk, bval), ("i", rng.integers(-2**31, 2**31 - 1, nb).astype(np.int32), None), ("v", np.arange(nb), None)]
    pcols = [("k", pk, pval), ("i", rng.integers(-2**31, 2**31 - 1, n).astype(np.int32), None), ("r", np.arange(n), None)]
    got = {}
    for partitioned in (False, True):
        spec = kb.join_spec(jt, probe_out=probe_out, build_out=build_out, radix_bits=4, max_output_rows=60_000,
                            build_rows_hint=nb if hint and partitioned else 0)
        j = kb.HashJoin(rt, spec, partitioned=partitioned, device_budget=budget)
        for s in np.array_split(np.arange(nb), 3):
            j.build_push_device(dev(kb, [(c, a[s], None if v is None else v[s]) for c, a, v in bcols]))
        j.build_finish()
        rows = []
        for s in np.array_split(np.arange(n), 2):
            outs = list(j.probe_device_all(dev(kb, [(c, a[s], None if v is None else v[s]) for c, a, v in pcols])))
            for r in outs:
                rows += rows_of(r)
        for r in j.finish_device():
            rows += rows_of(r)
        got[partitioned] = collections.Counter(rows)
        if partitioned and budget in (2 << 20, 400 << 10):
            assert j.spilled_partitions() > 0
    assert got[True] == got[False]
