"""The columns of the partitioned join's output are memory of their own: writing
to one changes no other, of the same batch or of another."""
import numpy as np
import pytest

from test_grace_gpu import dev

pytestmark = pytest.mark.gpu


def test_padded_columns_share_no_memory(kb, rt):
    rng = np.random.default_rng(2)
    nb, n = 20_000, 200_000
    j = kb.HashJoin(rt, kb.join_spec("left_outer", probe_out=[0, 1], build_out=[0, 1, 2], radix_bits=3), partitioned=True,
                    device_budget=64 << 20)
    j.build_push_device(dev(kb, [("k", rng.integers(0, 1000, nb), None), ("a", np.arange(nb), None),
                                 ("b", np.arange(nb, dtype=np.int32), None)]))
    j.build_finish()
    outs = []
    for half in np.array_split(np.arange(n), 2):  # keys that the filter rules out, keys that are NULL
        k = rng.integers(10**6, 10**7, half.size)
        outs += list(j.probe_device_all(dev(kb, [("k", k, rng.random(half.size) > 0.1), ("r", half, None)])))
    outs += list(j.finish_device())
    spans = []
    for o in outs:
        for t in [c for c in o.columns if c is not None] + [v for v in o.valid if v is not None]:
            spans.append((t.data_ptr(), t.data_ptr() + t.numel() * t.element_size()))
    assert sum(o.rows for o in outs) == n
    spans.sort()
    assert all(a[1] <= b[0] for a, b in zip(spans, spans[1:]))
