"""A batch of more rows than one round of the partitioned aggregate takes
(2^27): keys of an earlier round are the groups they were, checked against
torch's integer sums."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SLICE = 1 << 27  # rows of a round


@pytest.mark.parametrize("rows,groups", [
    (SLICE + 4097, 20_000),        # the cold keys of the first round come again in the second
    (2 * SLICE + 1, 300_000),      # a third round of one row
])
def test_groups_of_earlier_slices_are_found(kb, rt, rows, groups):
    g = torch.Generator(device="cuda")
    g.manual_seed(rows)
    k = torch.randint(0, groups, (rows,), device="cuda", generator=g)
    v = torch.randint(-1000, 1000, (rows,), dtype=torch.int32, device="cuda", generator=g)
    a = kb.HashAggregate(rt, kb.agg_spec(0, [("sum", 1), ("count_star", 0)], expected_groups=groups))
    a.push_device(kb.DeviceBatch([("k", k, None), ("v", v, None)]))
    a.finish()
    r = a.result_device()
    key, total, count = r.columns[:3]
    assert r.rows == groups and int(torch.unique(key).numel()) == groups
    for got, add in ((total, v.long()), (count, torch.ones_like(k))):
        want = torch.zeros(groups, dtype=torch.int64, device="cuda").index_add_(0, k, add)
        assert torch.equal(got, want[key])
