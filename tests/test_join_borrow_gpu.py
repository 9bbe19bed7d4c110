"""A probe of device columns returns when nothing it queued reads them any more:
the caller overwrites them from another stream at once. Exact."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("jt", ["existence", "right_semi", "inner", "left_semi"])
@pytest.mark.parametrize("dup", [1, 2])
def test_probe_columns_are_the_callers_again(kb, rt, jt, dup):
    nb, n = 1000, 50_001
    build = torch.arange(nb, device="cuda").repeat(dup)
    probe = torch.arange(n, device="cuda")
    j = kb.HashJoin(rt, kb.join_spec(jt, probe_out=[0], build_out=[] if jt in ("existence", "left_semi") else [0]))
    j.build_push_device(kb.DeviceBatch([("k", build, None)]))
    j.build_finish()
    batch = kb.DeviceBatch([("k", probe, None)])
    other = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(rt.torch_stream):
        torch.cuda._sleep(200_000_000)  # the probe's kernels wait behind this
    r = j.probe_device(batch)
    with torch.cuda.stream(other):
        probe.fill_(-1)
    other.synchronize()
    rt.synchronize()
    if jt == "right_semi":
        r = next(j.finish_device())
        assert np.array_equal(np.sort(r.columns[0].cpu().numpy()), np.sort(build.cpu().numpy()))
        return
    got = r.columns[0].cpu().numpy()
    if jt == "existence":
        assert np.array_equal(got, np.arange(n))
        hit = np.unpackbits(r.columns[1].cpu().numpy(), bitorder="little")[:n]
        assert np.array_equal(hit, np.arange(n) < nb)
    else:
        assert np.array_equal(np.sort(got), np.sort(np.tile(np.arange(nb), dup if jt == "inner" else 1)))
