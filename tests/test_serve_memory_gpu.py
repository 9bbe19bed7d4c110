"""A request that finds no memory when it is admitted waits; none is lost. Exact."""
import numpy as np
import pytest

from test_join_memory_gpu import BUDGET, ballast, small, status  # noqa: F401 (small: a fixture)
from test_serve_gpu import device_batch, got_of, load

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])
def test_requests_wait_for_memory(kb, small, mode):  # noqa: F811
    n, groups = 60_000, 20_000
    k = np.arange(n)
    srv = kb.Server(small, kb.server_options(mode=mode))
    tids, _keep = load(kb, srv, [(k, k % groups)])
    probes = [k[i::4] for i in range(4)]
    ids = [srv.submit(tids[0], device_batch(kb, [("k", p, None), ("x", p, None)])) for p in probes]
    b = ballast(kb, small, BUDGET, 1 << 14)  # a request's groups take 960 KB
    for _ in range(2):
        assert status(kb, srv.step, True) == kb.NEED_MEMORY
    b.close()
    results = {}
    for _ in range(50):
        srv.step(wait=True)
        while (r := srv.poll()) is not None:
            results[r[0]] = (r[1], got_of(r[2]))
    assert set(results) == set(ids)
    for i, p in zip(ids, probes):
        total = np.bincount(p % groups, p, minlength=groups).astype(np.int64)
        count = np.bincount(p % groups, minlength=groups)
        assert results[i] == (kb.OK, {int(g): (int(total[g]), int(count[g])) for g in np.flatnonzero(count)})
    srv.close()
