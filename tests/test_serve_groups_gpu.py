"""The request server's accumulators at their edges, against numpy: as many
groups as a copy per lane, one copy, one CTA of the first and of the second
launch hold, and one more; too few rows for shared memory to pay; unique dense,
unique sparse and duplicate keys; NULL keys; values at the ends of int64 (exact
sums of 96 and 128 bits, wrapped without ANSI). Exact."""
import numpy as np
import pytest

from test_serve_gpu import device_batch, load, run_all

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", ["dense", "sparse", "dups"])
@pytest.mark.parametrize("groups", [1, 32, 33, 64, 65, 2048, 2049, 7168, 7169])
def test_groups_at_the_edges(kb, rt, layout, groups):
    rng = np.random.default_rng(groups)
    nb = max(groups, 3000)
    k = rng.permutation(nb).astype(np.int64)
    g = (np.arange(nb) % groups).astype(np.int64) * 1_000_003 - 77
    if layout == "sparse":
        k = k * 1_000_003 - 9
    elif layout == "dups":
        k, g = np.concatenate([k, k[:500]]), np.concatenate([g, g[500:1000]])
    srv = kb.Server(rt, kb.server_options(ansi=0, tick_rows=100_000))
    tids, _keep = load(kb, srv, [(k, g)])
    subs, want = [], []
    for n, full in ((1, False), (2047, True), (40_000, False), (4 * 7169 + 5, True), (150_001, True)):
        pk = np.where(rng.random(n) < 0.8, k[rng.integers(0, k.size, n)], -(2**50))
        px = rng.integers(-2**63, 2**63 - 1, n, dtype=np.int64) if full else rng.integers(-9, 9, n)
        valid = rng.random(n) > 0.03 if full else None
        subs.append((tids[0], device_batch(kb, [("k", pk, valid), ("x", px, None)])))
        rows = {}
        for key, grp in zip(k.tolist(), g.tolist()):
            rows.setdefault(key, []).append(grp)
        out = {}
        ok = np.ones(n, bool) if valid is None else valid
        for key, x in zip(pk[ok].tolist(), px[ok].tolist()):
            for grp in rows.get(key, ()):
                s, c = out.get(grp, (0, 0))
                out[grp] = (s + x, c + 1)
        want.append({q: (((s + 2**63) % 2**64) - 2**63, c) for q, (s, c) in out.items()})
    for (status, got), w in zip(run_all(kb, srv, subs), want):
        assert status == kb.OK and got == w
    srv.close()
