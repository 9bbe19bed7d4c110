"""Tiles of more output rows than are staged at once (2048 of 1024 probe rows),
against numpy: one chain longer than several windows, tiles at the edge, chains
of even and of very different lengths, ragged last tiles; NULLs in the payload
columns, padded rows, a residual filter. Every (probe row, build row) pair is
compared, with its values and their validity."""
import numpy as np
import pytest

from test_grace_gpu import dev

pytestmark = pytest.mark.gpu


def chains(case, rng):
    """Build rows per key, and the probe rows' keys."""
    if case == "one":      # a chain of five windows, probed once, among rows without a match
        return [5 * 2048 + 7], np.where(np.arange(1500) == 700, 0, 1)
    if case == "edge":     # tiles of 2047, 2048 and 2049 output rows
        pk = np.ones(3 * 1024, np.int64)
        pk[0], pk[2 * 1024] = 0, 2
        return [1, 2, 3], pk
    if case == "even":
        return [9] * 400, rng.integers(0, 500, 4097)
    return rng.integers(0, 2, 300) * rng.integers(1, 1200, 300) ** 2 // 1200, rng.integers(0, 320, 2050)  # skewed


@pytest.mark.parametrize("filtered", [False, True])
@pytest.mark.parametrize("jt", ["inner", "left_outer", "full_outer"])
@pytest.mark.parametrize("case", ["one", "edge", "even", "skewed"])
def test_long_chains(kb, rt, case, jt, filtered):
    rng = np.random.default_rng(len(case) + 10 * len(jt))
    per_key, pk = chains(case, rng)
    bk = rng.permutation(np.repeat(np.arange(len(per_key)), per_key))
    nb, n = bk.size, pk.size
    bval, pval = rng.random(nb) > 0.3, rng.random(n) > 0.3
    v, w = rng.integers(0, 100, nb).astype(np.int32), rng.integers(0, 2**40, n)
    spread = np.int64(0x1E3779B97F4A7C15)
    j = kb.HashJoin(rt, kb.join_spec(jt, probe_out=[1, 2], build_out=[1, 2]),
                    filter=[(("build", 1), ">=", 2)] if filtered else None)
    j.build_push_device(dev(kb, [("k", bk * spread, None), ("b", np.arange(nb), None), ("v", v, bval)]))
    j.build_finish()
    outs = list(j.probe_device_all(dev(kb, [("k", pk * spread, None), ("p", np.arange(n), None), ("w", w, pval)])))
    outs += list(j.finish_device())

    def column(i, none):
        parts = []
        for r in outs:
            if r.rows == 0:
                continue
            c, bits = r.columns[i].cpu().numpy().astype(np.int64), r.valid[i]
            if bits is not None:
                c = np.where(np.unpackbits(bits.cpu().numpy(), bitorder="little")[:r.rows] == 1, c, none)
            parts.append(c)
        return np.concatenate(parts) if parts else np.zeros(0, np.int64)
    p, ww, b, vv = (column(i, -1) for i in range(4))
    # expected pairs
    order = np.argsort(bk, kind="stable")
    lo, hi = np.searchsorted(bk[order], pk, "left"), np.searchsorted(bk[order], pk, "right")
    wp = np.repeat(np.arange(n), hi - lo)
    wb = order[np.arange(wp.size) - np.repeat(np.cumsum(hi - lo) - (hi - lo), hi - lo) + np.repeat(lo, hi - lo)]
    if filtered:
        keep = wb >= 2
        wp, wb = wp[keep], wb[keep]
    if jt != "inner":
        miss = np.setdiff1d(np.arange(n), wp)
        wp, wb = np.concatenate([wp, miss]), np.concatenate([wb, np.full(miss.size, -1)])
    if jt == "full_outer":
        miss = np.setdiff1d(np.arange(nb), wb)
        wp, wb = np.concatenate([wp, np.full(miss.size, -1)]), np.concatenate([wb, miss])
    assert p.size == wp.size
    got, want = np.lexsort((b, p)), np.lexsort((wb, wp))
    assert np.array_equal(p[got], wp[want]) and np.array_equal(b[got], wb[want])
    assert np.array_equal(ww, np.where((p >= 0) & pval[p], w[p], -1))
    assert np.array_equal(vv, np.where((b >= 0) & bval[b], v[b], -1))
