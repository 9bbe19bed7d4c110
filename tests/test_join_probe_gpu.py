"""The probe kernel at the edges of its tiles (1024 probe rows) and staging
windows (1024 pairs), against the oracle: every lookup form (dense index,
unique keys, chains, rows only), ragged and empty batches, one key with a
chain longer than a window, NULL keys, and payload columns of 1-, 4-, 8- and
16-byte values with NULLs. Rows are compared exactly."""
import collections

import numpy as np
import pyarrow as pa
import pytest

from helpers import batch, concat

pytestmark = pytest.mark.gpu

TYPE_ID = {"inner": 0, "left_outer": 1, "left_semi": 2, "left_anti": 3, "null_aware_anti": 4, "right_outer": 8,
           "full_outer": 9}
SPREAD = 0x9E3779B97F4A7C15


def keys(form, rng, n, build):
    if form == "dense":
        return (rng.permutation(n) if build else rng.integers(0, 1500, n)).astype(np.int64)
    if form == "unique":
        k = rng.permutation(n) if build else rng.integers(0, 1500, n)
        return (k.astype(np.uint64) * np.uint64(SPREAD)).astype(np.int64)
    k = rng.integers(0, 700, n).astype(np.int64)
    if build:
        k[: n // 2] = 3  # a chain longer than a staging window
    elif n:
        k[k == 3] = 4
        k[n // 2] = 3  # probed once
    return k


@pytest.mark.parametrize("form", ["dense", "unique", "chains"])
@pytest.mark.parametrize("jt", list(TYPE_ID))
def test_tiles_and_windows(kb, rt, oracle, jt, form):
    rng = np.random.default_rng(len(form) * 100 + TYPE_ID[jt])
    nb = 3000 if form == "chains" else 1000
    bk = keys(form, rng, nb, True)
    bmask = rng.random(nb) < 0.02 if form == "chains" and jt != "null_aware_anti" else np.zeros(nb, dtype=bool)
    v4 = pa.array(rng.integers(-2**31, 2**31 - 1, nb).astype(np.int32), mask=rng.random(nb) < 0.1)
    dec = pa.array([int(x) * 10**20 for x in rng.integers(-1000, 1000, nb)], type=pa.decimal128(38, 2))
    build = batch(k=pa.array(bk, mask=bmask), bid=pa.array(np.arange(nb, dtype=np.int64)), v=v4, dec=dec)
    for n in (0, 1, 31, 1023, 1024, 1025, 5003):
        pk = keys(form, rng, n, False)
        pmask = rng.random(n) < 0.03
        small = pa.array(rng.integers(0, 255, n).astype(np.uint8), mask=rng.random(n) < 0.2)
        probe = batch(k=pa.array(pk, mask=pmask), pid=pa.array(np.arange(n, dtype=np.int64)), s=small)
        j = kb.HashJoin(rt, kb.join_spec(jt))
        j.build_push(build)
        j.build_finish()
        t = concat(j.probe(probe) + j.finish())
        p, b = oracle.hash_join(TYPE_ID[jt], [(bk, (~bmask).astype(np.uint8), False)],
                                [(pk, (~pmask).astype(np.uint8), False)], null_safe=[0])
        semi = jt in ("left_semi", "left_anti", "null_aware_anti")
        sp, bv, bd = small.to_pylist(), v4.to_pylist(), dec.to_pylist()
        want = collections.Counter()
        for x, y in zip(p.tolist(), b.tolist()):
            left = (x, int(pk[x]) if not pmask[x] else None, sp[x]) if x >= 0 else (None, None, None)
            right = () if semi else (y, bv[y], bd[y]) if y >= 0 else (None, None, None)
            want[left + right] += 1
        names = ["pid", "k", "s"] + ([] if semi else ["bid", "v", "dec"])
        cols = [t.column(t.schema.get_field_index(c) if c != "k" else 0).to_pylist() for c in names] if t is not None else []
        got = collections.Counter(zip(*cols)) if cols else collections.Counter()
        assert got == want, (jt, form, n)


def test_null_safe_null_is_not_zero(kb, rt, oracle):
    """A `<=>` key: NULL matches NULL and not the value 0 (one int64 key)."""
    for jt in ("inner", "left_outer", "left_semi"):
        bk, bm = np.array([0, 0, 5], dtype=np.int64), np.array([1, 0, 1], dtype=np.uint8)
        pk, pm = np.array([0, 0, 5, 7], dtype=np.int64), np.array([1, 0, 1, 0], dtype=np.uint8)
        j = kb.HashJoin(rt, kb.join_spec(jt, null_safe=[True]))
        j.build_push(batch(k=pa.array(bk, mask=bm == 0), bid=pa.array(np.arange(3, dtype=np.int64))))
        j.build_finish()
        t = concat(j.probe(batch(k=pa.array(pk, mask=pm == 0), pid=pa.array(np.arange(4, dtype=np.int64)))))
        p, b = oracle.hash_join(TYPE_ID[jt], [(bk, bm, False)], [(pk, pm, False)], null_safe=[1])
        bid = t.column("bid").to_pylist() if jt != "left_semi" else [None] * t.num_rows
        got = collections.Counter((x, -1 if y is None else y) for x, y in zip(t.column("pid").to_pylist(), bid))
        assert got == collections.Counter(zip(p.tolist(), b.tolist())), jt
