"""Snappy streams written element by element (not by a compressor), decoded by
the device against a plain Python decoder: pages small enough for one CTA and
pages of many short elements, which the whole device decodes in windows of
4096 stream bytes and pieces of 16384 output bytes. Literals of every length
form (past a window too), back-references of every offset form, overlapping
and far ones, elements across window and piece ends. Bytes are compared
exactly; streams that do not decode are reported."""
import numpy as np
import pytest

from test_parquet_gpu import _data_page, _varint

pytestmark = pytest.mark.gpu


def write_stream(rng, want, short):
    """About `want` output bytes (a multiple of 8): the stream and its output."""
    out, body = bytearray(), bytearray()

    def literal(n):
        data = rng.integers(0, 256, n, dtype=np.uint8).tobytes()
        if n <= 60:
            body.append((n - 1) << 2)
        else:
            nb = 1 if n <= 256 else 2 if n <= 65536 else 3
            body.append((59 + nb) << 2)
            body.extend((n - 1).to_bytes(nb, "little"))
        body.extend(data)
        out.extend(data)

    def copy(off, n):
        if 4 <= n <= 11 and off < 2048:
            body.extend([((off >> 8) << 5) | ((n - 4) << 2) | 1, off & 255])
        elif off < 65536 and rng.random() < 0.9:
            body.extend([((n - 1) << 2) | 2]), body.extend(off.to_bytes(2, "little"))
        else:
            body.extend([((n - 1) << 2) | 3]), body.extend(off.to_bytes(4, "little"))
        for _ in range(n):
            out.append(out[-off])
    literal(8)
    while len(out) < want:
        r = rng.random()
        if r < 0.45:
            literal(int(rng.integers(1, 9)))
        elif r < 0.6:
            copy(int(rng.integers(1, min(len(out), 9) + 1)), int(rng.integers(1, 65)))  # overlapping
        elif r < 0.98 or short:
            copy(int(rng.integers(1, min(len(out), 70_000) + 1)), int(rng.integers(1, 12)))
        else:
            literal(int(rng.choice([61, 300, 5000, 66_000])))
    literal(8 - len(out) % 8)
    return bytes(_varint(len(out))) + bytes(body), bytes(out)


@pytest.mark.parametrize("want,short", [(64, True), (4000, True), (16_000, False), (100_000, False), (140_000, True),
                                        (500_000, True), (1_000_000, False)])
def test_random_streams(kb, rt, want, short):
    rng = np.random.default_rng(want + short)
    stream, out = write_stream(rng, want, short)
    n = len(out) // 8
    res, _ = kb.parquet_decode_chunk(rt, _data_page(stream, len(out), n), kb.PQ_INT64, kb.PQ_SNAPPY, 0, n, "l")
    assert res.columns[0].cpu().numpy().tobytes() == out


@pytest.mark.parametrize("want", [4000, 300_000])
def test_streams_that_do_not_decode(kb, rt, want):
    rng = np.random.default_rng(want)
    stream, out = write_stream(rng, want, True)
    n = len(out) // 8
    head = len(_varint(len(out)))
    bad = {
        "cut short": stream[:-3],
        "no valid offset": stream[:-9] + bytes([2 << 2 | 2, 0, 0]) + stream[-9:],
        "more output": stream + bytes([0, 1]),
        "offset before the page": stream[:head] + bytes([0, 7, 0x05, 200]) + stream[head:],
    }
    for what, s in bad.items():
        with pytest.raises(kb.KrvError) as e:
            kb.parquet_decode_chunk(rt, _data_page(s, len(out), n), kb.PQ_INT64, kb.PQ_SNAPPY, 0, n, "l")
        assert e.value.status == kb.INVALID_ARGUMENT, what
    res, _ = kb.parquet_decode_chunk(rt, _data_page(stream, len(out), n), kb.PQ_INT64, kb.PQ_SNAPPY, 0, n, "l")
    assert res.columns[0].cpu().numpy().tobytes() == out
