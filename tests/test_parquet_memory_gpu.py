"""A column chunk whose large page is decoded without the device's tables when
they leave the decode no memory. Bytes are compared exactly."""
import numpy as np
import pytest

from test_join_memory_gpu import BUDGET, ballast, small  # noqa: F401 (small: a fixture)
from test_parquet_gpu import _data_page, _varint

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("free", [24 << 20, 12 << 20])  # the tables fit, but nothing beside them; they do not fit
def test_strings_beside_the_tables(kb, small, free):  # noqa: F811
    n = 200_000
    raw = np.zeros((n, 8), np.uint8)  # PLAIN BYTE_ARRAY: length 4, four bytes
    raw[:, 0] = 4
    raw[:, 4:] = np.random.default_rng(1).integers(0, 256, (n, 4))
    elements = np.concatenate([np.full((n, 1), 7 << 2, np.uint8), raw], axis=1)  # a literal of 8 bytes each
    page = _data_page(bytes(_varint(raw.size)) + elements.tobytes(), raw.size, n)
    b = ballast(kb, small, BUDGET, free)
    r, _ = kb.parquet_decode_chunk(small, page, kb.PQ_BYTE_ARRAY, kb.PQ_SNAPPY, 0, n, "z")
    if b is not None:
        b.close()
    assert np.array_equal(r.columns[0].cpu().numpy(), np.arange(n + 1) * 4)
    assert r.heaps[0].cpu().numpy().tobytes() == raw[:, 4:].tobytes()
