"""The kernels' sums in 32-bit words, compiled for the host: exact where a sum
passes the words' end, against Python's integers."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "krishiv-engine_b200", "csrc")
SHIM = """
#include "limbs.h"
extern "C" int add96(uint32_t *w, int64_t x) {
    return krv::sum96_add([w](int p, uint32_t v) { const uint32_t o = w[p]; w[p] = o + v; return o; }, x);
}
"""


@pytest.fixture(scope="module")
def limbs(tmp_path_factory):
    d = tmp_path_factory.mktemp("limbs")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, "-o", str(d / "shim.so"), str(d / "shim.cpp")],
                   check=True)
    lib = C.CDLL(str(d / "shim.so"))
    lib.add96.argtypes = [C.POINTER(C.c_uint32), C.c_int64]
    return lib


@pytest.mark.parametrize("start", [0, 2**95 - 1, 2**95 - 2**63, -(2**95), -(2**95) + 2**63 - 1, 2**64 - 1, -(2**64), 2**32 - 1])
@pytest.mark.parametrize("values", ["up", "down", "mixed"])
def test_sum_of_96_bits_passes_its_end(limbs, start, values):
    rng = np.random.default_rng(7)
    lo, hi = {"up": (2**62, 2**63 - 1), "down": (-2**63, -2**62), "mixed": (-2**63, 2**63 - 1)}[values]
    xs = [int(x) for x in rng.integers(lo, hi, 500, dtype=np.int64)] + [0, 1, -1, 2**63 - 1, -2**63, 2**32, -(2**32)]
    if values == "mixed":
        xs += [2**63 - 1, -2**63] * 20  # back and forth over the end
    w = (C.c_uint32 * 3)(*[(start >> (32 * i)) & 0xFFFFFFFF for i in range(3)])
    total, past = start, 0
    for x in xs:
        past += limbs.add96(w, x)
        total += x
        words = sum(v << (32 * i) for i, v in enumerate(w))
        words -= 2**96 if words >> 95 else 0
        assert words + past * 2**96 == total
