"""The part of a round that belongs to a row, at the distances where a 32-bit one
wraps around: the entries that a row's lane adds lie inside the round, and they
are the row's.  Compiled for the host: arrays of 2^31 entries are not needed."""

import ctypes
import itertools
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "asc_cpp_b200",
                    "csrc")
SOURCE = """
#include "round_part.h"
extern "C" void part(int64_t b, int64_t e, int64_t w, int length, int* out) {
  const ascb::RoundPart p = ascb::round_part(b, e, w, length);
  out[0] = p.from;
  out[1] = p.to;
}
"""


@pytest.fixture(scope="module")
def part(tmp_path_factory):
    where = tmp_path_factory.mktemp("round_part")
    (where / "part.cc").write_text(SOURCE)
    lib = str(where / "part.so")
    subprocess.run(["g++", "-std=c++20", "-O2", "-shared", "-fPIC", "-I", CSRC,
                    str(where / "part.cc"), "-o", lib], check=True)
    fn = ctypes.CDLL(lib).part
    fn.argtypes = [ctypes.c_int64] * 3 + [ctypes.c_int, ctypes.POINTER(ctypes.c_int)]
    fn.restype = None

    def call(b, e, w, length):
        out = (ctypes.c_int * 2)()
        fn(b, e, w, length, out)
        return out[0], out[1]

    return call


DISTANCES = [0, 1, 127, 128, 129, 2**31 - 1, 2**31, 2**31 + 200, 2**32 - 1, 2**32, 2**32 + 5,
             2**40]


@pytest.mark.parametrize("w", [0, 128, 2**31, 2**33 + 128])
def test_part_is_the_rows_share_of_the_round(part, w):
    points = sorted({w + s * d for d in DISTANCES for s in (1, -1) if w + s * d >= 0})
    for b, e in itertools.combinations_with_replacement(points, 2):
        expect = range(max(b, w), min(e, w + 128))
        start, stop = part(b, e, w, 128)
        assert 0 <= start <= 128 and 0 <= stop <= 128
        assert [w + q for q in range(start, stop)] == list(expect)
