"""Walks over CSR lists that end at the int32 limit (csrc/list_walk.h, compiled for the host)."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parents[1] / "indigo2suite_b200" / "csrc"
SOURCE = r"""
#include "list_walk.h"
extern "C" long walk(unsigned begin, unsigned end, unsigned first, unsigned step, unsigned* out, long cap) {
  long n = 0;
  i2::walk_list(begin, end, first, step, [&](unsigned j) { if (n < cap) out[n] = j; ++n; });
  return n;
}
extern "C" int share(unsigned k, unsigned end, unsigned t, unsigned width) { return i2::window_share(k, end, t, width); }
"""
LIMIT = 2**31 - 1


@pytest.fixture(scope="module")
def walks(tmp_path_factory):
    d = tmp_path_factory.mktemp("walk")
    (d / "walk.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", f"-I{CSRC}", "-o", str(d / "walk.so"),
                    str(d / "walk.cpp")], check=True)
    lib = C.CDLL(str(d / "walk.so"))
    lib.walk.restype = C.c_long
    u = C.c_uint
    lib.walk.argtypes = [u, u, u, u, C.c_void_p, C.c_long]
    lib.share.argtypes = [u, u, u, u]
    return lib


@pytest.mark.parametrize("end", [100, LIMIT - 1023, LIMIT - 1, LIMIT])
@pytest.mark.parametrize("length", [0, 1, 2, 31, 33, 255, 257, 1025, 5000])
def test_walks_stay_inside_lists_that_end_at_the_limit(walks, end, length):
    length = min(length, end)
    begin = end - length
    for width in (1, 32, 256):
        seen = []
        for t in range(width):
            out = np.zeros(length + 8, np.uint32)
            n = walks.walk(begin, end, t, width, out.ctypes.data, len(out))
            assert n == len(range(begin + t, end, width))
            seen.append(out[:n])
        np.testing.assert_array_equal(np.sort(np.concatenate(seen)), np.arange(begin, end))
        if width == 1:
            continue
        seen = []
        for k in range(begin, end, 4 * width):  # windows, as the scans take them
            for t in range(width):
                m = walks.share(k, end, t, width)
                assert 0 <= m <= 4
                seen += [k + t + r * width for r in range(m)]
        np.testing.assert_array_equal(np.sort(np.array(seen, np.int64)), np.arange(begin, end))


def test_a_list_begun_behind_its_end_is_empty(walks):
    # the links after a vertex's first two start two entries on, also at the limit
    out = np.zeros(4, np.uint32)
    for end in (0, 1, LIMIT):
        for first in (0, 31, 255):
            assert walks.walk(end + 2, end, first, 32, out.ctypes.data, 4) == 0
