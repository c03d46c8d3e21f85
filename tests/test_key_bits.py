"""Packing of vertex pairs into sort keys at the widths an ID can take (csrc/key_bits.h, compiled for the host)."""
import ctypes as C
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "indigo2suite_b200" / "csrc"
SOURCE = r"""
#include "key_bits.h"
typedef unsigned long long u64;
extern "C" void widths(int n, int* shift, int* bits, u64* drop) {
  const i2::KeyBits k = i2::key_bits(n);
  *shift = k.shift, *bits = k.bits, *drop = k.drop;
}
extern "C" u64 key(int n, u64 u, u64 v) { return i2::key_bits(n).key(u, v); }
extern "C" u64 hi(int n, u64 k) { return i2::key_bits(n).hi(k); }
extern "C" u64 lo(int n, u64 k) { return i2::key_bits(n).lo(k); }
"""


@pytest.fixture(scope="module")
def keys(tmp_path_factory):
    d = tmp_path_factory.mktemp("keys")
    (d / "keys.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", f"-I{CSRC}", "-o", str(d / "keys.so"),
                    str(d / "keys.cpp")], check=True)
    lib = C.CDLL(str(d / "keys.so"))
    u64 = C.c_ulonglong
    for f in (lib.key, lib.hi, lib.lo):
        f.restype = u64
    lib.key.argtypes = [C.c_int, u64, u64]
    lib.hi.argtypes = lib.lo.argtypes = [C.c_int, u64]
    return lib


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 2**16 - 1, 2**16, 2**16 + 1, 2**30 - 1, 2**30, 2**30 + 1, 2**31 - 2,
                               2**31 - 1])
def test_keys_round_trip_in_order_below_the_drop_mark(keys, n):
    shift, bits, drop = C.c_int(), C.c_int(), C.c_ulonglong()
    keys.widths(n, C.byref(shift), C.byref(bits), C.byref(drop))
    ids = sorted({x for x in (0, 1, n // 2, n - 2, n - 1) if 0 <= x < n})
    last = -1
    for u in ids:
        for v in ids:
            k = keys.key(n, u, v)
            assert (keys.hi(n, k), keys.lo(n, k)) == (u, v)
            assert last < k  # ascending by (u, v)
            last = k
    assert keys.key(n, n - 1, n - 1) < drop.value < 1 << bits.value
    assert bits.value <= 64 and drop.value == keys.key(n, n, 0)
    # the list of vertex u ends where the keys of u + 1 begin, up to the mark
    assert keys.key(n, n - 1, n - 1) < keys.key(n, n, 0)
