"""The powers of x that carry a slice's share of the PNG chunk CRC past the
slices behind it (png_crc.h), for every digit up to the largest file the
writer accepts (a zlib stream of 2^31 - 1 bytes), against square and multiply
on Python integers."""
import ctypes
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "zigtrace_b200" / "csrc"
POLY = 0x104C11DB7  # x^32 + x^26 + ... + 1
SLICE_BITS = 8 * 8192

PROGRAM = """
#include "png_crc.h"
static const zt::CrcPowers P = zt::make_crc_powers();
extern "C" unsigned following(unsigned n) { return zt::crc_slices_power(P, n, zt::crc_mulmod); }
extern "C" unsigned long long most_slices() { return zt::kPngMaxSlices; }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("crc")
    (d / "crc.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", f"-I{CSRC}", "-o", str(d / "crc.so"),
                    str(d / "crc.cpp")], check=True)
    return ctypes.CDLL(str(d / "crc.so"))


def _mul(a, b):
    r = 0
    while b:
        if b & 1:
            r ^= a
        b >>= 1
        a <<= 1
        if a >> 32:
            a ^= POLY
    return r


def _xpow(n):
    r, q = 1, 2
    while n:
        if n & 1:
            r = _mul(r, q)
        q, n = _mul(q, q), n >> 1
    return int(f"{r:032b}"[::-1], 2)  # bit 31 is the coefficient of x^0


def test_every_count_of_following_slices(lib):
    lib.following.restype = ctypes.c_uint32
    lib.most_slices.restype = ctypes.c_uint64
    top = lib.most_slices() - 1
    assert top == (41 + (1 << 31) - 1 + 16 + 31 + 8191) // 8192 - 1 == 262144
    for n in (0, 1, 63, 64, 65, 4095, 4096, 4097, 262143, top):
        assert lib.following(n) == _xpow(SLICE_BITS * n), n
