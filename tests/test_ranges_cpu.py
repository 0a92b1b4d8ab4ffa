"""The ends of pieces at the last positions that a matrix may have (csrc/ranges.h, compiled for the host), against
64-bit arithmetic."""
import ctypes
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
LAST = 2 ** 31 - 2  # entries of the largest matrix


@pytest.fixture(scope="module")
def ranges(tmp_path_factory):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("ranges")
    (d / "r.cpp").write_text('#include "ranges.h"\n'
                             'extern "C" int piece_end(int b, int l, int e) { return gbk::piece_end(b, l, e); }\n'
                             'extern "C" int pieces_of(int n, int l) { return gbk::pieces_of(n, l); }\n'
                             'extern "C" int look_ahead(long long n) { return gbk::can_look_ahead(n); }\n')
    subprocess.run([cxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-ftrapv", "-I", str(ROOT / "gb_kun_b200" / "csrc"),
                    str(d / "r.cpp"), "-o", str(d / "r.so")], check=True)
    return ctypes.CDLL(str(d / "r.so"))


@pytest.mark.parametrize("length", [1, 32, 64, 128, 256, 2048])
def test_pieces_cover_the_last_entries(ranges, length):
    for end in (LAST, LAST - 1, LAST - length, length, 1):
        for beg in {max(0, end - k) for k in (0, 1, length - 1, length, length + 1, 3 * length)}:
            assert ranges.piece_end(beg, length, end) == min(beg + length, end)
    for n in (0, 1, length - 1, length, length + 1, LAST - 1, LAST):
        assert ranges.pieces_of(n, length) == -(-n // length)


def test_look_ahead_stays_in_31_bits(ranges):
    # the degree bins form positions up to a chunk of 2,048 entries past the last one
    ranges.look_ahead.argtypes = [ctypes.c_longlong]
    for n in (0, 1, LAST - 8192, LAST - 4096, LAST - 4095, LAST - 2048, LAST - 1, LAST):
        if ranges.look_ahead(n):
            assert n + 2048 + 256 <= 2 ** 31 - 1
    assert ranges.look_ahead(LAST - 8192) and not ranges.look_ahead(LAST)
