"""Index arithmetic of the kernels that can be checked without a GPU: csrc/index_arithmetic.h through the host compiler."""
import ctypes
import os
import subprocess

import pytest

from conftest import PKG


@pytest.fixture(scope="module")
def arithmetic(tmp_path_factory):
    path = tmp_path_factory.mktemp("arithmetic")
    src, so = path / "arithmetic.cpp", path / "arithmetic.so"
    src.write_text('#include "index_arithmetic.h"\n'
                   'extern "C" unsigned places(int row, int first, int groups, int rows) { return clusten::list_places(row, first, groups, rows); }\n'
                   'extern "C" int fit(int n_rows, int m) { return clusten::pair_counts_fit(n_rows, m); }\n')
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-I", os.path.join(PKG, "csrc"), str(src), "-o", str(so)], check=True)
    return ctypes.CDLL(str(so))


@pytest.mark.parametrize("groups", [1, 5, 6, 8])
@pytest.mark.parametrize("rows", [1, 7, 8, 9, 16])
def test_rows_behind_the_last_one_name_nothing(arithmetic, groups, rows):
    """The dense bias of place p of row r is read at r * m + 8 (p - 1): a place in a row that does not exist is a read past the end."""
    arithmetic.places.restype = ctypes.c_uint
    for row in range(16):
        got = [(arithmetic.places(row, first, groups, rows) >> (8 * i)) & 0xff for first in range(0, 28, 4) for i in range(4)]
        assert got == [j + 1 if row < rows and j < groups else 0 for j in range(28)]


def test_pairs_of_lists_are_counted_in_16_bits(arithmetic):
    """n rows in lists of 8 whose m slots all name another target tile are ceil(n / 8) * m pairs."""
    for m in range(1, 65):
        for n in (16, 8184, 8185, 8191, 8192, 9361, 9362, 9216, 10922, 10923, 65000):
            pairs = max(-(-n // 8) * m, n * -(-m // 8))
            assert bool(arithmetic.fit(n, m)) == (pairs < 1 << 16), (n, m)
