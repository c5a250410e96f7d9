"""The rules that choose between the bit rows and the incidence lists
(csrc/host/form.h), on the CPU, at their edges."""
import ctypes as C
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DIRECT, ONDEMAND = 0, 1
U64 = 2 ** 64 - 1

SOURCE = """
#include "form.h"
extern "C" int pay(int v, uint64_t words, uint64_t lists) { return n34::rows_pay(v, words, lists); }
extern "C" uint64_t least(int v, uint64_t m) { return n34::rows_least_triangles(v, m); }
extern "C" int fit(uint64_t cells, uint64_t T, uint64_t m, int rounds, uint64_t room)
{ return n34::rows_fit(cells, T, m, rounds != 0, room); }
"""


@pytest.fixture(scope="module")
def form(tmp_path_factory):
    d = tmp_path_factory.mktemp("form")
    (d / "form.cpp").write_text(SOURCE)
    so = str(d / "form.so")
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "include"), "-I",
                    os.path.join(ROOT, "gpu-nucleus34_b200", "csrc", "host"), "-o", so, str(d / "form.cpp")], check=True)
    L = C.CDLL(so)
    L.pay.argtypes = [C.c_int, C.c_uint64, C.c_uint64]
    L.least.argtypes, L.least.restype = [C.c_int, C.c_uint64], C.c_uint64
    L.fit.argtypes = [C.c_uint64, C.c_uint64, C.c_uint64, C.c_int, C.c_uint64]
    return L


@pytest.mark.parametrize("lists", [0, 1, 1000, 10 ** 9 + 1, 10 ** 13])
def test_words_against_list_entries(form, lists):
    for variant, limit in ((DIRECT, lists + lists // 2), (ONDEMAND, 3 * lists + lists // 2 + 10 ** 8)):
        assert form.pay(variant, limit, lists) and not form.pay(variant, limit + 1, lists)


def test_least_triangles(form):
    assert form.least(DIRECT, 0) == form.least(ONDEMAND, 0) == 0
    assert form.least(DIRECT, 10 ** 7) == 5 * 10 ** 6
    assert form.least(ONDEMAND, 1 << 23) == 0 and form.least(ONDEMAND, (1 << 23) + 16) == ((1 << 23) + 16) // 16


def test_in_row_cells_stay_steppable(form):
    """k_in_firsts steps a 32-bit cell index by 32 until it passes the last cell: the
    step past any accepted number of cells must not wrap."""
    for cells in (0xffffffff, 0xffffffff - 30, 2 ** 32, 2 ** 33):
        assert not form.fit(cells, 0, 0, 0, U64)
    most = 0xffffffff - 31
    assert form.fit(most, 0, 0, 0, U64)
    last_start = (most - 1) // 32 * 32 + 31  # any start below `most`, at any offset from the first cell
    assert last_start < 2 ** 32 and most - 1 + 32 < 2 ** 32


def test_room(form):
    cells, T, m = 1000, 10 ** 6, 10 ** 5
    for rounds in (0, 1):
        need = 16 * cells + (24 if rounds else 20) * T + T // 8 + 16 * m + (1 << 20)
        assert form.fit(cells, T, m, rounds, need) and not form.fit(cells, T, m, rounds, need - 1)
