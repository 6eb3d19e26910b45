"""The decisions that need only a plan's numbers (csrc/spmm_rules.h), on the graphs that were timed for them."""
import ctypes
import os
import subprocess

import pytest

from conftest import PKG

SM = 148


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    src = d / "rules.cpp"
    src.write_text("""#include "spmm_rules.h"
extern "C" int few_form(int64_t units, int64_t rows, int64_t nnz, int64_t longest, int sm, int width) { return agcn::spmm_few_form({units, rows, nnz, longest, sm}, width); }
extern "C" int octets(int64_t units, int64_t nnz, int wide, int sm, int width, int columns) { return agcn::spmm_octets({units, 8 * units, nnz, wide != 0, sm}, width, columns); }
extern "C" int faults(const int64_t *words, int64_t most) { return agcn::plan_faults(words, most); }
""")
    lib = str(d / "librules.so")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I" + os.path.join(PKG, "csrc"), str(src), "-o", lib])
    dll = ctypes.CDLL(lib)
    dll.few_form.argtypes = [ctypes.c_int64] * 4 + [ctypes.c_int, ctypes.c_int]
    dll.octets.argtypes = [ctypes.c_int64] * 2 + [ctypes.c_int] * 4
    dll.faults.argtypes = [ctypes.POINTER(ctypes.c_int64), ctypes.c_int64]
    return dll


# thread blocks, rows, nonzeros, longest row; up to how many columns (of 32, 64, 128) products were measured no slower with three
# thread blocks per SM than with four (0: plans of pieces of 128, which lose at some width of each class, and beyond four per SM)
TIMED = {
    "power law 16384 x 9": (414, 16384, 155534, 2383, 128),
    "power law 25000 x 7": (519, 25000, 184356, 3534, 128),
    "power law 28000 x 6": (520, 28000, 176402, 3426, 128),
    "power law 35000 x 5": (582, 35000, 183644, 3420, 128),
    "power law 30000 x 9": (562, 30000, 285082, 4406, 128),
    "power law 24000 x 12": (550, 24000, 305212, 3718, 128),
    "skewed 20000 x 11": (567, 20000, 212738, 3641, 128),
    "skewed 22000 x 14": (592, 22000, 298821, 4007, 128),
    "power law 20000 x 10": (552, 20000, 211282, 2963, 64),
    "power law 18000 x 12": (585, 18000, 228918, 2862, 64),
    "power law 20000 x 15": (548, 20000, 317886, 3178, 64),
    "power law 16384 x 20": (579, 16384, 347708, 2708, 32),
    "power law 18000 x 18": (581, 18000, 344672, 2908, 32),
    "power law 20000 x 16": (581, 20000, 340234, 3191, 32),
    "skewed 12000 x 20": (564, 12000, 230524, 2199, 32),
    "skewed 16000 x 22": (590, 16000, 338397, 2922, 32),
    "power law 16384 x 25": (559, 16384, 434114, 2742, 0),
    "power law 23000 x 18": (592, 23000, 439086, 3747, 0),
    "power law 25000 x 14": (644, 25000, 371044, 3909, 0),
}


@pytest.mark.parametrize("graph", TIMED)
def test_three_blocks_per_sm_where_they_were_measured_faster(rules, graph):
    units, rows, nnz, longest, widest = TIMED[graph]
    for width in (16, 20, 32, 33, 60, 64, 65, 100, 128):
        form = rules.few_form(units, rows, nnz, longest, SM, width)
        assert form == (3 if width <= widest else 4), width


# thread blocks, nonzeros, the widths that were measured faster with 32-byte loads or no slower, those that were slower
OCTETS = {
    "dense 13000 x 180": (985, 2_340_000, (), (40, 64, 72, 88, 96, 112, 127, 128)),
    "dense 10000 x 250": (1163, 2_500_000, (), (40, 72, 80, 96, 109, 128)),
    "dense 9000 x 400": (1600, 3_600_000, (), (72, 93, 96, 104, 127)),
    "dense 20000 x 250": (2077, 5_000_000, (72, 77, 88, 96, 103, 112, 127, 128), (40, 48, 64)),
    "dense 60000 x 100": (2635, 6_000_000, (69, 85, 96, 109, 128), (40, 64)),
    "dense 60000 x 150": (3899, 9_000_000, (69, 80, 96, 112, 128), (37, 40, 45, 48, 56, 64)),
    "dense 60000 x 250": (6362, 15_000_000, (37, 40, 45, 48, 69, 88, 96, 128), (56, 64)),
    "power law 90000 x 12": (1124, 1_170_000, (69, 72, 77, 93, 96, 104, 112, 120, 128), (40, 64, 101, 103, 109, 119, 125, 127)),
    "power law 120000 x 10": (1445, 1_320_000, (72, 85, 96, 104, 128), (103, 110, 118, 126)),
    "skewed 100000 x 30": (1916, 3_000_000, (69, 88, 96, 112, 128), (48, 109, 127)),
    "power law 600000 x 15": (7731, 9_600_000, (37, 40, 48, 69, 72, 85, 88), (56, 64, 93, 96, 109, 128)),
}


@pytest.mark.parametrize("graph", OCTETS)
def test_32_byte_loads_where_they_were_measured_faster(rules, graph):
    units, nnz, faster, slower = OCTETS[graph]
    for columns in faster + slower:
        assert rules.octets(units, nnz, 0, SM, (columns + 7) // 8 * 8, columns) == (columns in faster), columns
        # five blocks per SM otherwise: products of few units keep those from 97 columns on
        if units <= 20 * SM and columns > 96:
            assert not rules.octets(units, nnz, 1, SM, (columns + 7) // 8 * 8, columns), columns


@pytest.mark.parametrize("words,most,faults", [
    ((5, 0, 800, 40, 0, 0, 0, 0), 800, 0), ((5, 0, 801, 40, 0, 0, 0, 0), 800, 16),          # pieces that do not fit are an error by themselves
    ((5, 0, 801, 40, 0, 0, 0, 0), 2**63 - 1, 0), ((0, 0, 0, 0, 0, 0, 0, 1), 800, 8), ((0, 0, 900, 0, 1, 0, 1, 0), 800, 5)])
def test_what_the_plan_kernel_reports(rules, words, most, faults):
    assert rules.faults((ctypes.c_int64 * 8)(*words), most) == faults
