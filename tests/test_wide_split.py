"""The partition of the line solves of one instance (linear_system_solvers_gb300/csrc/adi_split.hpp), compiled on
the host and checked without a GPU."""
import os
import subprocess
import tempfile

import pytest

from conftest import ROOT

SRC = os.path.join(ROOT, "tests", "cpp", "adi_split_t.cpp")
SMS = 152


class Split:
    def __init__(self, line):
        (self.L, self.PC, self.R, self.gs, self.tiles, self.groups, self.words, self.table) = (int(q) for q in line.split())


@pytest.fixture(scope="module")
def splits():
    out = os.path.join(tempfile.mkdtemp(), "adi_split_t")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "linear_system_solvers_gb300", "csrc"), SRC, "-o", out],
                   check=True, capture_output=True, text=True)

    def ask(queries):
        res = subprocess.run([out], input="\n".join(" ".join(str(int(x)) for x in q) for q in queries), check=True,
                             capture_output=True, text=True)
        return [Split(ln) for ln in res.stdout.splitlines()]

    return ask


def pitch(ny):
    return (ny + 3) // 4 * 4


def both(splits, nx, ny, word=8, ps=0, pv=0):
    return splits([(0, nx - 2, ny - 2, ps, SMS, word, pitch(ny)), (1, ny, nx - 2, pv, SMS, word, nx)])


@pytest.mark.parametrize("nx,ny", [(4, 4), (100, 50), (400, 200), (4096, 2048), (400000, 8), (8, 400000), (1 << 28, 4), (4, 1 << 28)])
def test_product_tables_stay_below_the_line_tables(splits, nx, ny):
    """The products of a sweep take less than one line table of the same direction: a chunk has at least four
    rows and two values, and at most one row of chunks is padding."""
    s, v = both(splits, nx, ny)
    for sp, rows, stride in ((s, nx - 2, pitch(ny)), (v, ny, nx)):
        assert sp.table == sp.tiles * (2 * sp.PC + sp.groups) * stride
        padded = sp.tiles * sp.PC * sp.R
        assert rows <= padded < rows + sp.PC * sp.R
        assert sp.table <= padded * stride * 3 // sp.R


@pytest.mark.parametrize("rows,lines", [(7000, 6), (7000, 302), (7000, 306), (7000, 1216), (7000, 1217), (2049, 4000)])
def test_few_long_lines_take_more_chunks(splits, rows, lines):
    for word in (4, 8):
        (s,) = splits([(0, rows, lines, 0, SMS, word, lines)])
        if -(-lines // 8) > SMS:
            assert (s.L, s.PC) == (8, 32)
        else:
            assert s.PC == 128 and s.L == (2 if word == 8 and lines <= 2 * SMS else 4)
