"""The partition of the line solves of one instance (linear_system_solvers_gb300/csrc/adi_split.hpp), compiled
on the host and checked without a GPU."""
import os
import subprocess
import tempfile

import pytest

from conftest import ROOT

SRC = os.path.join(ROOT, "tests", "cpp", "adi_split_t.cpp")


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


@pytest.mark.parametrize("nx,ny", [(4, 4), (100, 50), (400, 200), (4096, 2048), (400000, 8), (8, 400000), (1 << 28, 4), (4, 1 << 28)])
def test_product_tables_stay_below_the_line_tables(splits, nx, ny):
    """The products of a sweep take less than one line table of the same direction: a chunk has at least four
    rows and two values, and at most one row of chunks is padding."""
    ld = (ny + 3) // 4 * 4
    s, v = splits([(0, nx - 2, 0, ld), (1, ny, 0, nx)])
    for sp, rows, stride in ((s, nx - 2, ld), (v, ny, nx)):
        assert sp.table == sp.tiles * (2 * sp.PC + sp.groups) * stride
        padded = sp.tiles * sp.PC * sp.R
        assert rows <= padded < rows + sp.PC * sp.R
        assert sp.table <= padded * stride * 3 // sp.R
