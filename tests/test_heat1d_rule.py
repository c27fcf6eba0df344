"""Which FP64 lines take the sweep through memory (linear_system_solvers_gb300/csrc/heat1d_schedule.hpp,
memory_limit), compiled on the host, against the times of both sweeps on a GB300; and the lanes and rows of
the sweeps in registers."""
import os
import subprocess
import tempfile

import pytest

from conftest import ROOT

SMS = 152
# points, equal calls of 99 steps, ms through memory, ms in registers
MEASURED = [
    (8, 1000, 0.274, 0.134), (8, 8000, 0.275, 0.183), (8, 12000, 0.281, 0.399), (8, 60000, 0.711, 1.331),
    (16, 8000, 0.420, 0.183), (16, 20000, 0.474, 0.535), (16, 60000, 1.122, 1.350), (20, 8000, 0.507, 0.218),
    (20, 20000, 0.589, 0.713), (20, 60000, 1.369, 1.652), (28, 5000, 0.646, 0.228), (28, 60000, 1.798, 2.205),
    (36, 1000, 0.798, 0.250), (36, 20000, 0.941, 1.189), (36, 60000, 2.246, 2.671), (50, 32, 1.045, 0.318),
    (50, 5000, 1.055, 0.363), (50, 12000, 1.130, 1.037), (50, 20000, 1.245, 1.547), (50, 60000, 3.087, 3.430),
    (64, 16000, 1.451, 1.374), (64, 20000, 1.586, 2.029), (64, 60000, 3.988, 4.496), (72, 12000, 1.589, 1.235),
    (72, 30000, 2.381, 2.702), (80, 12000, 1.739, 1.360), (80, 30000, 2.716, 2.964), (100, 12000, 2.189, 1.722),
    (100, 60000, 6.860, 7.189), (128, 1000, 2.491, 0.424), (128, 20000, 3.895, 3.170), (128, 60000, 8.921, 8.697),
    (200, 20000, 6.266, 5.003), (512, 1000, 10.322, 0.643),
]


@pytest.fixture(scope="module")
def binary():
    out = os.path.join(tempfile.mkdtemp(), "heat1d_rule_t")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "linear_system_solvers_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "heat1d_rule_t.cpp"), "-o", out], check=True, capture_output=True, text=True)
    return out


def limits(binary, books):
    text = []
    for book in books:
        text.append(f"{len(book)} {SMS}")
        text.extend(" ".join(map(str, g)) for g in book)
    res = subprocess.run([binary], input="\n".join(text), capture_output=True, text=True, check=True)
    return [int(x) for x in res.stdout.split()]


def equal(n, count, steps=99):
    return [(n, n - 2, min(32, count - q), steps) for q in range(0, count, 32)]


def test_the_faster_sweep_is_chosen(binary):
    got = limits(binary, [equal(n, count) for n, count, _, _ in MEASURED])
    for (n, count, mem, reg), limit in zip(MEASURED, got):
        taken = mem if n <= limit else reg
        assert taken <= 1.02 * min(mem, reg), (n, count, limit)


def test_uneven_books(binary):
    # few short lines beside many long ones, an empty book, a book of long lines only
    long_lines = [(n, n - 2, 32, steps) for n in (256, 384, 512) for steps in (100, 500, 1000)] * 200
    got = limits(binary, [[], long_lines, long_lines + equal(16, 64), equal(10, 60000) + long_lines])
    assert got[:3] == [0, 0, 0] and got[3] == 10


def test_shapes_hold_every_row(binary):
    cases = [(rows, least) for rows in range(2, 513) for least in (2, 4)]
    res = subprocess.run([binary, "shape"], input="\n".join(f"{r} {l} 16" for r, l in cases), capture_output=True, text=True, check=True)
    for (rows, least), line in zip(cases, res.stdout.splitlines()):
        W, R = map(int, line.split())
        assert W in (2, 4, 8, 16, 32) and W >= least and 4 <= R <= 16 and W * R >= rows
        assert W == least or W // 2 * 16 < rows
        assert R == 4 or W * (R - 1) < rows
