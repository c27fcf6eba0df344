"""Offsets into the line tables of the batched kernels (linear_system_solvers_gb300/csrc/adi_index.hpp), compiled on
the host: exact for every grid that is accepted (2^30 points), whose rows of tables alone pass 2^31
elements when the v direction is long."""
import os
import re
import subprocess
import tempfile

from conftest import ROOT

CSRC = os.path.join(ROOT, "linear_system_solvers_gb300", "csrc")


def test_offsets_of_the_largest_grids():
    out = os.path.join(tempfile.mkdtemp(), "adi_index_t")
    subprocess.run(["g++", "-std=c++17", "-O2", "-fsanitize=undefined", "-fno-sanitize-recover", "-I", CSRC,
                    os.path.join(ROOT, "tests", "cpp", "adi_index_t.cpp"), "-o", out], check=True, capture_output=True, text=True)
    cases = []
    for nx, ny in ((4, 1 << 28), (1 << 28, 4), (1 << 15, 1 << 15), (6, 1 << 27), (100, 50)):
        for pitch, rows, slots in ((-(-ny // 8) * 8, nx, 18), (-(-ny // 4) * 4, nx, 10), (nx, ny, 5), (nx, ny, 3)):
            for t in (0, 1, rows - 1):
                for slot in (0, slots - 1):
                    cases.append((t, slot, pitch - 1, pitch, slots))
    near = (2**31 - 1) // 18 // 8 * 8 # the longest pitch of the FP32 kernels with int rows; v tables of any length
    for nx, pitch in ((8, near), (1000, 104), (1 << 26, 8)):
        for t in (0, 1, nx - 1):
            cases += [(t, 0, pitch - 1, pitch, 180), (t, 17, pitch - 1, pitch, 180)]
    for pitch, rows in ((1 << 28, 4), (4, 1 << 28)):
        cases += [(t, slot, pitch - 1, pitch, 50) for t in (0, rows - 1) for slot in (0, 4)]
    res = subprocess.run([out], input="\n".join(" ".join(map(str, c)) for c in cases), check=True, capture_output=True, text=True)
    got = [int(x) for x in res.stdout.split()]
    slots_of = lambda s: {180: 18, 50: 5}.get(s, s)
    assert got[:-1] == [(t * slots_of(slots) + slot) * pitch + q for t, slot, q, pitch, slots in cases]
    assert near <= got[-1] and 18 * got[-1] < 2**31


def test_kernels_reach_their_tables_through_it():
    src = open(os.path.join(CSRC, "adi_batched.cu")).read()
    view = re.search(r"struct inst_view \{.*?\n\};", src, re.S).group(0)
    assert "si.at(t, k, j)" in view and "vi.at(t, k, i)" in view
