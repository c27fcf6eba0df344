"""Set-up work over threads (linear_system_solvers_gb300/csrc/adi_threads.hpp): where no thread can be had the
caller's does the work (an exception that leaves a C entry point would end the program)."""
import os
import subprocess
import tempfile

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "linear_system_solvers_gb300", "csrc")


@pytest.mark.parametrize("args", [[], ["none"]])
def test_every_share_runs_with_and_without_threads(args):
    out = os.path.join(tempfile.mkdtemp(), "adi_threads_t")
    subprocess.run(["g++", "-std=c++17", "-O2", "-pthread", "-I", CSRC, os.path.join(ROOT, "tests", "cpp", "adi_threads_t.cpp"), "-o", out],
                   check=True, capture_output=True, text=True)
    res = subprocess.run([out] + args, capture_output=True, text=True)
    if res.returncode == 77:
        pytest.skip("threads start within the address space that is left")
    assert res.returncode == 0 and res.stdout.strip() == "ok", (res.returncode, res.stdout, res.stderr)


def test_set_up_starts_no_other_threads():
    for f in os.listdir(CSRC):
        if f.endswith((".cu", ".cuh", ".hpp")) and f != "adi_threads.hpp":
            assert "std::vector<std::thread>" not in open(os.path.join(CSRC, f)).read(), f
