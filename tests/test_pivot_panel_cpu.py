"""The panel pivot kernel's code on the CPU (tests/native/pivot_panel_check.cpp): fibers for the GPU's threads, remote
stores that arrive late, in any order, and, over some links, only when nothing else can go on. Pivots, D, panels
and statistics must be those of the reference's steps one after another, bit for bit, in FP64 and FP32, on one CTA, on
clusters of 2 to 16 with and without helper clusters, with and without the row copies, for values that make
interchanges, 2x2 pivots, rejected choices, perturbed pivots and partners from outside the block. With
"giveup" a wait runs out at a random moment: every thread must come to its end, with the status word set and nothing
written outside the front."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "native", "pivot_panel_check.cpp")
CUDA = "/usr/local/cuda/include"


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    if shutil.which("g++") is None or not os.path.isdir(CUDA):
        pytest.skip("needs g++ and the CUDA headers")
    exe = str(tmp_path_factory.mktemp("panel") / "pivot_panel_check")
    # no contraction, as the kernel is compiled
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-w", "-I", CUDA, "-o", exe, SRC], check=True)
    return exe


@pytest.mark.parametrize("args", [("1", "40"), ("2", "40"), ("3", "40"), ("4", "40"), ("1", "wide"), ("2", "wide"),
                                  ("1", "60", "giveup"), ("2", "60", "giveup")])
def test_panel_kernel_against_serial_steps(check, args):
    r = subprocess.run([check, *args], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-500:]
