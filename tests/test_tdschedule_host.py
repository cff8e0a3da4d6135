"""The triangle-dimer schedule drops refreshes that a later move overwrites
(csrc/rt_tdschedule.h).  On the host, moves in random order from random
states leave the arrays that the full phase program leaves, wherever the walk
is cut (tests/cpp/tdschedule_check.cpp)."""
from __future__ import annotations

import os
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def checker(tmp_path_factory) -> str:
    exe = str(tmp_path_factory.mktemp("tdschedule") / "tdschedule_check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "randomtilings_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "tdschedule_check.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("m,rounds,moves", [(4, 200, 60), (9, 60, 200), (33, 4, 150)])
def test_schedule_equals_the_full_program(checker, m, rounds, moves):
    out = subprocess.run([checker, str(m), str(rounds), str(moves)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.startswith("ok"), (out.stdout, out.stderr)
    words = out.stdout.replace(",", "").split()
    full, lazy, changed, sweep = int(words[1]), int(words[4]), int(words[7]), int(words[9])
    assert lazy < full and changed > 1000
    # lozenges 1 + 6 x 3, triangles 2 + 6 x 2, butterflies 3 + 30, 2 + 30, 2 + 30
    assert sweep == 130
