"""The rules that choose a level's kernels by its size (rf_rules.h), without a GPU."""
import os
import subprocess

import pytest

from helpers import align_up

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def ask(tmp_path_factory):
    exe = tmp_path_factory.mktemp("rules") / "rules"
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "reconflow_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "rules.cpp"), "-o", str(exe)],
                   check=True, capture_output=True, text=True)

    def run(questions):
        r = subprocess.run([str(exe)], input="\n".join(questions) + "\n", capture_output=True,
                           text=True, check=True)
        return [int(x) for x in r.stdout.split()]
    return run


# a grid has at most 65535 blocks in y; a pair block has four rows
@pytest.mark.parametrize("h", [1000, 262140, 262141, 270000, 524280])
@pytest.mark.parametrize("w,align", [(6, 32), (8, 4), (7, 4), (6, 2), (1504, 32)])
def test_pairs_fit_a_grid(ask, w, h, align):
    s = align_up(w, align)
    want = s % 4 == 0 and w * h >= 1500000 and -(-h // 4) <= 65535
    assert ask([f"pairs {w} {h} {s}"]) == [int(want)]
