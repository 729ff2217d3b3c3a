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


# the region's columns and rows that a block's tile keeps, in the order they are tried
TILES = [(24, 2), (24, 4), (20, 8), (24, 12)]


@pytest.mark.parametrize("sms", [1, 20, 148, 152, 160])
def test_tiles_have_an_sm_each(ask, sms):
    sizes = [(w, h) for w in (1, 24, 25, 96, 97, 160, 225, 240, 288, 289, 320)
             for h in (1, 2, 38, 61, 72, 84, 120, 144, 145, 152, 166, 168, 240)]
    got = ask([f"tile {w} {h} {sms}" for w, h in sizes])
    for (w, h), kind, blocks in zip(sizes, got[::2], got[1::2]):
        need = [-(-w // tw) * -(-h // th) for tw, th in TILES]
        fits = [i for i, n in enumerate(need) if n <= sms]
        assert (kind, blocks) == ((fits[0] + 1, need[fits[0]]) if fits else (0, 0)), (w, h)


@pytest.mark.parametrize("sms", [1, 148, 152])
def test_wide_convolution_tiles(ask, sms):
    n = 256 * sms
    q = [(n - 1, 1000), (n, 1000), (n, 113 * 1024), (n, 113 * 1024 + 1)]
    assert ask([f"conv {a} {b} {sms}" for a, b in q]) == [0, 1, 1, 0]
