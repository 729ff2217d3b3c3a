"""The worker threads that pose handles hold (rf_epipolar.cpp), without a GPU:
tests/cpp/pose_workers.cpp compiled with that file, one situation per run."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def tool(tmp_path_factory):
    exe = tmp_path_factory.mktemp("workers") / "pose_workers"
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-pthread", "-I",
                    os.path.join(ROOT, "reconflow_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "pose_workers.cpp"), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    return str(exe)


@pytest.mark.parametrize("situation", ["forked", "forked_busy", "throwing", "affinity"])
def test_workers(tool, situation):
    r = subprocess.run([tool, situation], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
