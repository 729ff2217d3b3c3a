"""rf_packed.cuh's quotients and roots are IEEE division and square root, bit for bit,
as the compiler at hand builds them (tests/cpp/quotients.cu, the solver's own flags):
the reciprocal and the root of every significand, every pair of significands whose
quotient is nearest a tie between two results, random bits as far as QuotientGuard lets
them pass, and products that are not contracted with the sums after them."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_quotients_and_roots_are_ieee(tmp_path):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from reconflow_gb300 import build

    exe = tmp_path / "quotients"
    subprocess.run([build.nvcc(), os.path.join(ROOT, "tests", "cpp", "quotients.cu"), "-o", str(exe)]
                   + build.ARCH + build.COMMON + build.SOURCES["rf_kernels.cu"],
                   check=True, capture_output=True, text=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    got = {a: (int(n), int(bad)) for a, n, bad in (line.split() for line in r.stdout.splitlines())}
    least = dict(reciprocals=3 << 23, near_ties=10 ** 7, guarded=10 ** 7, roots=6 << 23,
                 products=1024 * 256 * 64)
    assert set(got) == set(least)
    for what, (n, bad) in got.items():
        assert n >= least[what] and bad == 0, (what, n, bad)
