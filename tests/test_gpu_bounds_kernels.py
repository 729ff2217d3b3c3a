"""Bounds-checked debug build (RF_BOUNDS_CHECK) over the kernels that
tests/test_gpu_bounds.py is too small or too uniform to reach: the two-pixel
half-steps of a batch and of a single pair (64-bit loads and stores, 16-byte copies,
halo columns), the one-pixel half-steps of levels too large for register tiles, the
register tiles with and without padded rows, plain TV-L1's register tiles and the tiled
medians.  A child process loads the checked library; an index outside its plane is
counted and never followed, and the count has to be 0."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import ctypes, sys
import numpy as np
sys.path.insert(0, ROOT)
sys.path.insert(0, ROOT + "/tests")
import reconflow_gb300 as rf
from reconflow_gb300 import _native as N
from helpers import pad_rows, textured_pair

lib = rf.load()
assert lib._name.endswith("librfgb300_check.so"), lib._name


def take():
    c = ctypes.c_ulonglong(0)
    first = ctypes.c_longlong(-1)
    N.check(lib.rf_debug_bounds(ctypes.byref(c), ctypes.byref(first)))
    return c.value, first.value


def pose(seed):
    c, sn = np.cos(0.01 + 0.001 * seed), np.sin(0.01 + 0.001 * seed)
    return np.array([[c, 0, sn], [0, 1, 0], [-sn, 0, c]]), np.array([-0.1, 0.01, 0.02])


def K(w, h):
    return np.array([[0.8 * w, 0, w / 2], [0, 0.8 * w, h / 2], [0, 0, 1.0]])


def single(w, h, L, method, align, iters):
    rng = np.random.default_rng(w * h + method)
    s = -(-w // align) * align
    I0, I1 = (pad_rows(a, s) for a in textured_pair(rng, h, w, shift=(1.3, -0.6)))
    if method == 0:
        f = rf.CudaFlow(StrideAlignment=align)
        f.initialize(w, h, 1, 5, L, 2.0, 0, 50.0, 0.0, 0.33, 0.25, 2, iters)
        f.copyImagesToDevice(I0, I1)
        f.solveOpticalFlow()
    else:
        f = rf.ReconFlow(StrideAlignment=align)
        f.initializeR(w, h, 1, L, 2.0, method, 50.0, 0.0, 0.1, 100.0, 1 / 0.33, 60.0, 0.5, 0.25,
                      2, iters, cvType=5, fix_quirks=1)
        f.setCameraMatrices(K(w, h), K(w, h))
        f.copyImagesToDevice(I0, I1)
        if method != 14:
            uv = [pad_rows(rng.normal(1.0, 0.3, (h, w)).astype(np.float32), s) for _ in range(2)]
            m = pad_rows((rng.random((h, w)) < 0.3).astype(np.float32), s)
            f.copySparseOpticalFlowToDevice(*uv, m if method == 20 else None)
        f.solveR(*pose(method), 5.0)
    takes = [f.levelTakesTile(l) for l in range(L)]
    u, v = f.copyOpticalFlowToHost()
    f.close()
    assert np.isfinite(u[:, :w]).all()
    got = take()
    assert got == (0, -1), ((w, h, L, method, align), got)
    return takes


# pixel pairs (odd and even rows' ends, with and without padding, priors)
for w, h, method, align in [(1501, 1000, 14, 32), (1504, 1000, 14, 32), (1502, 1001, 20, 4),
                            (1503, 1003, 17, 4)]:
    assert single(w, h, 2, method, align, 3)[0] is False
# one pixel per thread: too large for tiles, and a single iteration
for w, h, method, align, iters in [(333, 211, 14, 32, 3), (333, 211, 20, 1, 3), (64, 48, 14, 32, 1)]:
    assert single(w, h, 1, method, align, iters)[0] is True
# register tiles
for w, h, method, align in [(97, 75, 14, 32), (96, 72, 17, 1), (121, 61, 14, 1), (161, 90, 20, 4),
                            (225, 166, 14, 32)]:
    assert single(w, h, 1, method, align, 5)[0] is False
# plain TV-L1: both tiles, and the medians of every size
for w, h, align in [(64, 48, 32), (37, 23, 1), (301, 211, 32), (5, 3, 32), (1, 1, 32)]:
    single(w, h, 1, 0, align, 7)

# a batch with pixel pairs on its first level and every edge of their tile
sizes = [(722, 560), (333, 61), (192, 48), (64, 33), (66, 5), (61, 7), (6, 4), (130, 70)]
for align, pairs in ((32, True), (4, True), (2, False)):
    b = rf.ReconFlowBatch(sizes, 2, method=14, lambda_=50.0, lambdaf=0.1, lambdams=100.0,
                          alphaTv=1 / 0.33, alphaProj=60.0, tau=0.25, nWarpIters=2, nSolverIters=3,
                          fix_quirks=1, StrideAlignment=align)
    assert b.levelTakesTile(0) is not pairs and b.levelTakesTile(1)
    Rs, ts = zip(*[pose(i) for i in range(len(sizes))])
    for i, (w, h) in enumerate(sizes):
        I0, I1 = textured_pair(np.random.default_rng(i), h, w, shift=(1.3, -0.6))
        s = b.strides[i]
        b.setCameraMatrices(i, K(w, h), K(w, h))
        b.copyImagesToDevice(i, pad_rows(I0, s), pad_rows(I1, s))
    b.solveR(Rs, ts)
    b.synchronize()
    b.close()
    got = take()
    assert got == (0, -1), ("batch", align, got)
print("BOUNDS OK")
"""


def test_checked_build_counts_nothing():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from reconflow_gb300 import build

    build.build(bounds_check=True)
    env = dict(os.environ, RF_BOUNDS_CHECK="1")
    r = subprocess.run([sys.executable, "-c", f"ROOT = {ROOT!r}\n" + CHILD], env=env,
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and "BOUNDS OK" in r.stdout, r.stdout + r.stderr
