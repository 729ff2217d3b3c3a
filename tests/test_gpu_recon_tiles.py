"""ReconFlow with several iterations per launch (small levels) against the FP32
oracle, bit for bit: sizes around the edges of the four tiles (24 x 2, 24 x 4,
20 x 8, 24 x 12), rows with and without padding (a row's last pixel reads the next
row's first one), iteration counts around a launch's two and three, and priors."""
import numpy as np
import pytest

from helpers import align_up, pad_rows, textured_pair
from reconflow_gb300.reconflow import CV_32F
from test_gpu_solve import _K, _pose

pytestmark = pytest.mark.gpu


def _check(oracle, rf, w, h, L, iters, align, method=14, fix=1, warps=2, still=False):
    rng = np.random.default_rng(100 * w + 10 * h + iters)
    I0, I1 = textured_pair(rng, h, w, shift=(1.3, -0.5))
    s = align_up(w, align)
    I0, I1 = pad_rows(I0, s), pad_rows(I1, s)
    K = _K(w, h)
    R, t = (np.eye(3), np.zeros(3)) if still else _pose(w + iters)
    prior = {}
    if method != 14:
        planes = [pad_rows(rng.normal(1.0, 0.3, (h, w)).astype(np.float32), s) for _ in range(2)]
        if method == 20:
            planes.append(pad_rows((rng.random((h, w)) < 0.4).astype(np.float32), s))
        prior = dict(zip(("ufn", "vfn", "mask"), planes))
    f = rf.ReconFlow(StrideAlignment=align)
    f.initializeR(w, h, 1, L, 2.0, method, 50.0, 0.0, 0.1, 100.0, 1 / 0.33, 60.0, 0.5, 0.25, warps,
                  iters, cvType=CV_32F, fix_quirks=fix)
    f.setCameraMatrices(K, K)
    f.copyImagesToDevice(I0, I1)
    if prior:
        f.copySparseOpticalFlowToDevice(*prior.values())
    f.solveR(R, t, 5.0)
    u, v = f.copyOpticalFlowToHost()
    X, Y, Z = f.copy3dToHost()
    p = oracle.make_params(w, h, L, method=method, lam=50.0, lambdaf=0.1, lambdams=100.0,
                           alpha_tv=1 / 0.33, alpha_proj=60.0, alpha_fn=0.5, tau=0.25,
                           n_warp_iters=warps, n_solver_iters=iters, fix_quirks=fix,
                           stride_alignment=align)
    want = oracle.solve(p, I0, I1, K0=K, K1=K, R1=R, t1=t, dtype=np.float32, **prior)
    for name, got in zip(("u", "v", "X", "Y", "Z"), (u, v, X, Y, Z)):
        a, b = np.asarray(got)[:h, :w], np.asarray(want[name])[:h, :w]
        same = (a.view(np.uint32) == b.view(np.uint32)) | (np.isnan(a) & np.isnan(b))
        assert same.all(), (name, int((~same).sum()), np.argwhere(~same)[0])


# the tiles in turn, at and beside their edges
SIZES = [(1, 1), (24, 2), (25, 3), (33, 9), (96, 72), (97, 75), (120, 84), (121, 61), (160, 120),
         (161, 90), (240, 144), (225, 166)]


@pytest.mark.parametrize("w,h", SIZES)
@pytest.mark.parametrize("iters,align", [(2, 32), (5, 1), (7, 4)])
def test_sizes(oracle, rf, w, h, iters, align):
    _check(oracle, rf, w, h, 1, iters, align)


@pytest.mark.parametrize("iters", [1, 2, 3, 4, 6, 13])
@pytest.mark.parametrize("fix", [0, 1])
def test_iteration_counts(oracle, rf, iters, fix):
    _check(oracle, rf, 230, 150, 3, iters, 32, fix=fix)


@pytest.mark.parametrize("method", [17, 20])
@pytest.mark.parametrize("w,h,align", [(64, 40, 1), (160, 96, 32), (225, 166, 32)])
def test_priors(oracle, rf, method, w, h, align):
    _check(oracle, rf, w, h, 2, 5, align, method=method)


def test_no_motion(oracle, rf):
    # points at infinity: the quotients' guards fail
    _check(oracle, rf, 90, 60, 2, 5, 32, still=True)
