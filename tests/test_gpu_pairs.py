"""The two-pixel half-steps (levels of at least 400 000 pixels over a batch, 1.5
million for a single pair) against the FP32 oracle, bit for bit: ragged sizes
in one batch, rows without padding, flat and empty frames, a pose without
motion, weights and strides that take the one-pixel kernels."""
import numpy as np
import pytest

from helpers import align_up, assert_bitexact, pad_rows, textured_pair
from test_gpu_solve import _K, _pose, compare, run_gpu, run_oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def need_gpu():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


# with the first pair the level is large enough; the others are small enough to
# reach every edge of a 64 x 4 tile
SIZES = [(720, 530), (333, 61), (192, 48), (64, 33), (66, 5), (61, 7), (5, 3), (1, 1), (130, 70),
         (96, 40)]


def _inputs(iters, fix):
    out = []
    for i, (w, h) in enumerate(SIZES):
        rng = np.random.default_rng(10 * i + iters)
        I0, I1 = textured_pair(rng, h, w, shift=(1.1 + 0.1 * i, -0.4))
        R, t = _pose(i + iters)
        if i == 8:  # flat frames: zero gradients, zero dual field
            I0[:], I1[:] = 0.25, 0.25
        if i == 9:  # a flat half, and no motion: points at infinity
            I0[:, : w // 2] = I1[:, : w // 2] = 0.0
            R, t = np.eye(3), np.zeros(3)
        out.append((w, h, I0, I1, _K(w, h), R, t))
    return out


@pytest.mark.parametrize("iters", [1, 2, 5])
@pytest.mark.parametrize("fix,align", [(0, 32), (1, 32), (1, 4), (1, 2)])
def test_batch_equals_oracle(oracle, rf, iters, fix, align):
    pairs = _inputs(iters, fix)
    b = rf.ReconFlowBatch([(p[0], p[1]) for p in pairs], 1, method=14, lambda_=50.0, lambdaf=0.1,
                          lambdams=100.0, alphaTv=1 / 0.33, alphaProj=60.0, tau=0.25,
                          nWarpIters=2, nSolverIters=iters, fix_quirks=fix, StrideAlignment=align)
    for i, (w, h, I0, I1, K, R, t) in enumerate(pairs):
        b.setCameraMatrices(i, K, K)
        s = b.strides[i]
        b.copyImagesToDevice(i, pad_rows(I0, s), pad_rows(I1, s))
    b.solveR([p[5] for p in pairs], [p[6] for p in pairs])
    for i, (w, h, I0, I1, K, R, t) in enumerate(pairs):
        s = align_up(w, align)
        p = oracle.make_params(w, h, 1, lam=50.0, lambdaf=0.1, lambdams=100.0, alpha_tv=1 / 0.33,
                               alpha_proj=60.0, tau=0.25, n_warp_iters=2, n_solver_iters=iters,
                               fix_quirks=fix, stride_alignment=align)
        want = oracle.solve(p, pad_rows(I0, s), pad_rows(I1, s), K0=K, K1=K, R1=R, t1=t,
                            dtype=np.float32)
        got = dict(zip("uv", b.copyOpticalFlowToHost(i)), **dict(zip("XYZ", b.copy3dToHost(i))))
        for k in got:
            assert_bitexact(got[k], want[k], f"pair {i} ({w}x{h}) {k}", region=(h, w))
    b.close()


@pytest.mark.parametrize("method", [14, 17, 20])
@pytest.mark.parametrize("w,h", [(1504, 1000), (1501, 1000)])
def test_single_pair_equals_oracle(oracle, rf, method, w, h):
    rng = np.random.default_rng(method)
    s = align_up(w)
    I0, I1 = (pad_rows(a, s) for a in textured_pair(rng, h, w))
    prior = None
    if method != 14:
        uv = [pad_rows(rng.normal(m, 0.3, (h, w)).astype(np.float32), s) for m in (1.5, -0.7)]
        mask = pad_rows((rng.random((h, w)) < 0.3).astype(np.float32), s)
        prior = (*uv, mask) if method == 20 else tuple(uv)
    R, t = _pose(method)
    kw = dict(warps=1, iters=3, fix=1, alpha_fn=20.0)
    got, _ = run_gpu(rf, w, h, 1, method, I0, I1, _K(w, h), R, t, prior=prior, **kw)
    want = run_oracle(oracle, w, h, 1, method, I0, I1, _K(w, h), R, t, prior=prior, **kw)
    compare(got, want, w, h)


@pytest.mark.parametrize("kw", [dict(lambdaf=100.0, alpha_proj=1.0, alpha_tv=3.0),
                                dict(lambdams=0.0), dict(lambdaf=0.0), dict(lam=0.0),
                                dict(tau=0.0)])
def test_weights(oracle, rf, kw):
    """The class's default weights, and weights of zero (lambdams = 0 takes the
    one-pixel kernels, the others the pairs' slow paths)."""
    w, h = 1504, 1000
    rng = np.random.default_rng(5)
    I0, I1 = textured_pair(rng, h, w)
    R, t = _pose(5)
    kw = dict(kw, warps=1, iters=2, fix=1)
    got, _ = run_gpu(rf, w, h, 1, 14, I0, I1, _K(w, h), R, t, **kw)
    want = run_oracle(oracle, w, h, 1, 14, I0, I1, _K(w, h), R, t, **kw)
    compare(got, want, w, h)
