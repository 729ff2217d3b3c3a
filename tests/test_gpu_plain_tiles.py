"""Plain TV-L1 with several iterations per launch against the FP32 oracle, bit
for bit: sizes around the edges of both tile shapes (24 x 24 from 60 000 pixels,
20 x 8 below), iteration counts around a launch's 4 and 6, flat frames, weights
that leave the fast quotients' range and weights that take one launch per step."""
import numpy as np
import pytest

from helpers import align_up, pad_rows, textured_pair
from test_gpu_solve import compare, run_gpu, run_oracle

pytestmark = pytest.mark.gpu


def _check(oracle, rf, w, h, iters, flat=0, L=1, **weights):
    rng = np.random.default_rng(1000 * w + h + iters)
    I0, I1 = textured_pair(rng, h, w, shift=(1.2, -0.6))
    if flat == 1:
        I0[:, : w // 2] = I1[:, : w // 2] = 0.5
    elif flat == 2:
        I0[:], I1[:] = 0.25, 0.75
    s = align_up(w)
    I0, I1 = pad_rows(I0, s), pad_rows(I1, s)
    kw = dict(warps=2, iters=iters, **weights)
    got, _ = run_gpu(rf, w, h, L, 0, I0, I1, None, None, None, **kw)
    want = run_oracle(oracle, w, h, L, 0, I0, I1, None, None, None, **kw)
    compare(got, want, w, h)


@pytest.mark.parametrize("w,h", [(1, 1), (1, 9), (33, 1), (19, 7), (20, 8), (21, 9), (40, 16),
                                 (41, 17), (300, 200), (312, 193), (265, 240)])
@pytest.mark.parametrize("iters", [1, 5, 13])
def test_sizes(oracle, rf, w, h, iters):
    _check(oracle, rf, w, h, iters)


@pytest.mark.parametrize("iters", [3, 4, 6, 7, 8, 12])
@pytest.mark.parametrize("w,h,L", [(90, 50, 1), (290, 230, 3)])
def test_iteration_counts(oracle, rf, w, h, L, iters):
    _check(oracle, rf, w, h, iters, L=L)


@pytest.mark.parametrize("flat", [1, 2])
@pytest.mark.parametrize("w,h", [(61, 43), (280, 240)])
def test_flat_frames(oracle, rf, w, h, flat):
    _check(oracle, rf, w, h, 7, flat=flat)


@pytest.mark.parametrize("weights", [dict(lam=0.0), dict(lam=-3.0), dict(lam=1e30), dict(lam=1e-25),
                                     dict(tau=0.0), dict(tau=1e-30), dict(tau=-0.1),
                                     dict(theta=1e-18), dict(theta=1e18)])
@pytest.mark.parametrize("w,h", [(61, 43), (280, 240)])
def test_weights(oracle, rf, w, h, weights):
    _check(oracle, rf, w, h, 7, **weights)
