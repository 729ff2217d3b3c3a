"""A level too tall for a grid of two-pixel blocks (four rows each, at most 65535
blocks), though large enough for them, solves with the one-pixel kernels."""
import numpy as np
import pytest

from helpers import align_up, pad_rows, textured_pair
from test_gpu_solve import _K, _pose, compare, run_gpu, run_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h", [262140, 262141])
def test_tall_level_equals_oracle(oracle, rf, h):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    w = 6
    s = align_up(w)
    I0, I1 = (pad_rows(a, s) for a in textured_pair(np.random.default_rng(h), h, w))
    R, t = _pose(3)
    kw = dict(warps=1, iters=2, fix=1)
    got, _ = run_gpu(rf, w, h, 1, 14, I0, I1, _K(w, h), R, t, **kw)
    want = run_oracle(oracle, w, h, 1, 14, I0, I1, _K(w, h), R, t, **kw)
    compare(got, want, w, h)
