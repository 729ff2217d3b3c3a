"""The warm-start network over a batch large enough for 256 positions per block
against the same images one at a time (128 positions per block): each
output is the same sum in the same order, so the bits are equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,W", [(3, 90, 160), (7, 90, 160), (9, 101, 93), (40, 5, 433), (160, 47, 11)])
def test_batch_equals_single(B, H, W):
    T = pytest.importorskip("torch")
    if not T.cuda.is_available():
        pytest.skip("no CUDA device")
    from reconflow_gb300.warmstart import WarmStartNet

    net = WarmStartNet(B, H, W, seed=5)
    x = T.as_tensor(np.random.default_rng(B + W).normal(0, 1, (B, H, W, 16)).astype(np.float32),
                    device="cuda")
    o16, o8 = (t.clone() for t in net.forward(x))
    for i in range(0, B, max(1, B // 6)):
        s16, s8 = net.forward(x[i:i + 1].contiguous())
        assert T.equal(o16[i], s16[0]) and T.equal(o8[i], s8[0]), i
    assert not net.wait_gave_up()
    net.close()
