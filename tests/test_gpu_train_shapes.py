"""Loss and gradients of the warm-start network against its FP64 oracle at
shapes that reach the edges of the tensor-core tiles: fewer pixels than a
K-chunk, odd and single-column rows, a ragged last chunk, several splits of the
weight gradient's reduction."""
import numpy as np
import pytest

from oracle import cnn_oracle as CO

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,W", [(1, 2, 2), (1, 3, 5), (2, 5, 7), (1, 9, 33), (3, 41, 2),
                                   (2, 70, 61)])
def test_gradients(B, H, W):
    T = pytest.importorskip("torch")
    if not T.cuda.is_available():
        pytest.skip("no CUDA device")
    from reconflow_gb300.warmstart import LOSS_WEIGHTS, WarmStartNet

    rng = np.random.default_rng(B * 100 + H + W)
    net = WarmStartNet(B, H, W, seed=3)
    h2, w2 = (H + 1) // 2, (W + 1) // 2
    x = rng.normal(0, 1, (B, H, W, 16)).astype(np.float32)
    # targets away from the predictions: the sign of the L1 loss is not in doubt
    t16, t8 = (rng.choice([-9.0, 9.0], s).astype(np.float32)
               for s in ((B, h2, w2, 8), (B, H, W, 8)))
    m16, m8 = ((rng.random(s) < 0.9).astype(np.float32) for s in ((B, h2, w2), (B, H, W)))
    loss = net.backward(*(T.as_tensor(a, device="cuda") for a in (x, t16, m16, t8, m8)))
    got = net.grads().astype(np.float64)
    want, lref, _ = CO.backward(net.params().astype(np.float64), x, t16, m16, t8, m8, LOSS_WEIGHTS)
    assert not net.wait_gave_up()
    net.close()
    assert abs(loss - lref) <= 1e-3 * abs(lref)
    off = 0
    for cin, cout, _, _ in CO.LAYERS:
        for n in (cout * 9 * cin, cout):
            g, w = got[off:off + n], want[off:off + n]
            off += n
            # both sides hold BF16 values at the same points; a value within FP32
            # rounding of a BF16 boundary may fall on either side (2^-8 of itself)
            assert np.linalg.norm(g - w) <= 2e-2 * np.linalg.norm(w) + 1e-12, (cin, cout, n)
