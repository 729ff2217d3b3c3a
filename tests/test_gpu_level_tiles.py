"""rf_level_takes_tile / rf_batch_level_takes_tile: which levels' inner iterations run
in the shape that the tile search picks."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def need_gpu():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("w,h,L,iters,want", [
    (1504, 1000, 3, 5, [0, 1, 1]),      # pixel pairs, then one pixel per thread
    (1280, 720, 6, 5, [1, 1, 1, 0, 0, 0]),
    (1280, 720, 6, 1, [1, 1, 1, 1, 1, 1]),  # one iteration: a launch each anyway
    (96, 72, 2, 5, [0, 0])])
def test_single(rf, w, h, L, iters, want):
    import torch

    if torch.cuda.get_device_properties(0).multi_processor_count != 152:
        pytest.skip("the levels of a device with 152 multiprocessors")
    f = rf.ReconFlow()
    f.initializeR(w, h, 1, L, 2.0, 14, 50.0, 0.0, 0.1, 100.0, 1 / 0.33, 60.0, 0.5, 0.25, 1, iters,
                  cvType=5, fix_quirks=1)
    assert [int(f.levelTakesTile(l)) for l in range(L)] == want
    for bad in (-1, L):
        with pytest.raises(ValueError):
            f.levelTakesTile(bad)
    f.close()


def test_plain(rf):
    f = rf.CudaFlow()
    f.initialize(640, 480, 1, 5, 3, 2.0)
    assert not any(f.levelTakesTile(l) for l in range(3))
    f.close()


@pytest.mark.parametrize("align,lambdams,want", [(32, 100.0, [0, 1]), (4, 100.0, [0, 1]),
                                                 (2, 100.0, [1, 1]), (32, 0.0, [1, 1])])
def test_batch(rf, align, lambdams, want):
    b = rf.ReconFlowBatch([(722, 560), (37, 23)], 2, method=14, lambda_=50.0, lambdaf=0.1,
                          lambdams=lambdams, alphaTv=1 / 0.33, alphaProj=60.0, tau=0.25,
                          nWarpIters=1, nSolverIters=2, fix_quirks=1, StrideAlignment=align)
    assert [int(b.levelTakesTile(l)) for l in range(2)] == want
    b.close()
