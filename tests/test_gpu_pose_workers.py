"""Pose handles that solve at the same time share one set of host worker threads:
each gets the result it gets alone, while handles come and go."""
import threading

import numpy as np
import pytest

from test_gpu_pose import _pose, _scene, _to8

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("handles", [1, 2, 7])
def test_concurrent_handles(rf, handles):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    scenes = [_scene(320 + 16 * i, 240, 20 + i) for i in range(handles)]

    def solve(sc):
        cp = _pose(rf, sc["K"])
        out = cp.solvePose_8uc1(_to8(sc["I0"]), _to8(sc["I1"]))
        return out, cp.matches()

    alone = [solve(sc) for sc in scenes]  # a handle at a time: workers start and end
    got = [[] for _ in scenes]

    def many(i):
        for _ in range(4):
            got[i].append(solve(scenes[i]))

    threads = [threading.Thread(target=many, args=(i,)) for i in range(handles)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(60)
        assert not t.is_alive()
    for (want, wm), results in zip(alone, got):
        assert len(results) == 4
        for (ret, R, t), m in results:
            assert ret == want[0]
            assert np.array_equal(R, want[1]) and np.array_equal(t, want[2])
            assert all(np.array_equal(a, b) for a, b in zip(m, wm))
