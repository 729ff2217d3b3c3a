"""The tile search, without a GPU: handles whose times depend on the shapes in a known
way.  What a level's shape decides is what the search has to time there."""
import time

import pytest

from reconflow_gb300 import autotune


class Handle:
    """A batch of one pair and a single handle in one: `inner[level]`, whether the inner
    iterations take the level's shape; only what the real ones' shape reaches depends on it,
    and the fastest shape of every level is `fast[level]`."""

    n = 1

    def __init__(self, inner, fast):
        self.inner, self.fast = inner, fast
        self.params = type("P", (), dict(n_levels=len(inner)))
        self.profiled = []

    def levelDims(self, i, level):
        return 1280 >> level, 720 >> level, 1280 >> level

    def levelTakesTile(self, level):
        return self.inner[level]

    def setTiles(self, tw, th):
        self.tiles = list(zip(tw, th))

    def solveR(self, *pose):
        pass

    def synchronize(self):
        pass

    def profileLevel(self, level, iters):
        self.profiled.append(level)
        if not self.inner[level]:
            return 1.0, 1.0  # the same launches whatever the shape
        return (0.5 if self.tiles[level] == self.fast[level] else 1.0), 1.0

    def solveWarm(self, level, R, t, warps, iters):
        assert len(warps) == len(iters) == level + 1
        time.sleep(0.002 + warps[level] * (1e-4 if self.tiles[level] == self.fast[level] else 1e-3))


@pytest.mark.parametrize("inner", [(False, False, True, True), (True, True), (False,)])
def test_batch_search_times_what_the_shape_decides(inner):
    fast = [(128, 2), (16, 16), (64, 2), (16, 8)][:len(inner)]
    h = Handle(inner, fast)
    table = autotune.autotune(h, [], [])
    assert [tuple(e["tile"]) for e in table] == fast
    assert [e["timed"] for e in table] == ["iterations" if i else "passes" for i in inner]
    assert h.tiles == fast


def test_single_search_keeps_the_default_where_no_shape_counts():
    inner, fast = (True, True, False, False), [(64, 2), (32, 4), (16, 16), (128, 2)]
    h = Handle(inner, fast)
    table = autotune.autotune_single(h, None, None, 4)
    want = [f if i else (32, 8) for i, f in zip(inner, fast)]
    assert [tuple(e["tile"]) for e in table] == want and h.tiles == want
    assert set(h.profiled) == {0, 1}
    assert [len(e["ms"]) for e in table] == [len(autotune.CANDIDATES) if i else 0 for i in inner]
