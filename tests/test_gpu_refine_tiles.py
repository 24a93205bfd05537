"""The single-launch tree refinement's tiles (csrc/tree.cu): a warp's tile is
256 points below 4 Mi points and 1024 from there on, and a level whose
splitting nodes are one tile each takes its counts without the prefix step.
Trees at the edges of both (points a multiple of the tile, one less, one more;
levels of one and of several tiles a node; nodes larger than a tile next to
smaller ones) equal the level-by-level launches bit for bit."""
import numpy as np
import pytest

import simplefmm_b200 as sf
from simplefmm_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    return sf.Context(0)


def _lopsided(n):
    """Half the points in one small corner, the rest uniform: at every level
    nodes of many tiles stand beside nodes of one."""
    r = np.random.default_rng(n).uniform(0, 1, (n, 3))
    r[: n // 2] *= 1e-3
    return r


@pytest.mark.parametrize("dist,n,ppn", [
    ("uniform", 2, 1), ("uniform", 33, 1), ("uniform", 255, 8), ("uniform", 256, 8), ("uniform", 257, 8),
    ("uniform", 2048, 300), ("uniform", 2049, 255), ("plummer", 8191, 64), ("lopsided", 30000, 40),
    ("lopsided", 300001, 256), ("uniform", (4 << 20) - 1, 200), ("uniform", 4 << 20, 200), ("lopsided", (4 << 20) + 1, 1500),
])
def test_refinement_tiles_equal_level_launches(monkeypatch, ctx, dist, n, ppn):
    pos = _lopsided(n) if dist == "lopsided" else W.points(dist, n, 3)
    a = sf.Tree(pos, 20, ppn, ctx=ctx).dump()
    monkeypatch.setenv("SFMM_TREE_REFINE", "levels")
    b = sf.Tree(pos, 20, ppn, ctx=ctx).dump()
    assert a.keys() == b.keys()
    for k in a:
        assert np.array_equal(a[k], b[k]), k
