"""The tiled FP64 M2L (csrc/m2l_tile.cu) against the row-owner kernel
(SFMM_M2L_KERNEL=rows) at the orders and sizes where its layout changes: row
tiles and K chunks that just fill or spill, narrow and full tiles, parts in
blocks of their own or added in turn, columns of one to three components, one
output alone, a tree of one split level, and sparse lists (group kernel).
Both sum the same terms in FP64 in another order: 1e-12 relative L2."""
import numpy as np
import pytest

import simplefmm_b200 as sf
from conftest import rel_l2
from simplefmm_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _both(monkeypatch, pos, q, p, qdim, leaf, pot=True, field=True):
    n = len(pos)
    ctx = sf.Context(0)
    t = sf.Tree(pos, 20, leaf, ctx=ctx)
    out = []
    for kernel in (None, "rows"):
        if kernel:
            monkeypatch.setenv("SFMM_M2L_KERNEL", kernel)
        pl = sf.Plan(t, p, qdim)
        if kernel:
            monkeypatch.delenv("SFMM_M2L_KERNEL")
        P = np.zeros((n,) if qdim == 1 else (n, qdim)) if pot else None
        F = np.zeros((n, 3)) if field and qdim != 2 else None
        pl.evaluate(q, P, F)
        out.append((P, F))
    for a, b in zip(*out):
        if a is not None:
            assert rel_l2(a, b) < 1e-12
    return t


@pytest.mark.parametrize("p", [2, 3, 6, 7, 8, 9, 10, 11, 12])
@pytest.mark.parametrize("n,leaf,qdim", [(1_500, 32, 1), (20_011, 16, 1), (6_007, 32, 3), (6_007, 32, 2)])
def test_tile_matches_rows(monkeypatch, p, n, leaf, qdim):
    _both(monkeypatch, W.points("plummer", n, p), W.charges(n, p, dim=qdim), p, qdim, leaf)


@pytest.mark.parametrize("p", [6, 8, 10, 12])
def test_tile_full_blocks(monkeypatch, p):
    n = 150_000                                    # more targets than a split tree has
    t = _both(monkeypatch, W.points("uniform", n, 3), W.charges(n, 3), p, 1, 4)
    assert t.stats()["nodes"] > 30_000


@pytest.mark.parametrize("pot,field", [(True, False), (False, True)])
@pytest.mark.parametrize("p,n,leaf", [(6, 30_000, 2), (10, 9_000, 32)])
def test_tile_one_output(monkeypatch, p, n, leaf, pot, field):
    _both(monkeypatch, W.points("uniform", n, 5), W.charges(n, 5), p, 1, leaf, pot, field)


def test_tile_single_level_and_sparse(monkeypatch):
    _both(monkeypatch, W.points("uniform", 600, 6), W.charges(600, 6), 8, 1, 32)       # depth 2
    _both(monkeypatch, W.points("shell", 60_000, 7), W.charges(60_000, 7), 8, 1, 64)   # group kernel


def test_batch_of_dense_and_sparse_sets():
    """A batch decides the kernel set by set: each set equals its batch of one."""
    sets = [(W.points(d, n, k), W.charges(n, k)) for k, (d, n) in
            enumerate([("shell", 30_000), ("plummer", 12_000), ("shell", 2_000), ("uniform", 9_001)])]
    ctx = sf.Context(0)
    together = sf.solve_batch(sets, 8, leaf=32, ctx=ctx)
    for s, (P, F) in zip(sets, together):
        (p1, f1), = sf.solve_batch([s], 8, leaf=32, ctx=ctx)
        assert np.array_equal(P, p1) and np.array_equal(F, f1)
