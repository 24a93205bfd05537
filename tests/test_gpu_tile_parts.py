"""The tiled FP64 M2L adds a tile's six parts in one fixed order, whether a block
runs them in turn or each has a block of its own and their sums are added
afterwards: the results are the same bit for bit (csrc/m2l_tile.cu)."""
import numpy as np
import pytest

import simplefmm_b200 as sf
from simplefmm_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dist,n,p,qdim,leaf", [("plummer", 2_003, 10, 1, 64), ("plummer", 30_011, 6, 1, 32),
                                                ("plummer", 12_007, 9, 3, 32), ("uniform", 20_001, 2, 2, 32),
                                                ("gauss2", 25_013, 12, 1, 64)])
def test_parts_in_turn_or_apart(monkeypatch, dist, n, p, qdim, leaf):
    ctx = sf.Context(0)
    pos, q = 0.37 * W.points(dist, n, p), W.charges(n, p, dim=qdim)     # a root cube that is no power of two wide
    tree = sf.Tree(pos, 20, leaf, ctx=ctx)
    out = []
    for kernel in (None, "whole"):
        if kernel:
            monkeypatch.setenv("SFMM_M2L_KERNEL", kernel)
        plan = sf.Plan(tree, p, qdim)
        if kernel:
            monkeypatch.delenv("SFMM_M2L_KERNEL")
        P = np.zeros((n,) if qdim == 1 else (n, qdim))
        F = np.zeros((n, 3)) if qdim != 2 else None
        plan.evaluate(q, P, F)
        out.append((P, F))
    (pa, fa), (pb, fb) = out
    assert np.array_equal(pa, pb) and (fa is None or np.array_equal(fa, fb))


def test_large_batch_equals_batches_of_one():
    """Eight sets whose trees are small enough for parts apart, together too large for it."""
    sets = [(W.points("uniform", 60_000 + k, k), W.charges(60_000 + k, k)) for k in range(8)]
    ctx = sf.Context(0)
    assert all(4_000 < sf.Tree(x, 20, 64, ctx=ctx).stats()["nodes"] < 24 * 1024 for x, _ in sets)
    together = sf.solve_batch(sets, 5, leaf=64, ctx=ctx)
    for s, (P, F) in zip(sets, together):
        (p1, f1), = sf.solve_batch([s], 5, leaf=64, ctx=ctx)
        assert np.array_equal(P, p1) and np.array_equal(F, f1)
