"""The serving loop and the memory of the tiled FP64 M2L's part sums
(csrc/tile_parts.h): a request is admitted without them where the budget has
no room, to the same results, and what requests take stays within what
admission counted, up to the largest trees that use part sums."""
import numpy as np
import pytest

import simplefmm_b200 as sf
from simplefmm_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _serve(pos, q, p, budget):
    srv = sf.Server(0, slots=2, memory_budget=budget)
    try:
        pot, fld, _ = srv.wait(srv.submit(pos, q, p, leaf=64))
        return pot, fld, srv.stats()["peak_bytes"], srv.memory()["worst_measured_over_estimate"]
    finally:
        srv.close()


@pytest.mark.parametrize("dist,n,p", [("plummer", 20_000, 10), ("plummer", 100_000, 8)])
def test_admitted_without_room_for_part_sums(dist, n, p):
    pos, q = W.points(dist, n, 3), W.charges(n, 3)
    pot, fld, peak, _ = _serve(pos, q, p, 8 << 30)
    pot2, fld2, peak2, ratio = _serve(pos, q, p, int(peak) - 1)
    assert peak2 < peak and ratio <= 1.0
    assert np.array_equal(pot, pot2) and np.array_equal(fld, fld2)


@pytest.mark.parametrize("dist,n,p,qdim", [("plummer", 370_000, 10, 1), ("plummer", 300_007, 12, 1), ("uniform", 215_000, 10, 3),
                                           ("shell", 100_000, 6, 1), ("uniform", 60_000, 5, 1), ("plummer", 2_000, 12, 3)])
def test_measured_memory_within_the_estimate(dist, n, p, qdim):
    ratio = _serve(W.points(dist, n, 4), W.charges(n, 4, dim=qdim), p, 8 << 30)[3]
    assert 0 < ratio <= 1.0
