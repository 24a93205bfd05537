"""The mixed near field of scalar charges (sources in packed pairs) at the edges
of its target passes, source slices, tiles and odd last pairs: one leaf, so the
near field is everything.  Against the FP64 near field: FP32 products and tile
sums of at most 128 terms, 1e-5 of the largest output."""
import numpy as np
import pytest

import simplefmm_b200 as sf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 5, 31, 33, 48, 63, 65, 95, 97, 127, 128, 129, 191, 255, 257, 400])
def test_mixed_near_field_edges(n):
    rng = np.random.default_rng(n)
    pos, q = rng.random((n, 3)), rng.uniform(-1, 1, n)
    if n == 1:
        pos = np.array([[0.1, 0.2, 0.3]])
    ctx = sf.Context(0)
    t = sf.Tree(pos, 20, 512, ctx=ctx, box=((0.0, 0.0, 0.0), 1.0))
    assert t.depth == 0
    for pot, field in ((True, True), (True, False), (False, True)):
        out = []
        for precision in ("mixed", "fp64"):
            P, F = (np.zeros(n) if pot else None), (np.zeros((n, 3)) if field else None)
            sf.Plan(t, 6, 1, precision=precision).evaluate(q, P, F)
            out.append((P, F))
        for m, f in zip(*out):
            if m is not None:
                assert np.max(np.abs(m - f)) <= 1e-5 * np.max(np.abs(f)) if n > 1 else np.array_equal(m, f)
