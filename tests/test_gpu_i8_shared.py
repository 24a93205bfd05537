"""The tensor-core M2L's shared operator rows (orders >= 7) on the GPU: at each
side of the rule and of a row chunk, against the FP64 path (5e-7 relative L2,
the mixed M2L's bound), and one output alone against both (integer sums: the
same bits)."""
import numpy as np
import pytest

import simplefmm_b200 as sf
from conftest import rel_l2
from simplefmm_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [6, 7, 9, 10, 12])
@pytest.mark.parametrize("n,qdim", [(3_000, 1), (20_011, 1), (9_001, 3)])
def test_i8_shared_rows(p, n, qdim):
    ctx = sf.Context(0)
    pos = W.points("plummer", n, 50 + p)
    q = W.charges(n, 50 + p, dim=qdim)
    t = sf.Tree(pos, 20, 32, ctx=ctx)
    shape = (n,) if qdim == 1 else (n, qdim)

    def run(precision, pot, field):
        P, F = (np.zeros(shape) if pot else None), (np.zeros((n, 3)) if field else None)
        sf.Plan(t, p, qdim, precision=precision).evaluate(q, P, F)
        return P, F

    P, F = run("mixed", True, True)
    P64, F64 = run("fp64", True, True)
    assert rel_l2(P, P64) < 5e-7 and rel_l2(F, F64) < 5e-7
    assert np.array_equal(run("mixed", True, False)[0], P)
    assert np.array_equal(run("mixed", False, True)[1], F)
