"""P2M with lanes over azimuthal orders (csrc/eval.cu) at every order:
even and odd orders (a middle order of its own or none), one to 32 points a
warp at a time, leaves of one point and of several rounds, one to three charge
components, one output alone.  Two checks, both on a tree whose near field is
the same: the solve equals the host restatement's (tests/native/emu.cpp, the
generic recurrences) to FP64 rounding, 1e-12 relative L2 (sums of about a
thousand terms of relative error 1e-16, amplified by the cancellation of
random charges); linear in the charges to the same bound."""
import numpy as np
import pytest

import simplefmm_b200 as sf
from conftest import rel_l2
from simplefmm_b200 import workloads as W
from test_ops_host import emu, run_emu  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    return sf.Context(0)


@pytest.mark.parametrize("p", range(17))
@pytest.mark.parametrize("n,leaf", [(700, 1), (1500, 70)])
def test_every_order_matches_host(emu, ctx, p, n, leaf):  # noqa: F811
    pos, q = W.points("uniform", n, p), W.charges(n, p)
    t = sf.Tree(pos, 20, leaf, ctx=ctx)
    assert t.depth >= 2
    P, F = np.zeros(n), np.zeros((n, 3))
    sf.Plan(t, p, 1).evaluate(q, P, F)
    hp, hf = run_emu(emu, t.dump(), pos, q, p)
    assert rel_l2(P, hp) < 1e-12 and rel_l2(F, hf) < 1e-12


@pytest.mark.parametrize("p", [3, 8, 13])
@pytest.mark.parametrize("qdim,pot,field", [(1, True, False), (1, False, True), (2, True, False), (3, True, True), (3, False, True)])
def test_components_are_linear(ctx, p, qdim, pot, field):
    n = 3000
    pos = W.points("plummer", n, 9)
    t = sf.Tree(pos, 20, 40, ctx=ctx)
    qs = [W.charges(n, s, dim=qdim) for s in (1, 2)]
    out = []
    for q in (qs[0], qs[1], qs[0] + 2.0 * qs[1]):
        P = np.zeros((n,) if qdim == 1 else (n, qdim)) if pot else None
        F = np.zeros((n, 3)) if field else None
        sf.Plan(t, p, qdim).evaluate(q, P, F)
        out.append((P, F))
    for a, b, c in zip(*out):
        if a is not None:
            assert rel_l2(c, a + 2.0 * b) < 1e-12
