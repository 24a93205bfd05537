"""A captured evaluation (fmm_plan_capture) after the plan was given a shard
and back: the graph launches on buffers the plan still holds, so a replay
gives the captured evaluation's results bit for bit, whatever was allocated
since."""
import pytest

import simplefmm_b200 as sf
from simplefmm_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,dist,n,p,leaf", [("fp64", "plummer", 40_000, 8, 32), ("fp64", "uniform", 150_000, 4, 4),
                                                     ("mixed", "plummer", 40_000, 8, 32)])
def test_replay_after_shard_switches(precision, dist, n, p, leaf):
    torch = pytest.importorskip("torch")
    ctx = sf.Context(0)
    pos, q = torch.from_numpy(W.points(dist, n, 5)).cuda(), torch.from_numpy(W.charges(n, 5)).cuda()
    tree = sf.Tree(pos, 20, leaf, ctx=ctx)
    plan = sf.Plan(tree, p, 1, precision=precision)
    pot, fld = torch.zeros(n, dtype=torch.float64, device="cuda"), torch.zeros(n, 3, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    plan.capture(q, pot, fld)

    def replay():
        pot.zero_()
        fld.zero_()
        torch.cuda.synchronize()
        plan.replay()
        ctx.synchronize()
        return pot.clone(), fld.clone()

    want = replay()
    others = []
    for index, count in ((0, 1), (1, 3), (0, 2), (0, 1)):
        plan.set_shard(index, count)
        # plans of the same tree take over whatever the switch released
        others.append(sf.Plan(tree, p, 1, precision=precision))
        o = torch.zeros(n, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        others[-1].evaluate(q, o, None)
        got = replay()
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    # unsharded again: a plain evaluation (a mixed plan keeps the FP64 M2L a shard switch gave it)
    o, f = torch.zeros_like(pot), torch.zeros_like(fld)
    torch.cuda.synchronize()
    plan.evaluate(q, o, f)
    ctx.synchronize()
    if precision == "fp64":
        assert torch.equal(o, want[0]) and torch.equal(f, want[1])
    else:
        assert float((o - want[0]).norm() / want[0].norm()) < 1e-6
