"""Plans on new points of nearly the same number, made and released one after
the other: the part sums' block of one plan serves the next (csrc/tile_parts.h),
so device memory does not grow by one such block per plan."""
import numpy as np
import pytest

import simplefmm_b200 as sf
from simplefmm_b200 import workloads as W

pytestmark = pytest.mark.gpu


def test_fresh_plans_reuse_the_part_sums_block():
    torch = pytest.importorskip("torch")
    p, ctx = 10, sf.Context(0)
    free = []
    for k in range(8):
        n = 60_000 + 7 * k
        tree = sf.Tree(W.points("plummer", n, 100 + k), 20, 64, ctx=ctx)
        nodes = tree.stats()["nodes"]
        plan = sf.Plan(tree, p, 1)
        pot = np.zeros(n)
        plan.evaluate(W.charges(n, k), pot, None)
        plan.close()
        tree.close()
        free.append(torch.cuda.mem_get_info()[0])
    block = 6 * 210 * 16 * nodes                   # bytes of the part sums
    assert block > 60 << 20
    assert free[1] - free[-1] < 3 * block          # six plans later (a block each: 6 x)
