"""The batch graphs' key (csrc/capi.cu evaluate_graph): batches of one depth,
order and outputs whose launch sequences differ -- the tiled M2L's parts apart
with a sum after it, or in turn -- keep a graph each, and taking turns updates
both in place instead of instantiating one anew every time."""
import pytest

import simplefmm_b200 as sf
from simplefmm_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _batch(sets, seed):
    return [(W.points("uniform", 60_000 + k, seed + k), W.charges(60_000 + k, seed + k)) for k in range(sets)]


def test_alternating_launch_sequences_keep_their_graphs():
    ctx = sf.Context(0)
    for x, _ in _batch(2, 0):                      # 4,681 nodes a set, 4 levels: two sets below 24K rows, eight above
        t = sf.Tree(x, 20, 64, ctx=ctx)
        assert t.depth == 4 and 8 * t.stats()["nodes"] > 24 * 1024 + 8 * 73
    for i in range(3):
        sf.solve_batch(_batch(2, 10 * i), 4, leaf=64, ctx=ctx)
        sf.solve_batch(_batch(8, 10 * i + 5), 4, leaf=64, ctx=ctx)
    assert sf.batch_graph_stats(ctx) == {"instantiated": 2, "updated": 4}
