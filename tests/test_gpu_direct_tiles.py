"""The direct-sum kernel at the edges of its target blocks, source tiles and
chunks, for one to three charge components, against numpy FP64 sums (rsqrt in
place of a square root and divisions: 1e-13 of the sum of magnitudes)."""
import numpy as np
import pytest

import simplefmm_b200 as sf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("qdim", [1, 2, 3])
@pytest.mark.parametrize("n,nt", [(1, 1), (2, 2), (127, 127), (129, 64), (511, 255), (1025, 257), (3000, 513)])
def test_direct_edges(n, nt, qdim):
    rng = np.random.default_rng(n + nt)
    pos = rng.random((n, 3))
    q = rng.uniform(-1, 1, (n,) if qdim == 1 else (n, qdim))
    tg = rng.integers(0, n, nt)
    pot, fld = sf.direct(pos, q, tg, field=qdim != 2)
    d = pos[tg][:, None, :] - pos[None, :, :]
    r2 = (d * d).sum(-1)
    r2[np.arange(nt), tg] = np.inf
    ir = 1.0 / np.sqrt(r2)
    q2 = q.reshape(n, -1)
    scale = (np.abs(ir) @ np.abs(q2)).max() + 1e-300
    np.testing.assert_allclose(pot.reshape(nt, -1), ir @ q2, rtol=0, atol=1e-13 * scale)
    if qdim == 2:
        return
    w = ir ** 3
    d = np.where(np.isfinite(r2)[..., None], d, 0.0)
    if qdim == 1:
        f = ((w * q)[..., None] * d).sum(1)
    else:
        f = (w[..., None] * np.cross(np.broadcast_to(q, d.shape), d)).sum(1)
    np.testing.assert_allclose(fld, f, rtol=0, atol=1e-13 * ((ir ** 2) @ np.abs(q2)).sum(-1).max() + 1e-300)
