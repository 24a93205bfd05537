"""Direct sums near the ends of the type's range: fields that are normal numbers
although q / r^3 is not.  Points and charges are scaled by powers of two, so the sums are
those of the unscaled set with other exponents."""
import numpy as np
import pytest

import simplefmm_b200 as sf
from conftest import rel_err_per_target

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("qdim", [1, 3])
@pytest.mark.parametrize("ex,eq", [(0, 0), (-345, 0), (-30, 946), (60, -880), (200, -500)])
def test_fields_beyond_the_range_of_q_over_r3(qdim, ex, eq):
    n = 700                                                  # two source chunks
    rng = np.random.default_rng(8)
    x, q = rng.random((n, 3)), rng.uniform(-1, 1, (n,) if qdim == 1 else (n, qdim))
    t = np.arange(0, n, 3)
    d = x[t, None] - x[None]
    r = np.sqrt((d * d).sum(-1))
    r[np.arange(len(t)), t] = np.inf
    Q = q.reshape(n, qdim)
    pot = (Q[None] / r[..., None]).sum(1)
    if qdim == 1:
        fld = (Q[None] * d / r[..., None] ** 3).sum(1)
    else:
        fld = (np.cross(Q[None], d) / r[..., None] ** 3).sum(1)
    sp, sf_ = (np.abs(Q).sum(1)[None] / r).sum(1), (np.abs(Q).sum(1)[None] / r ** 2).sum(1)
    P, F = sf.direct(np.ldexp(x, ex), np.ldexp(q, eq), t)
    # 700 terms of a few roundings each, relative to the sum of their sizes
    assert rel_err_per_target(np.ldexp(P.reshape(-1, qdim), ex - eq), pot, sp) < 1e-13
    assert rel_err_per_target(np.ldexp(F, 2 * ex - eq), fld, sf_) < 1e-13
