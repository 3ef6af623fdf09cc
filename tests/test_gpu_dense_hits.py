"""The FP64 pair kernel where the correlation lengths reach the box's size, so that
every pair of a block interacts: blocks without the queue, the ragged last ones with it,
and lengths where both kinds alternate.  Bound as in test_gpu_pair_vals."""
import numpy as np
import pytest

import oracle
from dachshund_gb300 import MapGrid, SignalCovarParams, WFVectorW, sigma_m_noise_dom

pytestmark = pytest.mark.gpu
VS = 0.0625


@pytest.mark.parametrize("scale", [30.0, 0.3])  # length over the box's side
@pytest.mark.parametrize("n,m", [(31, 1), (32, 32), (33, 33), (128, 127), (500, 129),
                                 (1000, 500)])
def test_map_and_noise_vs_oracle(ctx, n, m, scale):
    rng = np.random.default_rng(n + m)
    side = (12.5 * n) ** (1 / 3)
    rec = np.empty((n, 5))
    rec[:, :3] = rng.uniform(0, side, (n, 3))
    rec[:, 3] = 1 / rng.uniform(0.05, 0.3, n)
    rec[:, 4] = rng.standard_normal(n)
    pts = rng.uniform(0, side, (m, 3))
    lp = scale * side
    sp = SignalCovarParams(VS, lp, lp)
    x = rng.standard_normal(n)
    op, grid = WFVectorW(ctx, rec, sp), MapGrid(ctx, pts)
    ref = oracle.smp_product(rec[:, :3], pts, x, VS, lp, lp)
    lim = oracle.smp_product(rec[:, :3], pts, np.abs(x), VS, lp, lp)
    assert np.all(np.abs(grid.product(op, x) - ref) <= (n + 128) * 2.0 ** -53 * lim)
    grid.close()
    op.close()
    # the noise sum's terms are squares over N > 0: its bound is of its own value
    nrec = rec.copy()
    nrec[:, 3] = 1 / rec[:, 3] ** 2
    got = sigma_m_noise_dom(ctx, nrec, pts, sp)
    one = np.stack([oracle.smp_product(nrec[k:k + 1, :3], pts, np.ones(1), VS, lp, lp)
                    for k in range(n)])
    ref = (one ** 2 / nrec[:, 3:4]).sum(0)
    assert np.all(np.abs(got - ref) <= 2 * (n + 128) * 2.0 ** -53 * ref)
