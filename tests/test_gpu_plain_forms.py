"""A plain solve of few pixels in the form without grid barriers."""
import numpy as np
import pytest

import oracle
from dachshund_gb300 import PCGParams, SignalCovarParams, WFVectorW, synth

pytestmark = pytest.mark.gpu
VS, LP, LQ = synth.VAR_S, synth.L_PERP, synth.L_PARA


def records(n):
    rng = np.random.default_rng(n)
    rec = np.empty((n, 5))
    rec[:, :3] = rng.uniform(0, (12.5 * n) ** (1 / 3), (n, 3))
    rec[:, 3] = 1 / rng.uniform(0.05, 0.3, n)
    rec[:, 4] = rng.standard_normal(n)
    return rec


@pytest.mark.parametrize("n", [1, 129, 4000])
def test_kernels_one_by_one(ctx, n):
    """The form of iteration "graph" has no barrier to time out, and its recurrence is
    the cooperative one's: FP64 CG drifts from the true residual by rounding alone,
    below 1e-13 |b| here (200 iterations of 2^-53 |A| |x| each, |A| |x| < 30 |b|)."""
    rec = records(n)
    op = WFVectorW(ctx, rec, SignalCovarParams(VS, LP, LQ))
    op.set_iteration_form("graph")
    ctx.set_wait_limit(1)
    try:
        x, res = op.solve_pcg(PCGParams(2000, 50, 1e-10))
    finally:
        ctx.set_wait_limit(0)
    assert res.success and res.residual_norms.size == res.num_iters + 1
    r = oracle.A_residual("w", rec, x / rec[:, 3], VS, LP, LQ, exact=False)
    assert abs(np.linalg.norm(r) - res.final_norm) <= 1e-12 * res.norm_b
    op.set_iteration_form("auto")
    xa, ra = op.solve_pcg(PCGParams(2000, 50, 1e-10))
    assert ra.success
    # both residuals <= 1e-10 |b|, A >= I in the W form
    assert np.linalg.norm((x - xa) / rec[:, 3]) <= 2.1e-10 * res.norm_b
    op.close()
