"""The persistent mixed solve at block shapes that leave threads over (n_per not
dividing the CTA, ragged last cluster) and at the largest blocks, against the
per-kernel form of the same solve.

Bound: both stop on the FP64-accurate residual |b - A x| <= tol |b| and, in the
W form, A >= I, so the unscaled solutions y = x / w differ by at most 2 tol |b|."""
import numpy as np
import pytest

from dachshund_gb300 import MixedParams, SignalCovarParams, WFVectorW, pixel_to_wpixel, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_sk,n_per,cluster,band", [
    (5, 7, 4, 3), (31, 45, 4, 16), (103, 33, 4, 16), (41, 171, 4, 16), (17, 250, 4, 16),
    (9, 256, 4, 16), (10, 341, 3, 16), (6, 511, 2, 8), (3, 512, 2, 2), (2, 600, 1, 16)])
def test_forms_agree(ctx, n_sk, n_per, cluster, band):
    w = synth.small(n_sk, n_per, float(np.ceil(2.5 * np.sqrt(n_sk))), seed=n_per)
    rec = pixel_to_wpixel(w.pixels)
    op = WFVectorW(ctx, rec, SignalCovarParams(w.var_s, w.l_perp, w.l_para, eval="exact"))
    op.set_cluster_preconditioner(n_sk, n_per, cluster, min(band, cluster * n_per - 1))
    op.set_skewer_grid(n_sk, n_per)
    tol, y = 1e-11, []
    for form in ("auto", "graph"):
        op.set_iteration_form(form)
        x, res = op.solve_mixed(MixedParams(tol=tol))
        assert res.success
        y.append(x / rec[:, 3])
    assert np.linalg.norm(y[0] - y[1]) <= 2.1 * tol * res.norm_b
    op.close()
