"""The mixed-precision solve is the same in any units: with the data times 2^-k, or
the data times 2^k and every variance times 2^2k, all its vectors and scalars are
those of the unscaled solve times powers of two, so the iteration counts are equal
and the solutions equal bit for bit (2^-60 is 9e-19; the fluxes of physical units are about
1e-17).  The persistent solve's FP16 factor has no room for other variances."""
import numpy as np
import pytest

from dachshund_gb300 import (MixedParams, SignalCovarParams, WFVectorSN, pixel_to_npixel,
                             synth)

pytestmark = pytest.mark.gpu


def _solve(ctx, w, pixels, var, skewers, form):
    op = WFVectorSN(ctx, pixel_to_npixel(pixels), SignalCovarParams(var, w.l_perp, w.l_para,
                                                                    eval="exact"))
    if skewers:
        op.set_cluster_preconditioner(*skewers, 4, 16)
        op.set_skewer_grid(*skewers)
    op.set_iteration_form(form)
    x, res = op.solve_mixed(MixedParams(tol=1e-10))
    op.close()
    return x, res


@pytest.mark.parametrize("form,skewers,kd,kv", [
    ("auto", True, -60, 0), ("auto", True, 60, 0), ("graph", True, -60, -60),
    ("auto", False, -60, 0), ("auto", False, -60, -60), ("auto", False, 60, 60)])
def test_units(ctx, form, skewers, kd, kv):
    n_sk, n_per = 33, 45
    w = synth.small(n_sk, n_per, float(np.ceil(2.5 * np.sqrt(n_sk))), seed=7)
    pix = np.array(w.pixels)
    sk = (n_sk, n_per) if skewers else None
    x0, r0 = _solve(ctx, w, pix, w.var_s, sk, form)
    scaled = pix.copy()
    scaled[:, 3] *= 2.0 ** (kv // 2)  # the pixel's noise (standard deviation)
    scaled[:, 4] *= 2.0 ** kd
    x1, r1 = _solve(ctx, w, scaled, w.var_s * 2.0 ** kv, sk, form)
    assert r0.success and r1.success
    assert r1.num_iters == r0.num_iters
    np.testing.assert_array_equal(x1 * 2.0 ** (kv - kd), x0)
