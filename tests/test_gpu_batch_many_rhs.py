"""Batched solves with many right-hand sides (the API takes up to 1,024).

Bound between two solves of a system: both stop on the FP64-accurate residual
|b - A x| <= tol |b| and, in the W form, A >= I, so the unscaled solutions y = x / w
differ by at most 2 tol |b| (plus the residual's own error, far below)."""
import numpy as np
import pytest

from dachshund_gb300 import BatchSolver, MixedParams, SignalCovarParams, pixel_to_wpixel, synth

pytestmark = pytest.mark.gpu
EXACT = SignalCovarParams(synth.VAR_S, synth.L_PERP, synth.L_PARA, eval="exact")
TOL = 1e-9


@pytest.mark.parametrize("R", [512, 513, 768, 800, 1000, 1023, 1024])
def test_many_right_hand_sides(ctx, R):
    recs = [pixel_to_wpixel(synth.small(n_sk, 40, 6.0, seed=n_sk).pixels) for n_sk in (5, 2)]
    n = sum(len(r) for r in recs)
    rhs = np.random.default_rng(R).standard_normal((n, R))
    b = BatchSolver(ctx, "w", recs, EXACT, R)
    x, res = b.solve_mixed(rhs, MixedParams(tol=TOL))
    b.close()
    assert res.converged.all()
    w = np.concatenate([r[:, 3] for r in recs])[:, None]
    cols = np.unique(np.r_[np.arange(0, R, 97), 510, 511, min(512, R - 1), R - 1])
    few = BatchSolver(ctx, "w", recs, EXACT, len(cols))
    y, res = few.solve_mixed(np.ascontiguousarray(rhs[:, cols]), MixedParams(tol=TOL))
    few.close()
    assert res.converged.all()
    lo = 0
    for r in recs:
        s = slice(lo, lo + len(r))
        lo += len(r)
        d = np.linalg.norm((x[s][:, cols] - y[s]) / w[s], axis=0)
        assert (d <= 2.1 * TOL * np.linalg.norm(rhs[s][:, cols], axis=0)).all()
