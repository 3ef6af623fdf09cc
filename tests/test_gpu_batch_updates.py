"""Updates of the batched solve: one chunk's residual in segments, many chunks' in
whole items.

Bound between two solves of a chunk: both stop on the FP64-accurate residual
|b - A x| <= tol |b| and, in the W form, A >= I, so the unscaled solutions y = x / w
differ by at most 2 tol |b| (plus the residual's own error, far below)."""
import numpy as np
import pytest

from dachshund_gb300 import BatchSolver, MixedParams, SignalCovarParams, pixel_to_wpixel, synth

pytestmark = pytest.mark.gpu
EXACT = SignalCovarParams(synth.VAR_S, synth.L_PERP, synth.L_PARA, eval="exact")
TOL = 1e-9


def _chunk(seed, n_sk, n_per):
    pix = synth.small(n_sk, n_per, float(np.ceil(2.5 * np.sqrt(n_sk))), seed=seed).pixels
    return pixel_to_wpixel(pix)


def _solve(ctx, recs, rhs, variant, tol=TOL):
    b = BatchSolver(ctx, "w", recs, EXACT, rhs.shape[1])
    if variant == "cuda_core":
        b.set_variant(variant, 8 if rhs.shape[1] % 8 == 0 else 1)
    else:
        b.set_variant(variant)
    x, res = b.solve_mixed(rhs, MixedParams(tol=tol))
    b.close()
    assert res.converged.all()
    return x, res


# one tile and several; the copies' updates fall in the same iteration, as whole items
@pytest.mark.parametrize("n_sk,n_per,copies", [(4, 30, 700), (9, 45, 250)])
@pytest.mark.parametrize("R,variant", [(8, "cuda_core"), (16, "tensor")])
def test_copies_agree(ctx, n_sk, n_per, copies, R, variant):
    rec = _chunk(3, n_sk, n_per)
    rhs = np.random.default_rng(5).standard_normal((rec.shape[0], R))
    x1, r1 = _solve(ctx, [rec], rhs, variant)
    xm, rm = _solve(ctx, [rec] * copies, np.tile(rhs, (copies, 1)), variant)
    y1 = x1 / rec[:, 3:4]
    ym = xm.reshape(copies, *x1.shape) / rec[None, :, 3:4]
    bound = 2.1 * TOL * np.linalg.norm(rhs, axis=0)
    assert (np.linalg.norm(ym - y1, axis=1) <= bound).all()
    # the copies are the same problem: any two are equal bit for bit
    np.testing.assert_array_equal(xm.reshape(copies, -1), np.tile(xm[: len(rec)].ravel(), (copies, 1)))
