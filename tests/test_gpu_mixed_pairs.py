"""The persistent Jacobi form of the mixed solve with the FP32 pair kernels against
the per-kernel form: the same FP32 values and FP64 sums in the same order, so the
solutions, the iteration counts and the residual histories are equal bit for bit.
One tile; half a row block; fewer row blocks than SMs; tiles of every mask; more row
blocks than SMs; several rows per thread; a warm start; the iteration cap."""
import numpy as np
import pytest

from dachshund_gb300 import DsError, MixedParams, SignalCovarParams, WFVectorSN, WFVectorW, synth

pytestmark = pytest.mark.gpu
S = SignalCovarParams(synth.VAR_S, synth.L_PERP, synth.L_PARA, eval="exact")


def records(n, clumped=False):
    rng = np.random.default_rng(n)
    side = (12.5 * n) ** (1 / 3)
    rec = np.empty((n, 5))
    rec[:, :3] = rng.uniform(0, side, (n, 3))
    if clumped:  # half the pixels in a tenth of the box, the rest far apart
        rec[: n // 2, :3] *= 0.1 ** (1 / 3)
        rec[n // 2:, :3] *= 30.0
    rec[:, 3] = rng.uniform(0.05, 0.3, n)
    rec[:, 4] = rng.standard_normal(n) + 1.0
    return rec


def both(op, *args):
    out = []
    for form in ("auto", "graph"):
        op.set_iteration_form(form)
        out.append(op.solve_mixed(*args))
    (x, r), (xg, rg) = out
    assert r.num_iters == rg.num_iters and r.n_outer == rg.n_outer
    np.testing.assert_array_equal(x, xg)
    np.testing.assert_array_equal(r.residual_norms, rg.residual_norms)
    return x, r


@pytest.mark.parametrize("cls", [WFVectorSN, WFVectorW])
@pytest.mark.parametrize("n,clumped", [(1, False), (33, False), (129, False), (300, False),
                                       (5000, True), (20001, False)])
def test_forms_equal(ctx, cls, n, clumped):
    op = cls(ctx, records(n, clumped), S)
    x, r = both(op, MixedParams(tol=1e-10))
    assert r.success
    both(op, MixedParams(tol=1e-10), 0.999 * x)
    _, r = both(op, MixedParams(tol=1e-14, max_iter=3))
    assert r.num_iters <= 3
    op.close()


@pytest.mark.parametrize("n", [41000, 90000])
def test_forms_equal_large(ctx, n):
    op = WFVectorW(ctx, records(n), S)
    _, r = both(op, MixedParams(tol=1e-6))
    assert r.success
    op.close()


def test_barrier_timeout(ctx):
    op = WFVectorW(ctx, records(3001), S)
    ctx.set_wait_limit(1)
    try:
        with pytest.raises(DsError):
            op.solve_mixed(MixedParams(tol=1e-10))
    finally:
        ctx.set_wait_limit(0)
    x, r = op.solve_mixed(MixedParams(tol=1e-10))
    assert r.success
    op.close()
