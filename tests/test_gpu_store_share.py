"""The forms that evaluate pairs on every product, which run where the stored values
would take more than the context's share of the device memory: with a share of 0 they
run at any size.  Bounds as in test_gpu_pair_vals."""
import contextlib

import numpy as np
import pytest

import oracle
from dachshund_gb300 import (DsError, MixedParams, PCGParams, SignalCovarParams, WFVectorSN,
                             WFVectorW, map_covar_diag, synth)

pytestmark = pytest.mark.gpu
VS, LP, LQ = synth.VAR_S, synth.L_PERP, synth.L_PARA


def records(form, n, spread=1.0, seed=None):
    rng = np.random.default_rng(n if seed is None else seed)
    rec = np.empty((n, 5))
    rec[:, :3] = rng.uniform(0, spread * (12.5 * n) ** (1 / 3), (n, 3))
    noise = rng.uniform(0.05, 0.3, n)
    rec[:, 3] = noise ** 2 if form == "sn" else 1 / noise
    rec[:, 4] = rng.standard_normal(n)
    return rec


def params(exact):
    return SignalCovarParams(VS, LP, LQ, eval="exact" if exact else "table")


@contextlib.contextmanager
def share(ctx, s):
    ctx.set_store_share(s)
    try:
        yield
    finally:
        ctx.set_store_share()


@pytest.mark.parametrize("form", ["sn", "w"])
@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("n,spread", [(1, 1), (33, 1), (1000, 0.2), (3001, 1), (3001, 50),
                                      (20000, 1)])
def test_products_vs_oracle(ctx, form, exact, n, spread):
    rec = records(form, n, spread)
    a = np.random.default_rng(1).standard_normal(n)
    op = (WFVectorSN if form == "sn" else WFVectorW)(ctx, rec, params(exact))
    ref = oracle.A_product(form, rec, a, VS, LP, LQ, exact=exact)
    lim = (n + 128) * 2.0 ** -53 * oracle.A_product(form, rec, np.abs(a), VS, LP, LQ, exact=exact)
    if exact:
        w = np.ones(n) if form == "sn" else rec[:, 3]
        lim = lim + np.exp(-40.0) * VS * w * np.sum(w * np.abs(a))
    r = oracle.A_residual(form, rec, a, VS, LP, LQ, exact=exact)
    with share(ctx, 0.0):
        assert np.all(np.abs(op.A_product(a) - ref) <= lim)
        assert op.stored_bytes() == 0
        assert np.all(np.abs(op.A_residual(a) - r) <= lim + 2.0 ** -52 * np.abs(r))
    assert np.all(np.abs(op.A_product(a) - ref) <= lim)
    assert op.stored_bytes() > 0
    with share(ctx, 0.0):  # gives the values back
        assert np.all(np.abs(op.A_product(a) - ref) <= lim)
        assert op.stored_bytes() == 0
    op.close()


@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("n", [1, 33, 4000, 9800])
def test_pcg_vs_oracle_residual(ctx, n, exact):
    rec = records("w", n)
    op = WFVectorW(ctx, rec, params(exact))
    with share(ctx, 0.0):
        x, res = op.solve_pcg(PCGParams(2000, 50, 1e-10))
        assert op.stored_bytes() == 0
        x2, r2 = op.solve_pcg(PCGParams(3, 2, 0.0), x / rec[:, 3])
    assert res.success and res.final_norm <= 1e-10 * res.norm_b
    assert res.residual_norms.size == res.num_iters + 1
    r = oracle.A_residual("w", rec, x / rec[:, 3], VS, LP, LQ, exact=exact)
    assert abs(np.linalg.norm(r) - res.final_norm) <= 1e-12 * res.norm_b
    assert not r2.success and r2.num_iters == 3 and r2.residual_norms.size == 3
    op.close()


@pytest.mark.parametrize("n,m", [(100, 1), (3001, 17), (3001, 40)])
def test_covariance_forms(ctx, n, m):
    """sigma = b.x of solves to |r| <= tol |b|: x is within tol |b| / min N of the
    exact one in either form, and b.x within |b| times that."""
    rec, tol = records("sn", n), 1e-11
    pts = records("sn", m, (n / m) ** (1 / 3), seed=3)[:, :3].copy()
    pp = PCGParams(2000, 50, tol)
    s1, _, ok1 = map_covar_diag(ctx, rec, pts, params(False), pp)
    with share(ctx, 0.0):
        s0, _, ok0 = map_covar_diag(ctx, rec, pts, params(False), pp)
    assert ok0.all() and ok1.all()
    d2 = ((rec[:, None, :2] - pts[None, :, :2]) ** 2).sum(2) / (2 * LP ** 2)
    d2 += (rec[:, None, 2] - pts[None, :, 2]) ** 2 / (2 * LQ ** 2)
    bb = ((VS * np.exp(-d2)) ** 2).sum(0)
    # (the table's values are within 1e-3 of exp; 1.1 covers that)
    assert np.all(np.abs(s1 - s0) <= 1.1 * 2 * tol * bb / rec[:, 3].min())


@pytest.mark.parametrize("n", [300, 20001])
def test_mixed_forms_equal(ctx, n):
    """Without room for the row sums the per-kernel form runs: the same bits."""
    op = WFVectorW(ctx, records("w", n), params(True))
    x1, r1 = op.solve_mixed(MixedParams(tol=1e-10))
    with share(ctx, 0.0):
        ctx.set_wait_limit(1)  # (the persistent form would time out)
        try:
            x0, r0 = op.solve_mixed(MixedParams(tol=1e-10))
        finally:
            ctx.set_wait_limit(0)
    x2, r2 = op.solve_mixed(MixedParams(tol=1e-10))
    assert r1.success and r0.num_iters == r1.num_iters == r2.num_iters
    np.testing.assert_array_equal(x0, x1)
    np.testing.assert_array_equal(x2, x1)
    op.close()


def test_share_range(ctx):
    for s in (-0.1, 1.1, float("nan")):
        with pytest.raises(DsError):
            ctx.set_store_share(s)
    ctx.set_store_share()
