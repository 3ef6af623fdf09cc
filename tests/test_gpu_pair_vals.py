"""The FP64 operator's pair search and stored pair values (csrc/ds_pairhit.cuh,
csrc/pair_vals.cu, csrc/pair_f64.cu) against the CPU oracle.

Bound per element: every term of a row's sum is the oracle's within its own
rounding (argument below 40, three roundings each, exp or interpolation and two
scalings: under 128 units of 2^-53), and a sum of k terms taken in any order is
within k 2^-53 of the sum of their magnitudes, so |b_i - ref_i| <= (n + 128)
2^-53 (|A| |a|)_i, plus the terms beyond the exact kernel's cutoff, at most
exp(-40) of var_s each.
"""
import numpy as np
import pytest

import oracle
from dachshund_gb300 import (MapGrid, MixedParams, PCGParams, SignalCovarParams, WFVectorSN,
                             WFVectorW, synth)

pytestmark = pytest.mark.gpu
VS, LP, LQ = synth.VAR_S, synth.L_PERP, synth.L_PARA


def records(form, n, seed, spread=1.0, shift=0.0):
    """n scattered records at the workloads' density times spread^-3."""
    rng = np.random.default_rng(seed)
    side = spread * (12.5 * n) ** (1 / 3)
    rec = np.empty((n, 5))
    rec[:, :3] = shift + rng.uniform(0, side, (n, 3))
    noise = rng.uniform(0.05, 0.3, n)
    rec[:, 3] = noise ** 2 if form == "sn" else 1 / noise
    rec[:, 4] = rng.standard_normal(n)
    return rec


def bound(form, rec, a, scale, exact):
    n = len(rec)
    w = np.ones(n) if form == "sn" else rec[:, 3]
    cut = np.exp(-40.0) * VS * w * np.sum(w * np.abs(a)) if exact else 0.0
    return (n + 128) * 2.0 ** -53 * scale + cut


@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("form", ["sn", "w"])
@pytest.mark.parametrize("n,spread,shift", [(1, 1, 0), (31, 1, 0), (33, 1, 1e4), (129, 1, -3e3),
                                            (1000, 0.2, 0), (3001, 1, 0), (3001, 50, 1e5),
                                            (20000, 1, 0)])
def test_products_vs_oracle(ctx, form, exact, n, spread, shift):
    rec = records(form, n, n, spread, shift)
    a = np.random.default_rng(1).standard_normal(n)
    cls = WFVectorSN if form == "sn" else WFVectorW
    op = cls(ctx, rec, SignalCovarParams(VS, LP, LQ, eval="exact" if exact else "table"))
    ref = oracle.A_product(form, rec, a, VS, LP, LQ, exact=exact)
    lim = bound(form, rec, a, oracle.A_product(form, rec, np.abs(a), VS, LP, LQ, exact=exact),
                exact)
    assert np.all(np.abs(op.A_product(a) - ref) <= lim)
    assert np.all(np.abs(op.A_product(a) - ref) <= lim)  # the list a second time
    r = oracle.A_residual(form, rec, a, VS, LP, LQ, exact=exact)
    assert np.all(np.abs(op.A_residual(a) - r) <= lim + 2.0 ** -52 * np.abs(r))
    op.close()


def test_wide_indices_rows_vs_oracle(ctx):
    n = 66000  # column indices beyond 16 bits
    rec = records("w", n, 5)
    a = np.random.default_rng(1).standard_normal(n)
    op = WFVectorW(ctx, rec, SignalCovarParams(VS, LP, LQ))
    got = op.A_product(a)
    for r0 in (0, 33000, n - 32):
        ref = oracle.A_product_rows("w", rec, a, r0, r0 + 32, VS, LP, LQ)
        lim = oracle.A_product_rows("w", rec, np.abs(a), r0, r0 + 32, VS, LP, LQ)
        assert np.all(np.abs(got[r0:r0 + 32] - ref) <= (n + 128) * 2.0 ** -53 * lim)
    op.close()


@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("n,m,spread", [(1, 1, 1), (129, 33, 1), (3001, 4097, 1), (3001, 500, 50)])
def test_map_vs_oracle(ctx, exact, n, m, spread):
    rec = records("w", n, n, spread)
    pts = records("w", m, m + 1, spread)[:, :3].copy()
    x = np.random.default_rng(1).standard_normal(n)
    op = WFVectorW(ctx, rec, SignalCovarParams(VS, LP, LQ, eval="exact" if exact else "table"))
    grid = MapGrid(ctx, pts)
    ref = oracle.smp_product(rec[:, :3], pts, x, VS, LP, LQ, exact=exact)
    lim = oracle.smp_product(rec[:, :3], pts, np.abs(x), VS, LP, LQ, exact=exact)
    lim = (n + 128) * 2.0 ** -53 * lim + np.exp(-40.0) * VS * np.sum(np.abs(x))
    assert np.all(np.abs(grid.product(op, x) - ref) <= lim)
    grid.close()
    op.close()


@pytest.mark.parametrize("cutoff,spread", [(5.0, 1), (48.0, 1), (47.99, 1), (48.01, 1),
                                           (40.0, 3e3), (40.0, 3e4)])
def test_fixed_point_and_fp64_ranges(ctx, cutoff, spread):
    """The exact kernel on both sides of the fixed-point range (cutoff 48, extent
    2^16 scaled units; spread 3e3 is 2^15.1 of them, 3e4 beyond), products and map:
    the oracle has no cutoff, the terms beyond it are at most exp(-cutoff)."""
    n, m = 3001, 777
    rec = records("w", n, n, spread)
    rec[:3000:3, :3] = rec[1:3000:3, :3] + 0.5  # close pairs in the sparse sets
    pts = rec[:m, :3] + 1.25
    a = np.random.default_rng(1).standard_normal(n)
    op = WFVectorW(ctx, rec, SignalCovarParams(VS, LP, LQ, eval="exact", exact_cutoff=cutoff))
    lim = oracle.A_product("w", rec, np.abs(a), VS, LP, LQ, exact=True)
    w = rec[:, 3]
    lim = (n + 128) * 2.0 ** -53 * lim + np.exp(-cutoff) * VS * w * np.sum(w * np.abs(a))
    assert np.all(np.abs(op.A_product(a) - oracle.A_product("w", rec, a, VS, LP, LQ, exact=True))
                  <= lim)
    grid = MapGrid(ctx, pts)
    ref = oracle.smp_product(rec[:, :3], pts, a, VS, LP, LQ, exact=True)
    lim = oracle.smp_product(rec[:, :3], pts, np.abs(a), VS, LP, LQ, exact=True)
    lim = (n + 128) * 2.0 ** -53 * lim + np.exp(-cutoff) * VS * np.sum(np.abs(a))
    assert np.all(np.abs(grid.product(op, a) - ref) <= lim)
    grid.close()
    op.close()


def test_residual_evaluated_on_every_call(ctx):
    """A cutoff beyond the float-float range: the mixed form's outer residual is
    the evaluating FP64 kernel's; its solution is the FP64 solve's to tol."""
    rec = records("w", 3001, 9)
    op = WFVectorW(ctx, rec, SignalCovarParams(VS, LP, LQ, eval="exact", exact_cutoff=80.0))
    x, res = op.solve_mixed(MixedParams(tol=1e-11))
    xp, rp = op.solve_pcg(PCGParams(2000, 50, 1e-11))
    assert res.success and rp.success
    # both residuals <= 1e-11 |b|, A >= I in the W form (x = w y, w in [3.3, 20])
    assert np.linalg.norm((x - xp) / rec[:, 3]) <= 2.1e-11 * res.norm_b
    op.close()


@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("n", [1, 33, 129, 4000, 5000, 9700, 9800])
def test_pcg_forms_vs_oracle_residual(ctx, n, exact):
    """One CTA per slice (up to one per SM, two, and beyond the cooperative form):
    the recurrence's |r| and the true residual by the oracle's operator.  FP64 CG
    drifts from the true residual by rounding alone, below 1e-13 |b| here (200
    iterations of 2^-53 |A| |x| each, |A| |x| < 30 |b|)."""
    rec = records("w", n, n)
    op = WFVectorW(ctx, rec, SignalCovarParams(VS, LP, LQ, eval="exact" if exact else "table"))
    x, res = op.solve_pcg(PCGParams(2000, 50, 1e-10))
    assert res.success and res.final_norm <= 1e-10 * res.norm_b
    assert res.residual_norms.size == res.num_iters + 1
    r = oracle.A_residual("w", rec, x / rec[:, 3], VS, LP, LQ, exact=exact)
    assert abs(np.linalg.norm(r) - res.final_norm) <= 1e-12 * res.norm_b
    # a start from the solution stops after the first iteration's test; the cap counts
    x2, r2 = op.solve_pcg(PCGParams(3, 2, 0.0), x / rec[:, 3])
    assert not r2.success and r2.num_iters == 3 and r2.residual_norms.size == 3
    op.close()


def test_pcg_barrier_timeout(ctx):
    from dachshund_gb300 import DsError

    op = WFVectorW(ctx, records("w", 1000, 3), SignalCovarParams(VS, LP, LQ))
    ctx.set_wait_limit(1)
    try:
        with pytest.raises(DsError) as e:
            op.solve_pcg(PCGParams(100, 50, 1e-8))
        assert e.value.code == 8
    finally:
        ctx.set_wait_limit(0)
    assert op.solve_pcg(PCGParams(1000, 50, 1e-8))[1].success
    op.close()
