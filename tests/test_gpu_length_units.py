"""Products, maps and stored pair values do not depend on the unit of length: with
coordinates and correlation lengths times 2^k every FP64 quantity is the same up to a
power of two, so the table kernel's results are equal bit for bit, and the exact
kernel's within the bound of test_gpu_pair_vals.  Lengths of 1e21 (2^70 here) have
coefficients that are subnormal in FP32, 2^-70 overflows them, and the coordinates of
+-2^110 come near the ends of FP32's range."""
import numpy as np
import pytest

import oracle
from dachshund_gb300 import (MapGrid, PCGParams, SignalCovarParams, WFVectorSN, map_covar_diag,
                             smp_product, synth)

pytestmark = pytest.mark.gpu
VS, LP, LQ = synth.VAR_S, synth.L_PERP, synth.L_PARA
N, M = 3000, 700


def records(unit, n=N, seed=5):
    rng = np.random.default_rng(seed)
    rec = np.empty((n, 5))
    rec[:, :3] = rng.uniform(0, (12.5 * n) ** (1 / 3), (n, 3)) * unit
    rec[:, 3] = rng.uniform(0.05, 0.3, n) ** 2
    rec[:, 4] = rng.standard_normal(n)
    return rec


def params(unit, ev, **k):
    return SignalCovarParams(VS, LP * unit, LQ * unit, eval=ev, **k)


@pytest.mark.parametrize("ev", ["table", "exact"])
@pytest.mark.parametrize("k", [65, 70, 75, -70, 110, -110])
def test_units_of_length(ctx, ev, k):
    a = np.random.default_rng(1).standard_normal(N)
    out = []
    for unit in (1.0, 2.0 ** k):
        rec = records(unit)
        pts = records(unit, M, 6)[:, :3].copy()
        op = WFVectorSN(ctx, rec, params(unit, ev))
        grid = MapGrid(ctx, pts)
        out.append((op.A_product(a), grid.product(op, a)))
        grid.close()
        op.close()
    if ev == "table":
        for u, v in zip(*out):
            np.testing.assert_array_equal(u, v)
        return
    rec = records(1.0)
    pts = records(1.0, M, 6)[:, :3].copy()
    cut = np.exp(-40.0) * VS * np.sum(np.abs(a))
    lim = 2 * (N + 128) * 2.0 ** -53 * oracle.A_product("sn", rec, np.abs(a), VS, LP, LQ,
                                                        exact=True) + cut
    assert np.all(np.abs(out[1][0] - out[0][0]) <= lim)
    lim = 2 * (N + 128) * 2.0 ** -53 * oracle.smp_product(rec[:, :3], pts, np.abs(a), VS, LP, LQ,
                                                          exact=True) + cut
    assert np.all(np.abs(out[1][1] - out[0][1]) <= lim)


def test_covariance_in_units(ctx):
    """The table covariance's solves read the stored values: equal bit for bit."""
    got = [map_covar_diag(ctx, records(u), records(u, 5, 6)[:, :3].copy(), params(u, "table"),
                          PCGParams(500, 50, 1e-8)) for u in (1.0, 2.0 ** 70)]
    for u, v in zip(*got):
        np.testing.assert_array_equal(u, v)


def test_sparse_set_with_a_small_cutoff(ctx):
    """32 points 2,048 scaled units apart (a multiple of the fixed-point
    coordinates' period) and a cutoff of 1e-3: no two interact, although the search's
    threshold does not resolve them."""
    n = 32
    rec = np.zeros((n, 5))
    rec[:, 0] = 64.0 * 128 * np.arange(n)
    rec[:, 3] = 0.01
    a = np.random.default_rng(2).standard_normal(n)
    lp = 4 / np.sqrt(2.0)  # sqrt(c_perp) = 1/4 to rounding
    op = WFVectorSN(ctx, rec, SignalCovarParams(VS, lp, LQ, eval="exact", exact_cutoff=1e-3))
    ref = (VS + 0.01) * a
    assert np.all(np.abs(op.A_product(a) - ref) <= 8 * 2.0 ** -53 * np.abs(ref))
    op.close()


@pytest.mark.parametrize("ev", ["table", "exact"])
def test_infinite_length(ctx, ev):
    """An infinite perpendicular length: the kernel depends on z alone."""
    rec, pts = records(1.0), records(1.0, M, 6)[:, :3].copy()
    a = np.random.default_rng(1).standard_normal(N)
    got = smp_product(ctx, rec[:, :3].copy(), pts, SignalCovarParams(VS, np.inf, LQ, eval=ev), a)
    flat, flat_p = rec[:, :3].copy(), pts.copy()
    flat[:, :2] = flat_p[:, :2] = 0.0
    ref = oracle.smp_product(flat, flat_p, a, VS, LP, LQ, exact=ev == "exact")
    lim = oracle.smp_product(flat, flat_p, np.abs(a), VS, LP, LQ, exact=ev == "exact")
    assert np.all(np.abs(got - ref) <= (N + 128) * 2.0 ** -53 * lim
                  + np.exp(-40.0) * VS * np.sum(np.abs(a)))
