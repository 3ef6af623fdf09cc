"""The dense matvec's zero-block skipping (csrc/dense.cu) against the CPU oracle.

Bound per element: float-pair arithmetic keeps 2^-46 of every term and 2^-46 of
the running sum, so a sum of n terms is within (2 n + 128) 2^-46 of the sum of
their magnitudes in the worst case; FP64 arithmetic within (n + 128) 2^-53.
"""
import numpy as np
import pytest

import oracle
from dachshund_gb300 import SignalCovarParams, WFVectorW, synth

pytestmark = pytest.mark.gpu
VS, LP, LQ = synth.VAR_S, synth.L_PERP, synth.L_PARA


@pytest.mark.parametrize("arith", ["float_pair", "fp64"])
@pytest.mark.parametrize("n", [1, 65, 2000, 2100, 4200])
def test_blocks_vs_oracle(ctx, n, arith):
    rng = np.random.default_rng(n)
    rec = np.empty((n, 5))
    rec[:, :2] = rng.uniform(0, 12, (n, 2))  # a long box: most blocks are zero
    rec[:, 2] = rng.uniform(0, 12.5 * n / 144, n)
    rec[:, 3] = 1 / rng.uniform(0.05, 0.3, n)
    rec[:, 4] = rng.standard_normal(n)
    op = WFVectorW(ctx, rec, SignalCovarParams(VS, LP, LQ))
    op.set_dense(True)
    op.set_dense_arith(arith)
    a = rng.standard_normal(n)
    ref = oracle.A_product("w", rec, a, VS, LP, LQ)
    mag = oracle.A_product("w", rec, np.abs(a), VS, LP, LQ)
    eps = (2 * n + 128) * 2.0 ** -46 if arith == "float_pair" else (n + 128) * 2.0 ** -53
    assert np.all(np.abs(op.A_product(a) - ref) <= eps * mag)
    # a NaN multiplies the whole matrix, zero blocks included; the next finite
    # vector skips them again
    bad = a.copy()
    bad[n // 2] = np.nan
    assert np.all(np.isnan(op.A_product(bad)))
    assert np.all(np.abs(op.A_product(a) - ref) <= eps * mag)
    op.close()
