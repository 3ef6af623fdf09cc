"""The dense operator where the device has room for it only without the operator's
stored pair values."""
import numpy as np
import pytest

from dachshund_gb300 import SignalCovarParams, WFVectorW, synth

pytestmark = pytest.mark.gpu


def test_stored_values_make_room(ctx):
    import torch

    n = 20000
    rng = np.random.default_rng(n)
    rec = np.empty((n, 5))
    rec[:, :3] = rng.uniform(0, (12.5 * n) ** (1 / 3), (n, 3))
    rec[:, 3] = 1 / rng.uniform(0.05, 0.3, n)
    rec[:, 4] = rng.standard_normal(n)
    a = rng.standard_normal(n)
    op = WFVectorW(ctx, rec, SignalCovarParams(synth.VAR_S, synth.L_PERP, synth.L_PARA,
                                               eval="exact"))
    b = op.A_product(a)
    assert op.stored_bytes() > (300 << 20)
    n_pad = -(-n // 128) * 128
    room = 8 * n_pad ** 2 - (250 << 20)  # less than the matrix takes
    free, _ = torch.cuda.mem_get_info()
    rest = torch.empty(free - room, dtype=torch.uint8, device="cuda")  # never touched
    try:
        op.set_dense(True)
        dense = op.A_product(a)
        op.set_dense(False)
        again = op.A_product(a)
    finally:
        del rest
        torch.cuda.empty_cache()
    # |A| |a| <= 2e4 here; float pairs hold 2^-46 of it, FP64 sums far less
    assert np.abs(dense - b).max() <= 2e4 * 2.0 ** -45
    assert np.abs(again - b).max() <= 2e4 * 2.0 ** -45
    op.close()
