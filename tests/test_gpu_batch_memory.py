"""A small batch takes device memory of its size."""
import pytest

from dachshund_gb300 import BatchSolver, SignalCovarParams, pixel_to_wpixel, synth

pytestmark = pytest.mark.gpu


def test_small_batches(ctx):
    """Twenty batches of one tile with 32 right-hand sides: vectors of 128 x 32 numbers,
    88 bytes each, and at most 8 segments of 128 x 32 x 3 floats, 0.8 MB in all a batch;
    the library's pool grows by 32 MB at a time."""
    import torch

    exact = SignalCovarParams(synth.VAR_S, synth.L_PERP, synth.L_PARA, eval="exact")
    rec = pixel_to_wpixel(synth.small(3, 30, 6.0, seed=1).pixels)
    ctx.synchronize()
    free0, _ = torch.cuda.mem_get_info()
    batches = [BatchSolver(ctx, "w", [rec], exact, 32) for _ in range(20)]
    ctx.synchronize()
    free1, _ = torch.cuda.mem_get_info()
    for b in batches:
        b.close()
    assert free0 - free1 <= 20 * (1 << 20) + (128 << 20)
