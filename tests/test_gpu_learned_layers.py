"""The learned network's FP32 layers (csrc/learned_gemm.cu) and fused tensor-core
layers (csrc/learned_tc.cu) at the edges of their tiles, against the CPU oracle.

Bounds: the gradients of every parameter block within 2e-3 of their norm, as the
repository's gradient test asks of FP32 (a relu that switches within rounding
moves a block by far more than the sums' own 1e-6); the tensor-core forward within
2e-2 of the FP32 one (TF32 keeps 10 bits, four layers of 384 terms).
"""
import numpy as np
import pytest

from oracle import learned_ref as lr
from dachshund_gb300 import SignalCovarParams, synth
from dachshund_gb300.learned import LearnedPreconditioner, gpu_system

pytestmark = pytest.mark.gpu

VS, LP, LQ = synth.VAR_S, synth.L_PERP, synth.L_PARA
C_PERP, C_PARA = 1 / (2 * LP ** 2), 1 / (2 * LQ ** 2)
EXACT = SignalCovarParams(VS, LP, LQ, eval="exact")


def perturbed(ctx, H, seed):
    net = LearnedPreconditioner(ctx, EXACT, hidden=H, band=2, seed=seed)
    flat = net.get_params() + 0.05 * np.random.default_rng(seed).standard_normal(
        net.n_params).astype(np.float32)
    net.set_params(flat)
    return net, flat.astype(np.float64)


def padded_knn(rec, n_sk, n_per, c_perp, knn=lr.knn):
    """lr.knn with the missing neighbours of fewer than 9 skewers as the kernels
    take them: the skewer itself with weight 0."""
    nbr, g = knn(rec, n_sk, n_per, c_perp)
    k = min(n_sk - 1, lr.NB_K)
    own = np.repeat(np.arange(n_sk)[:, None], lr.NB_K, axis=1)
    own[:, :k] = nbr[:, :k]
    w = np.zeros((n_sk, lr.NB_K))
    w[:, :k] = g[:, :k]
    return own, w


# widths below, off and above one 128-column tile; fewer than 9 skewers (missing
# neighbours); rows off the 128-row tile; one-pixel skewers
@pytest.mark.parametrize("H,n_sk,n_per", [(32, 3, 1), (96, 5, 3), (128, 9, 131), (160, 12, 16),
                                          (288, 10, 13), (512, 4, 8)])
def test_gradients_vs_oracle(ctx, monkeypatch, H, n_sk, n_per):
    import torch

    monkeypatch.setattr(lr, "knn", padded_knn)
    rec = gpu_system(3, n_sk, n_per, box=2.5 * np.ceil(np.sqrt(n_sk)))
    rng = np.random.default_rng(5)
    ystar = 0.05 * rng.standard_normal(n_sk * n_per)
    probe = rng.standard_normal(n_sk * n_per).astype(np.float32)
    net, flat = perturbed(ctx, H, 7)
    net.train_step_dev(n_sk, n_per, rec, torch.tensor(ystar, device="cuda"),
                       torch.tensor(probe, device="cuda"), update=False)
    g = net.get_grads().astype(np.float64)
    _, ref, _ = lr.loss_and_grad(flat, rec.cpu().numpy(), ystar, probe, n_sk, n_per, H, 2, VS,
                                 C_PERP, C_PARA)
    off = 0
    for name, r, c in lr.layout(H, 2):
        a, b = g[off:off + r * c], ref[off:off + r * c]
        off += r * c
        assert np.linalg.norm(a - b) <= 2e-3 * np.linalg.norm(b) + 1e-30, name
    net.close()


# tiles that span skewers, that divide them, and skewers of several tiles
@pytest.mark.parametrize("n_sk,n_per", [(4, 96), (128, 1), (10, 128), (9, 384), (3, 896)])
def test_tensor_core_layers(ctx, n_sk, n_per):
    import torch

    rec = gpu_system(4, n_sk, n_per, box=2.5 * np.ceil(np.sqrt(n_sk)))
    net, _ = perturbed(ctx, 128, 11)
    net.set_inference(False)
    y, L = (t.clone() for t in net.forward_dev(n_sk, n_per, rec))
    net.set_inference(True)
    yt, Lt = net.forward_dev(n_sk, n_per, rec)
    for a, b in ((yt, y), (Lt, L)):
        assert float(torch.max(torch.abs(a - b))) <= 2e-2 * float(torch.max(torch.abs(b)))
    net.close()
