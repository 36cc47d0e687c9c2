"""GPU parity of the products that pairs of CTAs take (256 rows to a tile), at the edges of their tiles."""
import numpy as np
import pytest
import torch

import parity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 129, 520, 2056), (1, 257, 264, 1032), (3, 500, 520, 2056), (1, 2049, 264, 1032), (5, 600, 768, 3072)])
def test_channel_mixer_on_pairs(pkg, workloads, cuda, shape):
    """Tiles of 64 to 256 columns, a last pair whose second CTA has one row or none, K with a partial last slice, N with a partial
    tile; against a restatement that rounds where the kernels round, within the bound of the other channel-mixer tests: the fp32
    sums differ in order alone, which can move the rounding of hidden by one bf16 spacing."""
    B, T, C, F = shape
    x, ks, kw, vw = workloads.channel_mixer_inputs(B, T, C, F, seed=31)
    out = pkg.channel_mixer_custom(x.to(cuda), ks.to(cuda), kw.to(cuda), vw.to(cuda))
    torch.cuda.synchronize()
    assert pkg.read_device_status(0) == 0
    got = out.float().cpu().numpy().astype(np.float64)
    prev = torch.cat([torch.zeros(B, 1, C), x.float()[:, :-1]], 1)
    ki = (x.float() + (prev - x.float()) * ks.float()).to(torch.bfloat16).double().reshape(B * T, C)
    hid = (torch.relu(ki @ kw.double().T) ** 2).to(torch.bfloat16).double()
    fine = (hid @ vw.double().T).reshape(B, T, C).numpy()
    tol = 2e-3 * np.abs(fine).max() + 2 * parity.BF16_ULP * np.abs(fine)
    assert (np.abs(got - fine) <= tol).all(), float((np.abs(got - fine) - tol).max())


@pytest.mark.parametrize("R,C,V", [(129, 64, 30000), (255, 128, 777), (257, 64, 9000), (1030, 192, 8200), (3000, 64, 2064)])
def test_lm_head_on_pairs(pkg, oracle, workloads, cuda, R, C, V):
    """Ragged rows and vocabularies; tolerance as in the other LM-head tests (exact bf16 products, fp32 sums)."""
    x, w, tg = workloads.lm_head_inputs(R, C, V, seed=R)
    x = x * 4
    tg[::5] = -1
    tg[1] = V - 1
    lse_ref, loss_ref = oracle.lm_head_ce(x.float().numpy(), w.float().numpy(), tg.numpy())
    lse, loss = pkg.lm_head_ce(x.to(cuda), w.to(cuda), tg.to(cuda))
    torch.cuda.synchronize()
    assert pkg.read_device_status(0) == 0
    np.testing.assert_allclose(lse.cpu().numpy(), lse_ref, rtol=0, atol=2e-4)
    np.testing.assert_allclose(loss.cpu().numpy(), loss_ref, rtol=0, atol=2e-4)
