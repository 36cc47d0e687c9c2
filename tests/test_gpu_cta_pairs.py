"""GPU parity of the products that pairs of CTAs take (256 rows to a tile), at the edges of their tiles.  Each test asks the product's own plan
whether its shapes are on pairs."""
import numpy as np
import pytest
import torch

import parity
import plans

pytestmark = pytest.mark.gpu


def sms(cuda):
    return torch.cuda.get_device_properties(cuda).multi_processor_count


@pytest.mark.parametrize("shape,on_pairs", [
    ((1, 129, 520, 2056), (True, False)), ((1, 129, 2048, 264), (False, True)),     # one row more than a block: pieces of a long K beat a pair's padding
    ((1, 257, 264, 1032), (True, True)), ((3, 500, 520, 2056), (True, True)), ((1, 2049, 264, 1032), (True, True)), ((5, 600, 768, 3072), (True, True))])
def test_channel_mixer_on_pairs(pkg, workloads, cuda, shape, on_pairs):
    """Tiles of 64 to 256 columns, a last pair whose second CTA has one row or none, K with a partial last slice, N with a partial
    tile; against a restatement that rounds where the kernels round, within the bound of the other channel-mixer tests: the fp32
    sums differ in order alone, which can move the rounding of hidden by one bf16 spacing."""
    B, T, C, F = shape
    assert tuple(p["pair_width"] > 0 for p in plans.channel_mixer(B * T, C, F, sms(cuda))) == on_pairs
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


def check_lm_head(pkg, oracle, workloads, cuda, R, C, V, spread, shards=1):
    x, w, tg = workloads.lm_head_inputs(R, C, V, seed=R)
    x = x * spread
    tg[::5] = -1
    tg[1] = V - 1
    lse_ref, loss_ref = oracle.lm_head_ce(x.float().numpy(), w.float().numpy(), tg.numpy())
    xg, wg, tgg = x.to(cuda), w.to(cuda), tg.to(cuda)
    if shards == 1:
        lse, loss = pkg.lm_head_ce(xg, wg, tgg)
    else:
        cuts = np.linspace(0, V, shards + 1).astype(int)
        parts = [pkg.lm_head_ce_partial(xg, wg[lo:hi].contiguous(), tgg, int(lo)) for lo, hi in zip(cuts[:-1], cuts[1:])]
        lse, loss = pkg.lm_head_ce_finalize(torch.stack(parts), tgg)
    torch.cuda.synchronize()
    assert pkg.read_device_status(0) == 0
    np.testing.assert_allclose(lse.cpu().numpy(), lse_ref, rtol=0, atol=2e-4)
    np.testing.assert_allclose(loss.cpu().numpy(), loss_ref, rtol=0, atol=2e-4)


@pytest.mark.parametrize("R,C,V", [(129, 2048, 777), (255, 2048, 9000), (257, 4096, 777), (385, 2048, 9000), (500, 2048, 2064), (769, 2048, 777),
                                   (3000, 2048, 2064)])
def test_lm_head_on_pairs(pkg, oracle, workloads, cuda, R, C, V):
    """A last pair whose second CTA has one row or none, several row blocks, several tiles a split, vocabularies that are no multiple of 16 or
    32.  The products are exact in fp32; C / 16 sums of up to 6 at 2^-23 each are 1.8e-4 at the worst, the tolerance of the other LM-head tests."""
    assert plans.lm_head(R, C, V, sms(cuda))["pairs"]
    check_lm_head(pkg, oracle, workloads, cuda, R, C, V, 1)


def test_lm_head_on_pairs_over_vocabulary_shards(pkg, oracle, workloads, cuda):
    """Shards of 4097 and 4098 columns whose targets start at an offset."""
    R, C, V = 385, 2048, 3 * 4097 + 1
    assert all(plans.lm_head(R, C, n, sms(cuda))["pairs"] for n in (4097, 4098))
    check_lm_head(pkg, oracle, workloads, cuda, R, C, V, 1, shards=3)


@pytest.mark.parametrize("R,C,V", [(129, 64, 30000), (255, 128, 777), (257, 64, 9000), (1030, 192, 8200), (3000, 64, 2064)])
def test_lm_head_beside_pairs(pkg, oracle, workloads, cuda, R, C, V):
    """Ragged rows and vocabularies whose sums are too short for pairs; tolerance as in the other LM-head tests (exact bf16 products, fp32 sums)."""
    assert not plans.lm_head(R, C, V, sms(cuda))["pairs"]
    check_lm_head(pkg, oracle, workloads, cuda, R, C, V, 4)
