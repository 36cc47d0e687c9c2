"""GPU parity of the paths that only small batches take: the channel mixer's products cut along K (few rows), and the
LM head with more vocabulary splits than row blocks."""
import numpy as np
import pytest
import torch

import parity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 512, 1032), (2, 65, 1032, 2056), (1, 128, 520, 4096), (3, 1, 2048, 8192)])
def test_channel_mixer_split_along_k(pkg, workloads, cuda, shape):
    """Rows on both sides of one 128-row tile, K with a partial last step and a partial last piece, N with partial tiles;
    against a restatement that rounds where the kernels round."""
    B, T, C, F = shape
    x, ks, kw, vw = workloads.channel_mixer_inputs(B, T, C, F, seed=17)
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


@pytest.mark.parametrize("R,C,V", [(1, 64, 20000), (127, 128, 40000), (129, 64, 9000)])
def test_lm_head_with_many_splits(pkg, oracle, workloads, cuda, R, C, V):
    x, w, tg = workloads.lm_head_inputs(R, C, V, seed=19)
    lse_ref, loss_ref = oracle.lm_head_ce(x.float().numpy(), w.float().numpy(), tg.numpy())
    lse, loss = pkg.lm_head_ce(x.to(cuda), w.to(cuda), tg.to(cuda))
    torch.cuda.synchronize()
    assert pkg.read_device_status(0) == 0
    np.testing.assert_allclose(lse.cpu().numpy(), lse_ref, rtol=0, atol=2e-4)
    np.testing.assert_allclose(loss.cpu().numpy(), loss_ref, rtol=0, atol=2e-4)


@pytest.mark.parametrize("rows,room", [(1, "least"), (128, "least"), (128, 200), (128, 129)])
def test_channel_mixer_takes_a_workspace_for_another_batch(pkg, workloads, cuda, rows, room):
    """Room for key_input and hidden alone (no partial sums), or what a larger batch asks for (whose products are cut
    into fewer pieces of K): the same call with fewer pieces, within a rounding of the hidden tensor and one of the output."""
    C, F = 2048, 8192
    x, ks, kw, vw = (t.to(cuda) for t in workloads.channel_mixer_inputs(1, rows, C, F, seed=23))
    L = pkg.lib()
    least = sum((rows * n * 2 + 255) // 256 * 256 for n in (C, F))
    nbytes = least if room == "least" else L.rwkv7_channel_mixer_workspace_bytes(1, room, C, F)
    assert least <= nbytes < L.rwkv7_channel_mixer_workspace_bytes(1, rows, C, F)
    ws = torch.empty(nbytes + 4096, dtype=torch.uint8, device=cuda)
    ws[nbytes:] = 77
    got = pkg.channel_mixer_custom(x, ks, kw, vw, workspace=ws[:nbytes])
    want = pkg.channel_mixer_custom(x, ks, kw, vw)
    torch.cuda.synchronize()
    assert pkg.read_device_status(0) == 0 and (ws[nbytes:] == 77).all()
    got, want = got.float(), want.float()
    assert ((got - want).abs() <= 2e-3 * want.abs().max() + 2 * parity.BF16_ULP * want.abs()).all()
    with pytest.raises(pkg.KernelInputsError):
        pkg.channel_mixer_custom(x, ks, kw, vw, workspace=ws[:least - 256])


@pytest.mark.parametrize("rows,room", [(1, None), (128, None), (128, 129), (128, 200)])
def test_lm_head_takes_a_workspace_for_another_batch(pkg, workloads, cuda, rows, room):
    """16 triples per row, or what a larger batch asks for: fewer vocabulary splits, the same sums to fp32 rounding."""
    import ctypes
    C, V = 128, 65536
    x, w, tg = (t.to(cuda) for t in workloads.lm_head_inputs(rows, C, V, seed=29))
    L = pkg.lib()
    nbytes = 16 * rows * 12 if room is None else L.rwkv7_lm_head_ce_workspace_bytes(room, C, V)
    assert nbytes < L.rwkv7_lm_head_ce_workspace_bytes(rows, C, V)
    want = pkg.lm_head_ce_partial(x, w, tg)
    got = torch.empty_like(want)
    ws = torch.full((nbytes + 4096,), 77, dtype=torch.uint8, device=cuda)
    d = [pkg.describe(t) for t in (x, w, tg, got)]
    call = lambda n: L.rwkv7_fused_lm_head_ce_partial(  # noqa: E731
        *[ctypes.byref(t) for t in d[:3]], ctypes.c_int64(0), ctypes.byref(d[3]), ctypes.c_void_p(ws.data_ptr()), ctypes.c_size_t(n),
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert call(nbytes) == 0
    torch.cuda.synchronize()
    assert pkg.read_device_status(0) == 0 and (ws[nbytes:] == 77).all()
    torch.testing.assert_close(got, want, rtol=1e-5, atol=0)     # 256 sums of 256 terms in fp32
    assert L.rwkv7_status_string(call(16 * rows * 12 - 4)) == b"WorkspaceTooSmall"
