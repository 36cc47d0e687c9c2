"""GPU parity of the differentiable statepass on bf16 sequences with 64-element heads (the tensor-core training step):
forward scan with saved states, scan of the state's gradient over the transposed operators, per-chunk gradients."""
import numpy as np
import pytest
import torch

import parity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,state,decay,scale", [
    ((1, 64, 1, 64), True, "model", 1.0),       # one full chunk
    ((1, 80, 2, 64), False, "model", 1.0),      # one block in the last chunk
    ((2, 112, 3, 64), True, "edge", 1.0),       # three; the strongest decay a model has
    ((1, 1040, 1, 64), True, "model", 1e-7),    # gradients far below what fp16 resolves
    ((1, 192, 2, 64), True, "model", 1e5),      # and beyond what it holds
    ((2, 128, 2, 64), True, "beyond", 1.0),     # one batch row outside the reference points' range: token by token
])
def test_training_step_against_oracle(pkg, oracle, workloads, cuda, shape, state, decay, scale):
    B, T, H, N = shape
    inp = workloads.wkv7_inputs(*shape, seed=53, dtype=torch.bfloat16, state="normal" if state else None)
    if decay == "edge":
        inp["w"] = torch.full_like(inp["w"], -0.5)
    elif decay == "beyond":
        inp["w"][0] = 0.5
    gen = torch.Generator().manual_seed(13)
    dy = (scale * torch.randn(B, T, H, N, generator=gen)).to(torch.bfloat16)
    ds = scale * torch.randn(B, H, N, N, generator=gen) if state else None
    f = {n: inp[n].float().numpy() for n in inp}
    y_ref, s_ref = oracle.wkv7_train(*[f[n] for n in "rwkvab"], s0=f.get("s0"), chunk_len=16)[:2]
    ref = oracle.wkv7_backward(*[f[n] for n in "rwkvab"], dy.float().numpy(), s0=f.get("s0"),
                               ds_out=None if ds is None else ds.numpy())
    leaves = {n: t.to(cuda).requires_grad_(True) for n, t in inp.items()}
    y, s = pkg.wkv7_statepass_autograd(leaves.get("s0"), pkg.Wkv7PretrainForwardInputs(*[leaves[n] for n in "rwkvab"]))
    wrt = [leaves[n] for n in leaves]
    for _ in range(2):      # what the forward pass keeps is only read
        if state:
            grads = torch.autograd.grad((y, s), wrt, (dy.to(cuda), ds.to(cuda)), retain_graph=True)
        else:
            grads = torch.autograd.grad(y, wrt, dy.to(cuda), retain_graph=True)
    torch.cuda.synchronize()
    assert pkg.read_device_status(0) == 0
    parity.assert_close_bf16_store(y.detach().float().cpu().numpy(), y_ref, 1e-3, "y")
    parity.assert_close_f32(s.detach().cpu().numpy(), s_ref, 1e-3, "next_state")
    for n, got in zip(leaves, grads):
        want = ref[n]
        d = np.abs(got.float().cpu().numpy().astype(np.float64) - want).max() / np.abs(want).max()
        assert d <= (1e-3 if n == "s0" else 5e-3), f"d{n}: {d:.3e}"
