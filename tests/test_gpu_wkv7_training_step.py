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


def _step(pkg, leaves, dy, ds):
    leaves = [t.detach().requires_grad_(True) for t in leaves]
    y, s = pkg.wkv7_statepass_autograd(leaves[6], pkg.Wkv7PretrainForwardInputs(*leaves[:6]))
    return [y.detach(), s.detach(), *torch.autograd.grad((y, s), leaves, (dy, ds))]


@pytest.mark.parametrize("B,T,H", [(2, 1040, 20), (3, 80, 60)])     # 680 chunks of 40 chains, the last one short; 180 chains
def test_training_step_of_many_chunks(pkg, oracle, workloads, cuda, B, T, H):
    """More chunks than a CTA takes at a time, in every kernel, and more chains than SMs: each CTA of the chunk kernel goes through
    several chunks in both buffers, some of them token by token (a decay out of range, receptances beyond fp16) with ordinary ones
    behind.  Every chain has the bits it has in a call of its own, where a CTA has one chunk; chains of each kind against the oracle."""
    inp = workloads.wkv7_inputs(B, T, H, 64, seed=59, dtype=torch.bfloat16, state="normal")
    inp["w"][0, :, 1] = 0.5                              # every chunk of a chain out of range
    inp["w"][1, -16:, 3] = 0.5                           # the last chunk
    inp["w"][0, :64, H - 1] = 0.5                        # the first
    inp["w"][1, 64, 4] = 2.8                             # the second
    inp["r"][0, 16:32, 2] *= 1e5                         # a chunk whose receptances overflow
    inp["r"][1, -20:, 5] *= 1e5
    gen = torch.Generator().manual_seed(29)
    dy = torch.randn(B, T, H, 64, generator=gen).to(torch.bfloat16)
    ds = torch.randn(B, H, 64, 64, generator=gen)
    names = ["r", "w", "k", "v", "a", "b", "s0"]
    full = [inp[n].to(cuda) for n in names]
    got = _step(pkg, full, dy.to(cuda), ds.to(cuda))
    torch.cuda.synchronize()
    assert pkg.read_device_status(0) == 0
    what = ["y", "state", *("d" + n for n in names)]

    def chain(t, b, h):      # of a sequence tensor or a state, as a call of its own
        return t[b:b + 1, :, h:h + 1].contiguous() if t.dtype == torch.bfloat16 else t[b:b + 1, h:h + 1].contiguous()

    for b in range(B):
        for h in range(H):
            own = _step(pkg, [chain(t, b, h) for t in full], chain(dy, b, h).to(cuda), chain(ds, b, h).to(cuda))
            for n, whole, alone in zip(what, got, own):
                assert torch.equal(chain(whole, b, h), alone), (n, b, h)
    assert pkg.read_device_status(0) == 0
    for b, h in [(0, 0), (0, 1), (1, 3), (0, H - 1), (0, 2), (1, 5), (1, 4), (1, H - 1)]:
        f = {n: chain(inp[n], b, h).float().numpy() for n in names}
        y_ref, s_ref = oracle.wkv7_train(*[f[n] for n in "rwkvab"], s0=f["s0"], chunk_len=16)[:2]
        ref = oracle.wkv7_backward(*[f[n] for n in "rwkvab"], chain(dy, b, h).float().numpy(), s0=f["s0"], ds_out=chain(ds, b, h).numpy())
        parity.assert_close_bf16_store(chain(got[0], b, h).float().cpu().numpy(), y_ref, 1e-3, f"y of chain {b},{h}")
        parity.assert_close_f32(chain(got[1], b, h).cpu().numpy(), s_ref, 1e-3, f"state of chain {b},{h}")
        for n, g in zip(names, got[2:]):
            d = np.abs(chain(g, b, h).float().cpu().numpy().astype(np.float64) - ref[n]).max() / np.abs(ref[n]).max()
            assert d <= (1e-3 if n == "s0" else 5e-3), f"d{n} of chain {b},{h}: {d:.3e}"
