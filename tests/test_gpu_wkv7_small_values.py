"""GPU parity of the tensor-core WKV7 paths on values that lie below what fp16 resolves: receptances, keys, values and states are
brought up by powers of two on their way into the matrix instructions.  Tolerances are those of the other WKV7 tests, relative to
the largest value of the reference, so they are as tight at 1e-6 as at 1."""
import numpy as np
import pytest
import torch

import parity

pytestmark = pytest.mark.gpu

SCALES = [dict(v=1e-5, s0=1e-5), dict(v=1e-8, s0=1e-8), dict(r=1e-6), dict(k=1e-6), dict(k=1e-3, v=1e-3, s0=1e-6, r=1e-4), dict(s0=1e-7, v=1e-7, k=30.0)]


def _inputs(workloads, shape, scales, dtype, seed, model=False):
    inp = workloads.wkv7_inputs(*shape, seed=seed, dtype=torch.float32, state="normal")
    if model:
        g = torch.Generator().manual_seed(19)
        speed = torch.linspace(-6.0, 3.0, 64) + 0.3 * torch.randn(inp["w"].shape, generator=g)
        inp["w"] = -torch.nn.functional.softplus(-speed) - 0.5
    for n, x in scales.items():
        inp[n] = inp[n] * x
    return {n: t if n == "s0" else t.to(dtype) for n, t in inp.items()}


@pytest.mark.parametrize("scales", SCALES, ids=str)
@pytest.mark.parametrize("T,dtype,model", [(64, "bf16", False), (333, "bf16", True), (576, "bf16", False), (576, "f32", False)])
def test_prefill(pkg, oracle, workloads, cuda, T, dtype, model, scales):
    dt = torch.bfloat16 if dtype == "bf16" else torch.float32
    inp = _inputs(workloads, (2, T, 2, 64), scales, dt, 107, model)
    f = {n: t.float().numpy() for n, t in inp.items()}
    y_ref, s_ref = oracle.wkv7(*[f[n] for n in "rwkvab"], f["s0"])
    d = {n: t.to(cuda) for n, t in inp.items()}
    out = pkg.wkv7_statepass(d["s0"], pkg.Wkv7PretrainForwardInputs(*[d[n] for n in "rwkvab"]), reference_contract=False)
    torch.cuda.synchronize()
    assert pkg.read_device_status(0) == 0
    close = parity.assert_close_bf16_store if dtype == "bf16" else parity.assert_close_f32
    close(out.output.float().cpu().numpy(), y_ref, 1e-3, "y")
    parity.assert_close_f32(out.next_state.cpu().numpy(), s_ref, 1e-3, "state")


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_segments_scale_alike(pkg, workloads, cuda, dtype):
    """Magnitudes that change from chunk to chunk: a call cut into segments of one, two and three chunks looks back on the same
    chunks as one that is not cut, bit for bit."""
    B, T, H = 1, 64 * 9 - 5, 3
    inp = {n: t.to(cuda) for n, t in _inputs(workloads, (B, T, H, 64), {}, torch.float32, 109).items()}
    g = torch.Generator().manual_seed(3)
    size = 10.0 ** (-7.0 * torch.rand((B, 9, H), generator=g)).repeat_interleave(64, 1)[:, :T, :, None].to(cuda)
    size[:, 64:192, 0] = 0.0
    inp["v"] = inp["v"] * size
    inp["k"] = inp["k"] * size.flip(1).sqrt()
    inp["s0"] = inp["s0"] * 1e-6
    inp["s0"][:, 1] = 0.0
    inp = {n: t if n == "s0" else t.to(dtype) for n, t in inp.items()}
    seq = pkg.Wkv7PretrainForwardInputs(*[inp[n] for n in "rwkvab"])
    chains = B * H
    outs = []
    pkg.set_wkv7_path(pkg.WKV7_SPLIT)
    try:
        for chunks in (9, 1, 2, 3):
            ws = torch.empty(256 + 4096 + chains * 16384 + chunks * chains * 33280, dtype=torch.uint8, device=cuda)
            before = pkg.kernel_launch_count()
            outs.append(pkg.wkv7_statepass(inp["s0"], seq, reference_contract=False, workspace=ws))
            assert pkg.kernel_launch_count() - before == 2 * -(-9 // chunks) + (2 if dtype == torch.bfloat16 else 1)
    finally:
        pkg.set_wkv7_path(pkg.WKV7_AUTO)
    torch.cuda.synchronize()
    assert pkg.read_device_status(0) == 0
    for o in outs[1:]:
        assert torch.equal(o.output, outs[0].output) and torch.equal(o.next_state, outs[0].next_state)


@pytest.mark.parametrize("scales", SCALES + [dict(a=1e-5), dict(b=1e-5)], ids=str)
@pytest.mark.parametrize("model", [False, True])
def test_training_step(pkg, oracle, workloads, cuda, scales, model):
    B, T, H = 1, 208, 2
    inp = _inputs(workloads, (B, T, H, 64), scales, torch.bfloat16, 113, model)
    gen = torch.Generator().manual_seed(13)
    dy = torch.randn(B, T, H, 64, generator=gen).to(torch.bfloat16)
    ds = torch.randn(B, H, 64, 64, generator=gen) * scales.get("r", 1.0)
    f = {n: inp[n].float().numpy() for n in inp}
    y_ref, s_ref = oracle.wkv7_train(*[f[n] for n in "rwkvab"], s0=f["s0"], chunk_len=16)[:2]
    ref = oracle.wkv7_backward(*[f[n] for n in "rwkvab"], dy.float().numpy(), s0=f["s0"], ds_out=ds.numpy())
    leaves = {n: t.to(cuda).requires_grad_(True) for n, t in inp.items()}
    y, s = pkg.wkv7_statepass_autograd(leaves["s0"], pkg.Wkv7PretrainForwardInputs(*[leaves[n] for n in "rwkvab"]))
    grads = torch.autograd.grad((y, s), list(leaves.values()), (dy.to(cuda), ds.to(cuda)))
    torch.cuda.synchronize()
    assert pkg.read_device_status(0) == 0
    parity.assert_close_bf16_store(y.detach().float().cpu().numpy(), y_ref, 1e-3, "y")
    parity.assert_close_f32(s.detach().cpu().numpy(), s_ref, 1e-3, "next_state")
    worst = {}
    for n, got in zip(leaves, grads):
        worst[n] = np.abs(got.float().cpu().numpy().astype(np.float64) - ref[n]).max() / np.abs(ref[n]).max()
    print(scales, {n: f"{e:.1e}" for n, e in worst.items()})
    assert all(e <= (1e-3 if n == "s0" else 5e-3) for n, e in worst.items()), worst
