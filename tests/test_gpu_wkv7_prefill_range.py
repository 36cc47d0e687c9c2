"""GPU parity of the prefill that bf16 sequences take by themselves: block-wise reference points (a model's whole decay range)
at the edges of a chunk and of the tiers, and chains beyond them recomputed by the scan."""
import numpy as np
import pytest
import torch

import parity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,decay", [(64, "model"), (65, "edge"), (127, "model"), (333, "edge"), (511, "beyond"), (512, "edge"),
                                     (577, "mixed"), (2047, "model"), (6000, "model")])
def test_prefill_decay_range(pkg, oracle, workloads, cuda, T, decay):
    inp = workloads.wkv7_inputs(2, T, 3, 64, seed=61, dtype=torch.bfloat16, state="normal")
    g = torch.Generator().manual_seed(17)
    if decay == "model":        # -softplus - 0.5 over the speeds a model starts with
        speed = torch.linspace(-6.0, 3.0, 64) + 0.3 * torch.randn(inp["w"].shape, generator=g)
        inp["w"] = (-torch.nn.functional.softplus(-speed) - 0.5).to(torch.bfloat16)
    elif decay == "edge":       # the strongest decay a model has, in every channel
        inp["w"] = torch.full_like(inp["w"], -0.5)
    elif decay == "mixed":      # channels from hardly any decay to the edge, changing from token to token
        inp["w"] = (-0.5 - 6.0 * torch.rand(inp["w"].shape, generator=g)).to(torch.bfloat16)
    else:                       # one chain beyond what the reference points resolve
        inp["w"][0, :, 1] = 0.25
    f = {n: t.float().numpy() for n, t in inp.items()}
    y_ref, s_ref = oracle.wkv7_train(*[f[n] for n in "rwkvab"], s0=f["s0"], chunk_len=1)[:2]
    d = {n: t.to(cuda) for n, t in inp.items()}
    launches = pkg.kernel_launch_count()
    out = pkg.wkv7_statepass(d["s0"], pkg.Wkv7PretrainForwardInputs(*[d[n] for n in "rwkvab"]), reference_contract=False)
    torch.cuda.synchronize()
    assert pkg.kernel_launch_count() - launches == (2 if T < 512 else 4)
    assert pkg.read_device_status(0) == 0
    parity.assert_close_bf16_store(out.output.float().cpu().numpy(), y_ref, 1e-3, "y")
    parity.assert_close_f32(out.next_state.cpu().numpy(), s_ref, 1e-3, "next_state")


@pytest.mark.parametrize("T", [512, 1000])
def test_fp32_chains_of_a_models_decays_stay_fp32(pkg, oracle, workloads, cuda, T):
    """Chains whose log-decay passes 18 in 64 tokens are computed by the sequential scan when the tensors are fp32: 2e-5 of the
    largest value, as that kernel is held to, where fp16 operands give 5e-4.  One chain in range stays on the tensor cores."""
    inp = workloads.wkv7_inputs(2, T, 3, 64, seed=67, dtype=torch.float32, state="normal")
    g = torch.Generator().manual_seed(17)
    speed = torch.linspace(-6.0, 3.0, 64) + 0.3 * torch.randn(inp["w"].shape, generator=g)
    mild = inp["w"][0, :, 0].clone()
    inp["w"] = -torch.nn.functional.softplus(-speed) - 0.5
    inp["w"][0, :, 0] = mild
    f = {n: t.numpy() for n, t in inp.items()}
    y_ref, s_ref = oracle.wkv7(*[f[n] for n in "rwkvab"], f["s0"])
    d = {n: t.to(cuda) for n, t in inp.items()}
    out = pkg.wkv7_statepass(d["s0"], pkg.Wkv7PretrainForwardInputs(*[d[n] for n in "rwkvab"]), reference_contract=False)
    torch.cuda.synchronize()
    assert pkg.read_device_status(0) == 0
    y, s = out.output.cpu().numpy(), out.next_state.cpu().numpy()
    for b in range(2):
        for h in range(3):
            tol = 1e-3 if b == h == 0 else 2e-5
            parity.assert_close_f32(y[b, :, h], y_ref[b, :, h], tol, f"y, chain {b},{h}")
            parity.assert_close_f32(s[b, h], s_ref[b, h], tol, f"state, chain {b},{h}")


@pytest.mark.parametrize("alias", [False, True])
def test_recomputation_goes_on_from_the_first_marked_chunk(pkg, oracle, workloads, cuda, alias):
    """Chains under 512 tokens with a decay out of range in one chunk: the scan runs up to it and goes on token by token from the state
    there; where a value in front of it overflows fp16, from the beginning.  The state may be updated in place."""
    T, H = 500, 8
    inp = workloads.wkv7_inputs(1, T, H, 64, seed=71, dtype=torch.bfloat16, state="normal")
    for h, t in ((0, 0), (1, 63), (2, 64), (3, 200), (4, 499), (5, 320)):
        inp["w"][0, t, h] = 2.8
    inp["r"][0, 100, 5] *= 1e5      # (marked and overflowing)
    inp["r"][0, 400, 3] *= 1e5      # (only behind the mark: token by token by then)
    inp["r"][0, 10, 6] *= 1e5
    f = {n: t.float().numpy() for n, t in inp.items()}
    y_ref, s_ref = oracle.wkv7(*[f[n] for n in "rwkvab"], f["s0"])
    d = {n: t.to(cuda) for n, t in inp.items()}
    out = pkg.wkv7_statepass(d["s0"], pkg.Wkv7PretrainForwardInputs(*[d[n] for n in "rwkvab"]), reference_contract=False,
                             next_state=d["s0"] if alias else None)
    torch.cuda.synchronize()
    assert pkg.read_device_status(0) == 0
    y, s = out.output.float().cpu().numpy(), out.next_state.cpu().numpy()
    for h in range(H):
        parity.assert_close_bf16_store(y[:, :, h], y_ref[:, :, h], 1e-3, f"y, head {h}")
        parity.assert_close_f32(s[:, h], s_ref[:, h], 1e-3, f"state, head {h}")
