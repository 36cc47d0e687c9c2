"""GPU parity of the prefill that bf16 sequences take by themselves: block-wise reference points (a model's whole decay range)
at the edges of a chunk and of the tiers, and chains beyond them recomputed by the scan."""
import numpy as np
import pytest
import torch

import parity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,decay", [(64, "model"), (65, "edge"), (127, "model"), (333, "edge"), (511, "beyond"), (512, "edge"),
                                     (577, "mixed")])
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
