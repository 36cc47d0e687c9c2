"""GPU parity of WKV7 calls on caller-given workspaces that are not as the library would ask for them."""
import pytest
import torch

import parity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,dtype", [(64, torch.bfloat16), (500, torch.bfloat16), (576, torch.bfloat16), (576, torch.float32)])
@pytest.mark.parametrize("offset", [4, 8, 16])
def test_workspace_off_the_bulk_copies_boundary(pkg, oracle, workloads, cuda, T, dtype, offset):
    """The two-kernel prefill copies its operators in bulk, from 16-byte boundaries: a workspace that starts elsewhere goes to the
    kernel that keeps only ints (bf16) or nothing (fp32) there."""
    inp = workloads.wkv7_inputs(2, T, 2, 64, seed=101, dtype=dtype, state="normal")
    f = {n: t.float().numpy() for n, t in inp.items()}
    y_ref, s_ref = oracle.wkv7(*[f[n] for n in "rwkvab"], f["s0"])
    d = {n: t.to(cuda) for n, t in inp.items()}
    seq = pkg.Wkv7PretrainForwardInputs(*[d[n] for n in "rwkvab"])
    room = torch.empty(64 + (8 << 20), dtype=torch.uint8, device=cuda)
    assert room.data_ptr() % 256 == 0
    before = pkg.kernel_launch_count()
    out = pkg.wkv7_statepass(d["s0"], seq, reference_contract=False, workspace=room[offset:])
    torch.cuda.synchronize()
    launches = pkg.kernel_launch_count() - before
    assert pkg.read_device_status(0) == 0
    if offset == 16:
        assert launches == (2 if T < 512 else 4 if dtype == torch.bfloat16 else 3)
        y, s = out.output, out.next_state
        aligned = pkg.wkv7_statepass(d["s0"], seq, reference_contract=False)
        assert torch.equal(y, aligned.output) and torch.equal(s, aligned.next_state)
    else:
        assert launches == (2 if dtype == torch.bfloat16 else 1)   # tf32 chunked kernel and its flagged chains; sequential scan
        if dtype == torch.bfloat16:
            with pytest.raises(pkg.KernelInputsError):
                pkg.set_wkv7_path(pkg.WKV7_SPLIT)
                try:
                    pkg.wkv7_statepass(d["s0"], seq, reference_contract=False, workspace=room[offset:])
                finally:
                    pkg.set_wkv7_path(pkg.WKV7_AUTO)
    close = parity.assert_close_bf16_store if dtype == torch.bfloat16 else parity.assert_close_f32
    close(out.output.float().cpu().numpy(), y_ref, 1e-3, "y")
    parity.assert_close_f32(out.next_state.cpu().numpy(), s_ref, 1e-3, "state")
