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


@pytest.mark.parametrize("B,T,H,chunks", [(2, 64, 3, 1), (1, 500, 5, 8), (2, 640, 3, 10)])
def test_workspace_of_a_call_that_is_not_cut(pkg, workloads, cuda, B, T, H, chunks):
    """Nothing is carried from segment to segment where there is one: flags and operators are all the call asks for and needs; a
    byte less cuts it, with the same bits, or (one chunk) gives it to the tf32 kernel."""
    inp = workloads.wkv7_inputs(B, T, H, 64, seed=103, dtype=torch.bfloat16, device=cuda, state="normal")
    seq = pkg.Wkv7PretrainForwardInputs(*[inp[n] for n in "rwkvab"])
    need = pkg.lib().rwkv7_wkv7_workspace_bytes(B, T, H, 64, pkg.BF16)
    assert need == 256 + chunks * B * H * 33280
    full = pkg.wkv7_statepass(inp["s0"], seq, reference_contract=False)
    tail = 2 if T >= 512 else 0
    for given, launches in ((need, 2 + tail), (need - 1, 4 + tail if chunks > 1 else 2)):
        ws = torch.full((need + 4096,), 77, dtype=torch.uint8, device=cuda)
        before = pkg.kernel_launch_count()
        out = pkg.wkv7_statepass(inp["s0"], seq, reference_contract=False, workspace=ws[:given])
        torch.cuda.synchronize()
        assert pkg.kernel_launch_count() - before == launches and (ws[given:] == 77).all()
        if given == need or chunks > 1:
            assert torch.equal(out.output, full.output) and torch.equal(out.next_state, full.next_state)
    assert pkg.read_device_status(0) == 0


def test_workspace_of_very_many_short_chains(pkg, cuda):
    """1024 x 64 tokens x 40 heads: the tf32 kernel's ints, not 1.4 GB of operators; 24 000 chains still get theirs."""
    ask = lambda B, T, H: pkg.lib().rwkv7_wkv7_workspace_bytes(B, T, H, 64, pkg.BF16)  # noqa: E731
    assert ask(1024, 64, 40) == 1024 * 40 * 4
    assert ask(600, 64, 40) == 96000 + 600 * 40 * 33280
    assert ask(1024, 512, 40) > 1 << 30
