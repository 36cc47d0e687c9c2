"""The sequential scan with one, two and four value rows per thread: whichever the number of chains selects, the bits are those of a
row per thread, which the other tests hold against the oracle."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B,T", [(3, 5), (4, 8), (5, 23), (7, 9), (13, 16), (13, 31)])
def test_rows_per_thread_agree_bitwise(pkg, workloads, cuda, B, T, dtype):
    H = 32
    inp = {n: t.to(cuda) for n, t in workloads.wkv7_inputs(B, T, H, 64, seed=67, dtype=dtype, state="normal").items()}

    def run(rows):
        six = pkg.Wkv7PretrainForwardInputs(*[inp[n][rows].contiguous() for n in "rwkvab"])
        out = pkg.wkv7_statepass(inp["s0"][rows].contiguous(), six, reference_contract=False)
        return out.output, out.next_state

    pkg.set_wkv7_path(pkg.WKV7_SEQUENTIAL)
    try:
        y, s = run(slice(0, B))
        parts = [run(slice(b, b + 1)) for b in range(B)]      # 32 chains: a row per thread
        torch.cuda.synchronize()
    finally:
        pkg.set_wkv7_path(pkg.WKV7_AUTO)
    assert torch.equal(y, torch.cat([p[0] for p in parts])) and torch.equal(s, torch.cat([p[1] for p in parts]))
