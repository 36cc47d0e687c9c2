"""GPU parity of mix6 where its window of rows meets its limits: fewer rows than the window, one row more, many times round it, sequences
shorter than a step of it, and rows that are longer than the grid two CTAs an SM make.  Tolerances as in the other mixing tests: the
arithmetic is fp32 with one rounding."""
import numpy as np
import pytest
import torch

import parity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape", [(1, 1, 8), (1, 2369, 2048), (5, 977, 136), (3000, 3, 96), (2, 700, 1000), (1, 3, 620008)])
def test_mix6_window(pkg, workloads, cuda, shape, dtype):
    x, mus = workloads.mix_inputs(*shape, seed=5, dtype=dtype)
    out = pkg.mix6_custom(x.to(cuda), *[m.to(cuda) for m in mus])
    torch.cuda.synchronize()
    xd = x.double()
    prev = torch.cat([torch.zeros_like(xd[:, :1]), xd[:, :-1]], 1)
    for name, m in zip(pkg.MIX6_BRANCHES, mus):
        ref = (xd + (prev - xd) * m.double()).numpy()
        got = out[name].float().cpu().numpy().astype(np.float64)
        # the difference and the sum are rounded to fp32 each, at operands of up to 6; bf16 rounds once more
        bound = 2e-6 + (parity.BF16_ULP * np.abs(ref) if dtype == torch.bfloat16 else 0.0)
        assert (np.abs(got - ref) <= bound).all()
