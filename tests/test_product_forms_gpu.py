"""Which form of the tcgen05 product takes a prompt's rows, where they are near each other: none of these may cost more than another by a margin."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


# short K, in 32 bits and in bfloat16, where an estimate that is a microsecond off takes the wrong one; four ranges of K and two; wide layers
@pytest.mark.parametrize("M,N,K,dtype,form,splits", [
    (300, 4096, 2048, torch.float32, "prompt128", 0), (513, 2048, 2048, torch.float32, "prompt128", 0), (256, 8192, 2048, torch.float32, "prompt128", 0),
    (600, 2048, 1024, torch.bfloat16, "prompt128", 0), (1024, 2048, 1024, torch.bfloat16, "prompt128", 0), (150, 1024, 1024, torch.bfloat16, "prompt128", 0),
    (256, 3072, 4096, torch.bfloat16, "weights_first", 0), (600, 3072, 4096, torch.bfloat16, "pair", 1), (217, 6144, 4096, torch.bfloat16, "pair", 2),
    (527, 4096, 12288, torch.bfloat16, "pair", 1), (200, 4096, 4096, torch.bfloat16, "weights_first", 0)])
def test_form(M, N, K, dtype, form, splits):
    from qwen3_b200.csrc import ops
    from qwen3_b200.parts import linear as L
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        may_row = dtype == torch.bfloat16
        assert L.tcgen05_form(M, N, K, may_row=may_row) == form
        assert form != "pair" or L.pair_plan(M, N, K, may_row)[1] == splits
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randn(N, K, generator=g, device="cuda").to(torch.bfloat16)
    out = torch.full((M, N), float("nan"), dtype=dtype, device="cuda")
    L.linear(x, w, out)
    assert ops.tcgen05_status("cuda") == 0
    want = x.double() @ w.double().T
    # the bounds of a sum of K products in 32 bits, rounded to the output's type
    base, rel = (4e-5 * math.sqrt(K) * 4, 1e-6) if dtype == torch.float32 else (0.02 * math.sqrt(K), 2.0 ** -8)
    assert ((out.double() - want).abs() - (base + rel * want.abs())).max().item() <= 0
