"""The prompt product's tiles: every tile of the output is computed once, whatever the order and the widths they come in."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def operands(M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M + 3 * N + K)
    x = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randn(N, K, generator=g, device="cuda").to(torch.bfloat16)
    return x, w


def check(out, x, w):
    """Against 64 bits; the bounds of a sum of K products in 32 bits, rounded to the output's type."""
    from qwen3_b200.csrc import ops
    K = x.shape[1]
    assert ops.tcgen05_status("cuda") == 0, "a wait inside the kernel gave up"
    want = x.double() @ w.double().T
    base, rel = (4e-5 * math.sqrt(K) * 4, 1e-6) if out.dtype == torch.float32 else (0.02 * math.sqrt(K), 2.0 ** -8)
    excess = ((out.double() - want).abs() - (base + rel * want.abs())).max().item()
    assert excess <= 0, f"an output is {excess:.3e} beyond its bound"


# one band of 16 tiles of tokens, one more token, two bands of unequal height, five bands with a lower last one
@pytest.mark.parametrize("M", [4096, 4097, 16 * 256 + 300, 66 * 256 - 1])
@pytest.mark.parametrize("N", [256, 257, 1300])
def test_bands_of_token_tiles(M, N):
    from qwen3_b200.csrc import ops
    x, w = operands(M, N, 72)
    out = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda")
    ops.gemm_tcgen05_pair(x, w, out)
    check(out, x, w)
