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


# tiles of 32 to 256 tokens (equal, with a short last one, one token in it), rows of W that end inside a warp's 32, a pair's second
# block without rows, more tiles than pairs; outputs whose rows are no whole packets, which stay with whole 256s
@pytest.mark.parametrize("M,N,K", [(129, 4096, 200), (160, 264, 64), (289, 4096, 72), (300, 1288, 136), (527, 24576, 72), (385, 6144, 512),
                                   (1300, 4096, 264), (2500, 4096, 72), (527, 4100, 72), (200, 8, 64)])
def test_tiles_of_equal_tokens(M, N, K):
    from qwen3_b200.csrc import ops
    x, w = operands(M, N, K)
    out = torch.full((M + 1, N), float("nan"), dtype=torch.bfloat16, device="cuda")
    ops.gemm_tcgen05_pair(x, w, out[:M])
    check(out[:M], x, w)
    assert bool(out[M].isnan().all()), "written beyond the last token"
    wide = torch.full((M, N), float("nan"), dtype=torch.float32, device="cuda")     # tokens first: 32-bit output
    ops.gemm_tcgen05_pair(x, w, wide)
    assert torch.equal(wide.to(torch.bfloat16), out[:M])


@pytest.mark.parametrize("M,inter,K", [(129, 4096, 136), (300, 1160, 72), (527, 12288, 64), (385, 104, 200), (1300, 2048, 72)])
@pytest.mark.parametrize("activation", ["silu", "gelu_tanh"])
def test_tiles_of_equal_tokens_gated(M, inter, K, activation):
    """The gate in the drain of the rows form gives the bits of the product followed by the gating kernel."""
    from qwen3_b200.csrc import ops
    x, gate = operands(M, inter, K)
    up = operands(M + 1, inter, K)[1]
    w = ops.interleave_gate_up(gate * 0.2, up * 0.2)
    fused = torch.full((M + 1, inter), float("nan"), dtype=torch.bfloat16, device="cuda")
    ops.gemm_tcgen05_pair(x, w, fused[:M], gated=True, activation=activation)
    assert ops.tcgen05_status("cuda") == 0
    gate_up = torch.empty(M, 2 * inter, dtype=torch.bfloat16, device="cuda")
    ops.gemm_tcgen05_pair(x, w, gate_up)
    check(gate_up, x, w)
    blocks = gate_up.float().view(M, inter // 8, 2, 8)
    g, u = blocks[:, :, 0].reshape(M, inter), blocks[:, :, 1].reshape(M, inter)
    act = torch.nn.functional.silu(g) if activation == "silu" else torch.nn.functional.gelu(g, approximate="tanh")
    want = act.to(torch.bfloat16).float() * u
    # the activation's last bit may round to the other neighbour: one rounding of it and one of the product
    assert bool(((fused[:M].float() - want).abs() <= 2.0 ** -7 * want.abs() + 1e-30).all())
    assert bool(fused[M].isnan().all()), "written beyond the last token"
    if activation == "silu":
        two = torch.empty(M, inter, dtype=torch.bfloat16, device="cuda")
        ops.silu_mul(gate_up, two, interleaved=True)
        assert torch.equal(fused[:M], two)


@pytest.mark.parametrize("M", [1, 3, 4, 8])
@pytest.mark.parametrize("N,K", [(7168, 4096), (9472, 4104), (24576, 4096), (7104, 4096)])
def test_large_matrices_of_few_rows(M, N, K):
    """Up to eight rows: the weights-first kernel for the largest matrices from four rows on and for little more than a wave of the other kernel's blocks,
    the other kernel beside (7,104 rows of W are one wave)."""
    from qwen3_b200.parts import linear as L
    assert L.few_rows_weights_first(M, N, K) == (N != 7104 and (N != 24576 or M >= 4))
    x, w = operands(M, N, K)
    for dtype in (torch.bfloat16, torch.float32):
        out = torch.full((M + 1, N), float("nan"), dtype=dtype, device="cuda")
        L.linear(x, w, out[:M])
        check(out[:M], x, w)
        assert bool(out[M].isnan().all())
