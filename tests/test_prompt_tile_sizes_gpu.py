"""The prompt product with W as the 256-row operand, in every number of tokens that its tiles can have, and which form a plain call takes."""
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


TILES = [32, 64, 96, 128, 160, 192, 224, 256]
# A last tile with few tokens or one, with none for its second block or for the second four drain warps; rows of W that end inside a warp's
# 32 or a pair's first block; more tiles than pairs; K steps of W asked into the L2 (K a multiple of 128) and not
SHAPES = [(129, 4096, 200), (160, 264, 64), (289, 4096, 72), (300, 1288, 1280), (527, 2568, 72), (1300, 520, 264), (385, 6144, 512), (5, 8, 64),
          (97, 136, 4104)]


@pytest.mark.parametrize("tile", TILES)
@pytest.mark.parametrize("M,N,K", SHAPES)
def test_every_tile(M, N, K, tile):
    """W as the 256-row operand gives the bits of the tokens first."""
    from qwen3_b200.csrc import ops
    x, w = operands(M, N, K)
    out = torch.full((M + 1, N), float("nan"), dtype=torch.bfloat16, device="cuda")
    ops.gemm_tcgen05_pair(x, w, out[:M], tile=tile)
    check(out[:M], x, w)
    assert bool(out[M].isnan().all()), "written beyond the last token"
    wide = torch.full((M, N), float("nan"), dtype=torch.float32, device="cuda")     # tokens first: 32-bit output
    ops.gemm_tcgen05_pair(x, w, wide)
    assert torch.equal(wide.to(torch.bfloat16), out[:M])


@pytest.mark.parametrize("tile", TILES)
@pytest.mark.parametrize("M,inter,K", [(129, 2048, 136), (300, 1160, 1280), (527, 1000, 72), (385, 104, 200), (7, 8, 64)])
@pytest.mark.parametrize("activation", ["silu", "gelu_tanh"])
def test_every_tile_gated(M, inter, K, tile, activation):
    """The gate in the drain of that form gives the bits of the product followed by the gating kernel."""
    from qwen3_b200.csrc import ops
    x, gate = operands(M, inter, K)
    up = operands(M + 1, inter, K)[1]
    w = ops.interleave_gate_up(gate * 0.2, up * 0.2)
    fused = torch.full((M + 1, inter), float("nan"), dtype=torch.bfloat16, device="cuda")
    ops.gemm_tcgen05_pair(x, w, fused[:M], gated=True, activation=activation, tile=tile)
    assert ops.tcgen05_status("cuda") == 0
    gate_up = torch.empty(M, 2 * inter, dtype=torch.bfloat16, device="cuda")
    ops.gemm_tcgen05_pair(x, w, gate_up, tile=256)
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


@pytest.mark.parametrize("M,N,K", [(300, 4096, 4096), (527, 24576, 1024), (1300, 4096, 2048), (200, 8, 64), (527, 4100, 1024), (4096, 4096, 512)])
def test_the_form_that_is_taken(M, N, K):
    """The product without a split of K is that of the tiles that `gemm_tcgen05_pair_tile` names: equal tokens for a few hundred of them,
    whole 256s where these leave nothing idle and where the rows of the output are no whole packets."""
    from qwen3_b200.csrc import ops
    tile = ops.gemm_tcgen05_pair_tile(M, N, K)
    assert tile in ([0] if N % 8 or N == 8 or M == 4096 else TILES)
    assert ops.gemm_tcgen05_pair_tile(M, N, K, may_row=False) == 0
    x, w = operands(M, N, K)
    out, same = (torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    ops.gemm_tcgen05_pair(x, w, out)
    check(out, x, w)
    if tile:
        ops.gemm_tcgen05_pair(x, w, same, tile=tile)
        assert torch.equal(out, same)


@pytest.mark.parametrize("tile,N,dtype,splits", [(16, 256, torch.bfloat16, 1), (40, 256, torch.bfloat16, 1), (288, 256, torch.bfloat16, 1),
                                                 (64, 252, torch.bfloat16, 1), (64, 256, torch.float32, 1), (64, 256, torch.bfloat16, 2)])
def test_tiles_that_are_refused(tile, N, dtype, splits):
    from qwen3_b200.csrc import ops
    x, w = operands(100, N, 64)
    with pytest.raises(ops.KernelError):
        ops.gemm_tcgen05_pair(x, w, torch.empty(100, N, dtype=dtype, device="cuda"), tile=tile, splits=splits)
