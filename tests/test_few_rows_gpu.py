"""Products of up to eight rows on the kernel that has W as the 128-row operand: how K is split, and what a row's value depends on."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def operands(M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M + 5 * N + K)
    x = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    return x, torch.randn(N, K, generator=g, device="cuda").to(torch.bfloat16)


def check(out, x, w):
    """Against 64 bits: the bound of a sum of K products in 32 bits, rounded to bfloat16."""
    from qwen3_b200.csrc import ops
    assert ops.tcgen05_status("cuda") == 0, "a wait inside the kernel gave up"
    want = x.double() @ w.double().T
    excess = ((out.double() - want).abs() - (0.02 * math.sqrt(x.shape[1]) + 2.0 ** -8 * want.abs())).max().item()
    assert excess <= 0, f"an output is {excess:.3e} beyond its bound"


# (rows of W, K, K ranges on 148 SMs): clusters of four and of eight that just run at once and that do not, and shapes far from there
@pytest.mark.parametrize("N,K,splits", [(7168, 4096, 4), (8960, 4104, 4), (9088, 4096, 4), (9216, 4096, 3), (9344, 8192, 3), (9472, 4096, 3),
                                        (4224, 8192, 8), (4352, 8200, 6), (4736, 8192, 6), (12288, 8192, 4), (24576, 4096, 2)])
def test_all_ranges_run_at_once(N, K, splits):
    from qwen3_b200.csrc import ops
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert [ops.gemm_tcgen05_mid_splits(M, N, K) for M in (1, 8)] == [splits] * 2
    rows = []
    x, w = operands(8, N, K)
    for M in (1, 4, 8):
        out = torch.full((M + 1, N), float("nan"), dtype=torch.bfloat16, device="cuda")
        ops.gemm_tcgen05_mid(x[:M], w, out[:M])
        check(out[:M], x[:M], w)
        assert bool(out[M].isnan().all()), "written beyond the last row"
        rows.append(out[0])
        gated = torch.full((M + 1, N // 2), float("nan"), dtype=torch.bfloat16, device="cuda")
        ops.gemm_tcgen05_mid_gated(x[:M], w, gated[:M])
        blocks = out[:M].float().view(M, N // 16, 2, 8)
        want = torch.nn.functional.silu(blocks[:, :, 0]).to(torch.bfloat16).float() * blocks[:, :, 1]
        # the activation's last bit may round to the other neighbour: one rounding of it and one of the product
        assert bool(((gated[:M].float() - want.reshape(M, -1)).abs() <= 2.0 ** -7 * want.reshape(M, -1).abs() + 1e-30).all())
        assert bool(gated[M].isnan().all())
    assert torch.equal(rows[0], rows[1]) and torch.equal(rows[0], rows[2])


def test_where_it_is_taken():
    """Up to one wave of its blocks, three an SM, and not beyond; a little more than one wave of the other kernel's, and not one."""
    from qwen3_b200.parts import linear as L
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    most = 3 * sms * 128
    for M in (4, 8):
        assert L.few_rows_weights_first(M, most, 4096) and L.few_rows_weights_first(M, most, 8192)
        assert not L.few_rows_weights_first(M, most + 8, 4096) and not L.few_rows_weights_first(M, most + 512, 8192)
    for M in (1, 8):
        assert L.few_rows_weights_first(M, 3 * sms * 16 + 8, 4096) and L.few_rows_weights_first(M, 4 * sms * 16, 4096)
        assert not L.few_rows_weights_first(M, 3 * sms * 16, 4096) and not L.few_rows_weights_first(M, 4 * sms * 16 + 8, 4096)
        assert not L.few_rows_weights_first(M, 3 * sms * 16 + 8, 4088)


@pytest.mark.parametrize("N,K", [(24576, 4096), (5120, 17408), (9472, 4096)])
def test_a_row_alone_and_among_others(N, K):
    """Two kernels take the largest matrices, one up to three rows and the other from four on: between them a row may change by a rounding, each
    as near to 64 bits as the other; on either side it does not hang on the rows beside it."""
    from qwen3_b200.parts import linear as L
    x, w = operands(8, N, K)
    rows, errors = {}, {}
    want = x[:1].double() @ w.double().T
    for M in (1, 2, 3, 4, 5, 8):
        out = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
        L.linear(x[:M], w, out)
        check(out, x[:M], w)
        rows[M], errors[M] = out[0], ((out[:1].double() - want).norm() / want.norm()).item()
    assert all(torch.equal(rows[M], rows[1]) for M in (2, 3)) and all(torch.equal(rows[M], rows[4]) for M in (5, 8))
    # rounding to bfloat16 alone is 2^-9 / sqrt(3) in norm: the order of a sum in 32 bits adds nothing that shows
    assert max(errors.values()) <= 2.0 ** -9 and abs(errors[1] - errors[4]) <= 0.02 * errors[1]
