"""Attention of prompts with heads of 192 and 256 and values of their own size on tcgen05: against 64 bits and beside the mma.sync
kernel that takes the same calls."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def exact(q, k, v, scale, pos0, window, sink):
    """q [n, H, d], k [keys, G, d], v [keys, G, vd] of one sequence, the new tokens at pos0 ..: [n, H, vd] in 64 bits."""
    n, H, _ = q.shape
    G = k.shape[1]
    s = torch.einsum("ngid,kgd->ngik", q.double().view(n, G, H // G, -1), k.double()).reshape(n, H, -1) * scale
    p, j = torch.arange(pos0, pos0 + n, device=q.device)[:, None], torch.arange(k.shape[0], device=q.device)[None, :]
    hidden = (j > p) | ((p - j >= window) if window else torch.zeros_like(j > p))
    s = s.masked_fill(hidden[:, None, :], -math.inf)
    top = s.amax(-1, keepdim=True)
    if sink is not None:
        top = torch.maximum(top, sink.double().view(1, H, 1))
    e = (s - top).exp()
    total = e.sum(-1, keepdim=True) + (0 if sink is None else (sink.double().view(1, H, 1) - top).exp())
    return torch.einsum("ngik,kgv->ngiv", (e / total).view(n, G, H // G, -1), v.double()).reshape(n, H, -1)


# (tokens before, new tokens): a tile's edges, a last tile of one row, prompts that continue, a sequence much shorter than the others
@pytest.mark.parametrize("spans", [[(0, 128)], [(0, 129), (0, 1), (63, 127)], [(70, 300), (0, 64), (1, 385)]])
@pytest.mark.parametrize("d,vd", [(256, 192), (192, 128), (256, 256), (192, 64)])
@pytest.mark.parametrize("window,with_sink", [(None, False), (None, True), (100, True), (64, False), (1, True), (1000, False)])
def test_wide_heads(spans, d, vd, window, with_sink):
    from qwen3_b200.csrc import ops
    H, G = (6, 2) if d == 192 else (5, 1)
    g = torch.Generator(device="cuda").manual_seed(d + vd + len(spans) + (window or 0))
    rnd = lambda *shape: torch.randn(shape, generator=g, device="cuda").to(torch.bfloat16)  # noqa: E731
    totals = [a + b for a, b in spans]
    pages = [-(-t // 64) for t in totals]
    order = torch.randperm(sum(pages), generator=torch.Generator().manual_seed(1))
    table = torch.zeros(len(spans), max(pages) + 1, dtype=torch.int32)
    kp, vp = rnd(sum(pages), G, 64, d), rnd(sum(pages), G, 64, vd)
    at = 0
    for i, n in enumerate(pages):
        table[i, :n] = order[at:at + n].int()
        at += n
    N = sum(b for _, b in spans)
    q = rnd(N, H * d)
    start = torch.tensor(np.cumsum([0] + [b for _, b in spans]), dtype=torch.int32, device="cuda")
    pos0 = torch.tensor([a for a, _ in spans], dtype=torch.int32, device="cuda")
    sink = torch.randn(H, generator=g, device="cuda") if with_sink else None
    scale, longest, table_d = d ** -0.5, max(b for _, b in spans), table.cuda()
    out = torch.full((N + 1, H * vd), float("nan"), dtype=torch.bfloat16, device="cuda")
    ops.attention_wide_prefill_tc(q, kp, vp, out[:N], start, pos0, table_d, len(spans), longest, N, H, G, d, vd, scale, window=window,
                                  sink=with_sink, sink_values=sink)
    assert ops.tcgen05_status("cuda") == 0
    tiled = torch.empty(N, H * vd, dtype=torch.bfloat16, device="cuda")
    ops.attention_capped_prefill(q, kp, vp, tiled, start, pos0, table_d, len(spans), longest, H, G, d, vd, scale, 0.0, None, with_sink,
                                 window=window, sink_values=sink)
    assert bool(out[N].isnan().all()), "written beyond the last token"
    for i, ((a, b), t) in enumerate(zip(spans, totals)):
        rows = slice(int(start[i]), int(start[i]) + b)
        ks, vs = (x[table[i, :pages[i]].long().cuda()].permute(0, 2, 1, 3).reshape(-1, G, x.shape[-1])[:t] for x in (kp, vp))
        want = exact(q[rows].view(b, H, d), ks, vs, scale, a, window, sink).reshape(b, H * vd)
        # half a last place of a bfloat16 output and the weights' 16 bits of values up to 5
        for name, got in (("tcgen05", out[rows]), ("mma.sync", tiled[rows])):
            bound = 2.0 ** -8 * want.abs() + 4e-4
            worst = ((got.double() - want).abs() - bound).max().item()
            assert worst <= 0, (name, i, worst)


def test_sizes_that_stay_where_they_were():
    from qwen3_b200.csrc import ops
    assert [ops.attention_wide_prefill_tc_fits(d, v) for d, v in ((128, 128), (64, 128), (200, 128), (256, 100), (256, 320))] == [False] * 5
