"""Attention of prompts on tcgen05 with sinks that weigh nothing and with values that are no numbers, against 64 bits."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def exact(q, k, v, scale, pos0, window, sink, chunk=0):
    """q [n, H, d], k [keys, G, d], v [keys, G, vd] of one sequence, the new tokens at pos0 ..: [n, H, vd] in 64 bits."""
    n, H, _ = q.shape
    G = k.shape[1]
    s = torch.einsum("ngid,kgd->ngik", q.double().view(n, G, H // G, -1), k.double()).reshape(n, H, -1) * scale
    p, j = torch.arange(pos0, pos0 + n, device=q.device)[:, None], torch.arange(k.shape[0], device=q.device)[None, :]
    hidden = (j > p) | ((p - j >= window) if window else torch.zeros_like(j > p))
    if chunk:
        hidden = hidden | (j < p // chunk * chunk)
    s = s.masked_fill(hidden[:, None, :], -math.inf)
    top = s.amax(-1, keepdim=True)
    if sink is not None:
        top = torch.maximum(top, sink.double().view(1, H, 1))
    e = (s - top).exp()
    total = e.sum(-1, keepdim=True) + (0 if sink is None else (sink.double().view(1, H, 1) - top).exp())
    return torch.einsum("ngik,kgv->ngiv", (e / total).view(n, G, H // G, -1), v.double()).reshape(n, H, -1)


def paged(spans, G, d, vd, g):
    """Keys and values of the sequences in pages in a mixed order: the pages, their table and what each sequence sees of them."""
    totals = [a + b for a, b in spans]
    pages = [-(-t // 64) for t in totals]
    order = torch.randperm(sum(pages), generator=torch.Generator().manual_seed(2))
    table = torch.zeros(len(spans), max(pages), dtype=torch.int32)
    at = 0
    for i, n in enumerate(pages):
        table[i, :n] = order[at:at + n].int()
        at += n
    kp, vp = (torch.randn(sum(pages), G, 64, n, generator=g, device="cuda").to(torch.bfloat16) for n in (d, vd))
    own = lambda x, i: x[table[i, :pages[i]].long().cuda()].permute(0, 2, 1, 3).reshape(-1, G, x.shape[-1])[:totals[i]]  # noqa: E731
    return kp, vp, table.cuda(), own


LOWEST = [-math.inf, torch.finfo(torch.float32).min, torch.finfo(torch.bfloat16).min, -1e30, 0.25, 3.0]


# Sinks that weigh nothing, down to minus infinity, one per head beside ordinary ones.  Behind a window, or with chunks, half of a tile's rows
# see nothing of its first page, so that the sink alone stands there.
@pytest.mark.parametrize("d,vd,window,chunk", [(256, 192, 64, 0), (256, 192, 100, 0), (192, 128, 64, 0), (256, 256, None, 0),
                                               (64, 64, None, 100), (128, 128, None, 64), (128, 128, None, 100)])
def test_sinks_that_weigh_nothing(d, vd, window, chunk):
    from qwen3_b200.csrc import ops
    H, G, spans = 6, 1, [(0, 300), (70, 129)]
    g = torch.Generator(device="cuda").manual_seed(d + vd)
    kp, vp, table, own = paged(spans, G, d, vd, g)
    N = sum(b for _, b in spans)
    q = torch.randn(N, H * d, generator=g, device="cuda").to(torch.bfloat16)
    start, pos0 = (torch.tensor(x, dtype=torch.int32, device="cuda") for x in ([0, 300, N], [0, 70]))
    sink, scale = torch.tensor(LOWEST, device="cuda"), d ** -0.5
    out = torch.full((N, H * vd), float("nan"), dtype=torch.bfloat16, device="cuda")
    if d > 128:
        ops.attention_wide_prefill_tc(q, kp, vp, out, start, pos0, table, 2, 300, N, H, G, d, vd, scale, window=window, sink=True,
                                      sink_values=sink)
    else:
        ops.attention_capped_prefill_tc(q, kp, vp, out, start, pos0, table, 2, 300, N, H, G, d, scale, 0.0, chunk, True, sink_values=sink)
    assert ops.tcgen05_status("cuda") == 0
    for i, (a, b) in enumerate(spans):
        rows = slice(int(start[i]), int(start[i]) + b)
        want = exact(q[rows].view(b, H, d), own(kp, i), own(vp, i), scale, a, window, sink, chunk).reshape(b, H * vd)
        excess = (out[rows].double() - want).abs() - (2.0 ** -8 * want.abs() + 4e-4)         # as above
        assert not bool(excess.isnan().any()) and excess.max().item() <= 0, (i, excess.max().item())


# Values that are no numbers, in pages of which some rows of a tile see other keys: behind the last token (slots nobody wrote), later than
# some rows, before the window of others, in a tile's first page and in later ones, twice the same column.  They belong to the rows that see
# them; all others are what they are without them.
@pytest.mark.parametrize("d,vd,window", [(256, 192, None), (256, 192, 100), (192, 128, 64), (256, 256, 1)])
@pytest.mark.parametrize("bad", [[(0, 5, 0, math.inf)], [(0, 130, 63, -math.inf), (0, 299, 40, math.nan)], [(1, 198, 17, math.inf), (1, 70, 33, math.nan)],
                                 [(0, 64, 8, math.inf), (0, 65, 8, -math.inf), (1, 0, 1, math.nan)], [(0, 300, 2, math.nan), (1, 199, 60, math.inf)]])
def test_values_that_are_no_numbers(d, vd, window, bad):
    from qwen3_b200.csrc import ops
    H, G, spans = 4, 2, [(0, 300), (70, 129)]
    g = torch.Generator(device="cuda").manual_seed(d + vd + 1)
    kp, vp, table, own = paged(spans, G, d, vd, g)
    N = sum(b for _, b in spans)
    q = torch.randn(N, H * d, generator=g, device="cuda").to(torch.bfloat16)
    start, pos0 = (torch.tensor(x, dtype=torch.int32, device="cuda") for x in ([0, 300, N], [0, 70]))
    want = [exact(q[s:s + b].view(b, H, d), own(kp, i), own(vp, i), d ** -0.5, a, window, None) for i, (s, (a, b)) in enumerate(zip((0, 300), spans))]
    touched = [torch.zeros_like(w, dtype=torch.bool) for w in want]
    for seq, key, col, value in bad:                       # in the second kv head, whose queries are the heads 2 and 3
        vp[table[seq, key // 64].item(), 1, key % 64, col] = value
        a, b = spans[seq]
        sees = torch.arange(a, a + b, device="cuda") - key
        touched[seq][:, 2:, col] |= ((sees >= 0) & (sees < (window or 1 << 30)))[:, None]
    out = torch.full((N, H * vd), float("nan"), dtype=torch.bfloat16, device="cuda")
    ops.attention_wide_prefill_tc(q, kp, vp, out, start, pos0, table, 2, 300, N, H, G, d, vd, d ** -0.5, window=window)
    assert ops.tcgen05_status("cuda") == 0
    for i, (s, (a, b)) in enumerate(zip((0, 300), spans)):
        got = out[s:s + b].double().view(b, H, vd)
        assert bool((~got[touched[i]].isfinite()).all()), "a value that a row sees is lost"
        excess = (got - want[i]).abs() - (2.0 ** -8 * want[i].abs() + 4e-4)              # as above
        assert bool((excess <= 0)[~touched[i]].all()), "a value reaches rows that do not see it"
