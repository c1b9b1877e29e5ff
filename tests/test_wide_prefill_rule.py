"""Which kernel takes the prompts of wide heads: the tcgen05 tiles of 128 rows or the `mma.sync` tiles of 64, by the spans of the step."""
import types

import pytest
import torch


# long prompts and several of them; short spans behind small windows; a prompt beside single tokens; prompts that continue
@pytest.mark.parametrize("spans,heads,d,vd,window,pays", [
    ([(0, 2048), (0, 911), (0, 1203)], 16, 256, 256, 0, True), ([(0, 2048), (0, 911), (0, 1203)], 16, 256, 256, 1024, True),
    ([(0, 4000)], 16, 256, 192, 128, True), ([(0, 512)], 16, 192, 64, 128, False), ([(0, 512)], 2, 192, 64, 16, False),
    ([(0, 130)] + [(500, 1)] * 15, 16, 192, 64, 128, False), ([(0, 2000)] + [(1000, 1)] * 31, 16, 256, 192, 64, False),
    ([(0, 128)], 1, 192, 64, 0, False), ([(3000, 512)], 16, 256, 256, 0, True), ([(0, 300)] * 6, 16, 256, 192, 0, True)])
def test_which_kernel(spans, heads, d, vd, window, pays, monkeypatch):
    from qwen3_b200.csrc import ops
    from qwen3_b200.parts import attention
    pos0, n_new = [a for a, _ in spans], [b for _, b in spans]
    assert attention.wide_prefill_pays(tuple(pos0), tuple(n_new), heads, d, vd, window, 148) == pays
    calls = []
    monkeypatch.setattr(attention, "_sm_count", lambda device: 148)
    monkeypatch.setattr(ops, "attention_wide_prefill_tc", lambda *a, **k: calls.append(k["window"]))
    part = types.SimpleNamespace(plain=False, keep_first=0, shared_values=False, softcap=0.0, chunk=None, bias_table=None, pooled=lambda c, k: None,
                                 value_heads=1, num_kv_heads=1, num_heads=heads, head_dim=d, value_dim=vd, scale=0.1, window=window or None, sink=False,
                                 sink_values=None)
    N = sum(n_new)
    ctx = types.SimpleNamespace(max_new=max(n_new), max_context=max(a + b for a, b in spans), n_tokens=N, n_seqs=len(spans), host_pos0=pos0,
                                host_n_new=n_new, seq_start=None, seq_pos0=None, device="cpu")
    out = torch.empty(N, heads * vd, dtype=torch.bfloat16, device="meta")
    cache = types.SimpleNamespace(keys=None, values=None)
    assert attention._prefill_wide_tcgen05_kernel(part, out, cache, out, ctx, None) == pays
    assert len(calls) == int(pays)


def test_without_the_lengths_of_the_sequences():
    """Of a step that does not say them the longest is looked at."""
    from qwen3_b200.parts import attention
    for window in (0, 64, 512, 4096):
        assert attention.wide_prefill_pays((100,), (700,), 16, 256, 192, window, 148)
