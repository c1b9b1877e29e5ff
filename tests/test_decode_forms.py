"""Which form of the decode attention a step gets, by the blocks that a (sequence, kv head) can have."""
import types

import pytest
import torch


@pytest.mark.parametrize("n_tokens,nkv,expected", [(1, 8, (8, False)), (4, 8, (8, False)), (5, 8, (4, False)), (6, 8, (4, False)),
                                                   (7, 8, (5, False)), (8, 8, (4, False)), (12, 8, (3, True)), (16, 8, (2, False)),
                                                   (24, 8, (1, True)), (12, 4, (4, False)), (20, 4, (3, True))])
def test_blocks_of_a_row(n_tokens, nkv, expected, monkeypatch):
    from qwen3_b200.csrc import ops
    from qwen3_b200.parts import attention
    seen = {}
    monkeypatch.setattr(attention, "_sm_count", lambda device: 148)
    monkeypatch.setattr(ops, "attention_decode_flat_parts", lambda d, group: 64)
    monkeypatch.setattr(ops, "attention_decode_fused_max_splits", lambda d, device: 16)
    monkeypatch.setattr(ops, "attention_decode_fused", lambda *a, **k: seen.update(splits=a[18], parts=k["parts"]))
    part = types.SimpleNamespace(plain=True, num_heads=4 * nkv, num_kv_heads=nkv, head_dim=128, scale=1.0, window=None)
    scratch = types.SimpleNamespace(get=lambda name, shape, dtype: torch.empty(shape, dtype=dtype),
                                    counters=lambda name, n: torch.zeros(n, dtype=torch.int32))
    ctx = types.SimpleNamespace(n_tokens=n_tokens, device="cpu", max_context=4096, scratch=scratch, token_seq=None, token_pos=None)
    cache = types.SimpleNamespace(keys=None, values=None, shared=False)
    assert attention._decode_fused_kernel(part, None, cache, None, ctx, None, None, None, 1e-6, None, None)
    assert (seen["splits"], seen["parts"] is not None) == expected
