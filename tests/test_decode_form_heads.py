"""Which form of the decode attention a step gets, by the head size: clusters of small blocks all fit."""
import types

import pytest
import torch


@pytest.mark.parametrize("d,n_tokens,nkv,expected", [(128, 5, 8, (4, False)), (64, 5, 8, (7, False)), (32, 5, 8, (7, False)), (96, 6, 8, (4, False)),
                                                     (64, 6, 8, (6, False)), (256, 6, 8, (4, False)), (64, 4, 8, (8, False)), (64, 7, 8, (5, False)),
                                                     (128, 6, 16, (3, True)), (64, 6, 16, (3, False)), (256, 6, 16, (3, False)),
                                                     (128, 96, 1, (3, True)), (64, 24, 8, (1, True)), (64, 8, 16, (2, False))])
def test_blocks_of_a_row(d, n_tokens, nkv, expected, monkeypatch):
    from qwen3_b200.csrc import ops
    from qwen3_b200.parts import attention
    seen = {}

    def fused(qkv, k_pages, v_pages, out, q_norm_w, k_norm_w, cos, sin, eps, token_seq, token_pos, page_table, n, nq, nkv, d, scale, window,
              n_splits, write_kv=True, parts=None, counters=None):
        seen.update(splits=n_splits, parts=parts)
    monkeypatch.setattr(attention, "_sm_count", lambda device: 148)
    monkeypatch.setattr(ops, "attention_decode_flat_parts", lambda d, group: 64)
    monkeypatch.setattr(ops, "attention_decode_fused_max_splits", lambda d, device: 16)
    monkeypatch.setattr(ops, "attention_decode_fused", fused)
    part = types.SimpleNamespace(plain=True, num_heads=4 * nkv, num_kv_heads=nkv, head_dim=d, scale=1.0, window=None)
    scratch = types.SimpleNamespace(get=lambda name, shape, dtype: torch.empty(shape, dtype=dtype),
                                    counters=lambda name, n: torch.zeros(n, dtype=torch.int32))
    ctx = types.SimpleNamespace(n_tokens=n_tokens, device="cpu", max_context=4096, scratch=scratch, token_seq=None, token_pos=None)
    cache = types.SimpleNamespace(keys=None, values=None, shared=False)
    assert attention._decode_fused_kernel(part, None, cache, None, ctx, None, None, None, 1e-6, None, None)
    assert (seen["splits"], seen["parts"] is not None) == expected
