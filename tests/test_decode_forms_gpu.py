"""Decode steps whose rows (sequences x kv heads) would be split in three, as the engine reaches them by itself: against the plain model."""
import pytest

import schedules
from helpers import make_folder, tiny
from test_engine_gpu import check, make_requests, run_steps

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("head_dim,shared_out", [(128, True), (64, False)])
@pytest.mark.parametrize("kv_heads,sequences,use_graphs", [(16, 6, True), (16, 5, False), (8, 12, False), (4, 24, True)])
def test_three_blocks_a_row(tmp_path, head_dim, shared_out, kv_heads, sequences, use_graphs, monkeypatch):
    import torch
    from qwen3_b200 import Engine
    from qwen3_b200.csrc import ops
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the numbers of sequences are those of 148 SMs")
    cfg = tiny("D", hidden_size=128, num_attention_heads=2 * kv_heads, num_key_value_heads=kv_heads, head_dim=head_dim, intermediate_size=96)
    folder, weights = make_folder(tmp_path, cfg, seed=31)
    requests = make_requests(cfg, [20 + 37 * i % 150 for i in range(sequences)], seed=3)
    prompts = {rid: len(t) - 4 for rid, t in requests.items()}
    forms, real = set(), ops.attention_decode_fused

    def fused(*a, parts=None, **k):
        forms.add((a[18], parts is not None))
        return real(*a, parts=parts, **k)
    monkeypatch.setattr(ops, "attention_decode_fused", fused)
    engine = Engine.from_folder(folder, dtype="bfloat16", max_tokens=64 * 4 * sequences, use_graphs=use_graphs, guard_scratch=True)
    steps, rows = schedules.batched(requests, prompts, sequences)
    got = run_steps(engine, steps, rows)
    check(got, requests, cfg, weights, "bfloat16", f"{sequences} sequences of {kv_heads} kv heads")
    engine.check_kernels()
    assert forms == {(3, shared_out)} and engine.scratch_violations() == []
