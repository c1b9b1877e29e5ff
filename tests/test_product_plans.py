"""Products whose epilogue needs tiles of whole 256 tokens are planned by the time that these take."""
import types

import pytest
import torch


@pytest.fixture
def asked(monkeypatch):
    """The estimates asked for, on a stand-in device: 100 us in whole 256s, 10 us where tiles of equal tokens may be taken."""
    from qwen3_b200.csrc import ops
    from qwen3_b200.parts import linear as L
    seen = []
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch.cuda, "get_device_properties", lambda device: types.SimpleNamespace(multi_processor_count=148))
    monkeypatch.setattr(ops, "gemm_tcgen05_pair_capacity", lambda splits: 0)
    monkeypatch.setattr(ops, "gemm_tcgen05_mid_splits", lambda M, N, K: 1)
    monkeypatch.setattr(ops, "gemm_tcgen05_pair_us", lambda M, N, K, may_row=True: seen.append(may_row) or (10.0 if may_row else 100.0))
    for f in (L.pair_plan, L.tcgen05_form):
        f.cache_clear()
    yield seen
    for f in (L.pair_plan, L.tcgen05_form):
        f.cache_clear()


def test_squared_relu(asked, monkeypatch):
    from qwen3_b200.csrc import ops
    from qwen3_b200.parts import mlp
    forms = []
    monkeypatch.setattr(ops, "gemm_relu2", lambda x, w, out, form, splits=0: forms.append(form))
    monkeypatch.setattr(mlp, "linear", lambda x, w, out: out)
    part = mlp.DenseMLP(4096, 4096, activation="relu2")
    scratch = types.SimpleNamespace(get=lambda name, shape, dtype: torch.empty(shape, dtype=dtype, device="meta"))
    part.forward(torch.empty(300, 4096, dtype=torch.bfloat16, device="meta"), types.SimpleNamespace(n_tokens=300, dtype=torch.bfloat16, scratch=scratch))
    # weights first: 64 K steps of 0.40 us and 5 us, less than whole 256s and more than the tiles that this product cannot have
    assert forms == ["mid"] and asked and not any(asked)


def test_fused_projection(asked):
    from qwen3_b200.parts import attention
    part = types.SimpleNamespace(plain=True, num_heads=32, num_kv_heads=8, head_dim=128, hidden_size=4096)
    ctx = types.SimpleNamespace(n_tokens=attention.fused_projection_rows)
    # 128 x 128 tiles take longer than the 10 us and less than the 100: only by the wrong estimate would the fused kernel run
    from qwen3_b200.parts import linear as L
    L._STEP_US["prompt128"], kept = 0.05, L._STEP_US["prompt128"]
    try:
        assert not attention._projection_pair_kernel(part, None, None, None, ctx, None, None, None, 1e-6, None, None)
    finally:
        L._STEP_US["prompt128"] = kept
    assert asked and not any(asked)


def test_other_products_may_take_them(asked):
    from qwen3_b200.parts import linear as L
    assert L.pair_plan(300, 4096, 4096) == (10.0, 1) and L.tcgen05_form(300, 24576, 4096, gated=True) == "pair"
    assert L.pair_plan(300, 4096, 4096, may_row=False) == (100.0, 1)
