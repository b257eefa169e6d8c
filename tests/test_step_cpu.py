"""The launches of a generation step without a GPU: model.Llama's step with recorders in the place of the kernels."""
import pytest


@pytest.fixture
def step(pkg, monkeypatch):
    """step(weight_type, kv_sink) -> [(entry, keyword arguments)] in launch order."""
    import torch
    from llm_infer_b200 import model as M
    cfg = M.ModelConfig(dim=64, hidden_dim=64, n_layers=2, n_heads=1, n_kv_heads=1, head_dim=64, vocab_size=32, max_seq_len=300,
                        norm_eps=1e-5, rope_theta=1e4)
    calls = []

    def recorder(name):
        return lambda *args, **kwargs: calls.append((name, kwargs))

    for name in ("rmsnorm", "rope_kv_insert", "attn_decode", "argmax"):
        monkeypatch.setattr(M.A, name, recorder(name))

    def run(weight_type, kv_sink):
        del calls[:]
        m = M.Llama.__new__(M.Llama)
        act = torch.int32 if weight_type == "q8_0" else torch.float32
        z = lambda *s, dtype=torch.float32: torch.zeros(*s, dtype=dtype)  # noqa: E731
        m.cfg, m.batch, m.weight_type, m._rows, m.kv_early, m._k_split, m.partials = cfg, 1, weight_type, {}, True, 1, None
        m.wg = {k: [None] * cfg.n_layers for k in ("rms_att", "rms_ffn", "wqkv", "wo", "w13", "w2")}
        m.wg.update(embed=None, rms_final=None, wcls=None)
        m._gemv, m._embed = recorder("gemv"), recorder("embed")
        m._q_dim = m._kv_dim = 64
        m.x, m.xb, m.hb, m.logits = z(1, 64), z(1, 64, dtype=act), z(1, 64, dtype=act), z(1, 32)
        m.q, m.k, m.v, m.att = z(1, 1, 64), z(1, 1, 64), z(1, 1, 64), z(1, 1, 64, dtype=act)
        m.tokens, m.next_token, m.status = (z(1, dtype=torch.int32) for _ in range(3))
        m.pos, m.kv_pos, m.kv_len = (z(1, dtype=torch.int32) for _ in range(3))
        m.k_cache, m.v_cache, m.workspace = z(cfg.n_layers, 1), z(cfg.n_layers, 1), None
        m._launch_step(kv_sink, True)
        return list(calls)

    return run


@pytest.mark.parametrize("weight_type", ["f16", "q8_0"])
def test_every_step_asks_for_the_form_with_one_order_of_sums(step, weight_type):
    """Whatever the weights: the order of the attention's sums decides fp16 ties of the next layers' cache rows."""
    attention = [kw for name, kw in step(weight_type, 0) if name == "attn_decode"]
    assert len(attention) == 2 and all(kw["two_pass"] for kw in attention)


@pytest.mark.parametrize("kv_sink", [0, 4])
def test_early_streaming_stops_at_the_sliding_window(step, kv_sink):
    """In the window the rotary kernel writes a row inside the ring and turns the sink rows: no row may be read before it."""
    calls = step("f16", kv_sink)
    assert [kw["kv_sink"] for name, kw in calls if name == "rope_kv_insert"] == [kv_sink] * 2
    assert [bool(kw["kv_early"]) for name, kw in calls if name == "attn_decode"] == [kv_sink == 0] * 2
