"""Which calls the one-call forward takes (host logic; the library is a stand-in)."""
import pytest

from rwkv_quant_b200 import _lib
from rwkv_quant_b200.backends.cuda import quant_model


class _Lib:
    """Answers as the library does for a model whose layouts it serves in both regimes."""
    @staticmethod
    def rwkvq_forward_seq_ok(model, n_rows):
        return int(n_rows >= 2)


def _model(monkeypatch, **kw):
    monkeypatch.setattr(_lib, "load", lambda *a, **k: _Lib)
    m = object.__new__(quant_model.QuantRWKV7)
    m._model_c, m.fused_prep, m._seq_ok = _lib.ModelStruct(), True, {}
    m.gemv_max_batch, m.gemm_min_batch, m.batch_max = 2, 128, 64
    m.__dict__.update(kw)
    return m


def test_an_empty_call_does_not_close_the_route(monkeypatch):
    m = _model(monkeypatch)
    assert not m._one_call_ok(0)
    assert m._one_call_ok(5) and m._one_call_ok(64) and m._one_call_ok(65)


@pytest.mark.parametrize("kw,served,refused", [
    (dict(gemv_max_batch=8), (2, 9, 64, 65, 500), (3, 5, 8)),        # single-vector kernels up to 8 rows were asked for
    (dict(gemv_max_batch=0), (3, 64, 65), (2,)),
    (dict(batch_max=16), (2, 3, 16, 65), (17, 40, 64)),
    (dict(gemv_max_batch=100), (2, 101), (3, 64, 65, 100)),
])
def test_row_limits_of_the_model_are_kept(monkeypatch, kw, served, refused):
    m = _model(monkeypatch, **kw)
    assert [n for n in served if not m._one_call_ok(n)] == []
    assert [n for n in refused if m._one_call_ok(n)] == []


@pytest.mark.parametrize("n,given", [(2, iter), (3, list), (1, list)])
def test_states_of_another_count_take_the_layers_they_name(monkeypatch, n, given):
    """Any iterable, one entry a layer; with another count the layers and the states are paired up as far as both go."""
    import torch
    calls = []
    m = _model(monkeypatch, n_layer=2, blocks=["a", "b"], device=torch.device("cpu"), n_embd=8192, vocab_size=5, head="h")
    m._forward_one_call = lambda idx, states, tail, hidden: calls.append(("one", len(states))) or (None, 0, 0)
    m._materialize = lambda states, B: list(states)
    m._embed = lambda idx: torch.zeros(*idx.shape, 8192)
    m.ln0 = m.ln_out = (torch.ones(8192), torch.zeros(8192))
    m.emb = type("E", (), {"outliers": None})
    m._block_seq = lambda i, L, x, v, st: calls.append((L, st)) or (x, v, st)
    m._linear = lambda dq, x: torch.zeros(x.shape[0], 5)
    m.forward_stateful(torch.zeros(1, 5, dtype=torch.long), given(["s0", "s1", "s2"][:n]))
    assert calls == ([("one", 2)] if n == 2 else [("a", "s0"), ("b", "s1")][:n])
