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
