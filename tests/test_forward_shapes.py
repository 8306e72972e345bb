"""rwkvq_forward_seq_ok accepts a model only if every tensor has the shape its place in the pass needs: the kernels are
given addresses and sizes that follow from the model's dimensions.  Host logic, no GPU."""
import ctypes as C

import pytest

from rwkv_quant_b200 import _lib

D, F, V, R = 256, 1024, 512, 32
LINEAR = {"Wr": (D, D), "Wk": (D, D), "Wv": (D, D), "Wo": (D, D), "Wfk": (F, D), "Wfv": (D, F)}


def _sb6(rows, cols):
    t = _lib.QTensorStruct(kind=_lib.KIND["sb6"], bits=4, rows=rows, cols=cols, gs=32, sb=8)
    t.codes = t.qsqm = t.d = t.dm = t.dev_meta = 0x1000
    return t


def _rtn(rows, cols):
    t = _lib.QTensorStruct(kind=_lib.KIND["rtn"], bits=8, rows=rows, cols=cols)
    t.codes = t.scale = 0x1000
    return t


def _model():
    layers = (_lib.LayerStruct * 2)()
    for i, L in enumerate(layers):
        for n, shape in LINEAR.items():
            setattr(L, n, _sb6(*shape))
        for b in "wagv" if i else "wag":
            setattr(L, b + "1", _rtn(D, R))
            setattr(L, b + "2", _rtn(R, D))
    m = _lib.ModelStruct(n_layer=2, n_embd=D, head_size=64, vocab_size=V, ffn_dim=F, max_rank=R)
    m.emb, m.head = _sb6(V, D), _sb6(V, D)
    m.layers = C.cast(layers, C.POINTER(_lib.LayerStruct))
    return m, layers


def _ok(m):
    return [_lib.load().rwkvq_forward_seq_ok(C.byref(m), n) for n in (5, 40, 100)]


def test_a_model_of_one_set_of_dimensions_is_served():
    m, layers = _model()
    assert _ok(m) == [1, 1, 1]


@pytest.mark.parametrize("name", [*LINEAR, "w1", "w2", "v1", "v2", "head", "emb"])
@pytest.mark.parametrize("side", ["rows", "cols"])
def test_a_tensor_of_another_shape_is_not(name, side):
    m, layers = _model()
    t = getattr(m if name in ("head", "emb") else layers[1], name)
    if (name, side) == ("emb", "rows"):
        return                                            # tokens are clamped to the table
    setattr(t, side, getattr(t, side) + 256)
    assert _ok(m) == [0, 0, 0]


def test_a_rank_above_the_scratch_is_not():
    m, layers = _model()
    layers[1].g1, layers[1].g2 = _rtn(D, 2 * R), _rtn(2 * R, D)
    assert _ok(m) == [0, 0, 0]


@pytest.mark.parametrize("name", ["v1", "v2", "w1", "g2", "Wo"])
def test_a_tensor_without_its_buffers_is_refused_before_any_launch(name):
    m, layers = _model()
    getattr(layers[1], name).codes = None
    two = (C.c_void_p * 2)(0x1000, 0x1000)
    for T in (5, 100):
        rc = _lib.load().rwkvq_forward_seq(C.byref(m), 1, T, 0x1000, two, two, two, two, two, two, 0, None, None, 0x1000, 0, None)
        assert rc == -7, rc                               # RWKVQ_E_NULL, not the workspace's RWKVQ_E_LIMIT behind it
