"""Weights or states in host memory are refused before the library is called: a kernel would read the pointers.  Runs
without a GPU: the rows claim to be CUDA tensors, and reaching the library fails the test."""
import pytest
import torch

from rwkv_quant_b200 import _lib, synth
from rwkv_quant_b200.backends.cuda import linear_for, ops, quant_model


class _Rows(torch.Tensor):
    is_cuda = True


@pytest.fixture(autouse=True)
def _no_library(monkeypatch):
    def reached(*a, **k):
        raise AssertionError("the call reached the library")
    monkeypatch.setattr(_lib, "load", reached)


def _rows(n, cols=256):
    return torch.zeros(n, cols).as_subclass(_Rows)


def _tensor(layout="sb6", bits=4):
    return getattr(synth, "quant_" + layout)("w", "proj", torch.randn(256, 256, generator=torch.Generator().manual_seed(0)), bits)


@pytest.mark.parametrize("layout,bits", [("sb6", 4), ("sym", 8), ("rtn", 8)])
@pytest.mark.parametrize("n", [1, 2, 3, 20, 200])
def test_operator_with_weights_on_the_host(layout, bits, n):
    op = linear_for(_tensor(layout, bits), "cpu")               # constructible: its sizes can be asked for
    assert op.weight_nbytes() > 0
    with pytest.raises(RuntimeError, match="CUDA tensors only"):
        op(_rows(n))


def test_library_wrappers_with_weights_on_the_host():
    dq = ops.DeviceQT(_tensor(), "cpu")
    rows = ops.PreparedRows(4, 256)
    rows.x16, rows.scale = _rows(4), _rows(1)
    for call in (lambda: ops.gemv_direct(dq, _rows(1)), lambda: ops.gemv_batch(dq, _rows(4)), lambda: ops.gemm(dq, _rows(4)),
                 lambda: ops.gemm_x16(dq, rows), lambda: ops.gemv_fused([dq, dq], _rows(2)),
                 lambda: ops.lora_pair([(dq, dq)], [_rows(4)], [0])):
        with pytest.raises(RuntimeError, match="CUDA tensors only"):
            call()


@pytest.mark.parametrize("which", [0, 1, 2])
def test_states_on_the_host(monkeypatch, which):
    m = object.__new__(quant_model.QuantRWKV7)
    m.n_layer, m.n_head, m.head_size, m.n_embd, m.vocab_size, m.device = 1, 4, 64, 256, 512, torch.device("cpu")
    m._one_call_ok = lambda n: True
    state = [_rows(4 * 64, 64).reshape(1, 4, 64, 64), _rows(1).reshape(1, 1, 256), _rows(1).reshape(1, 1, 256)]
    state[which] = state[which].as_subclass(torch.Tensor)
    for T in (1, 5):
        with pytest.raises(RuntimeError, match="CUDA tensors only"):
            m.forward_stateful(torch.zeros(1, T, dtype=torch.long), [tuple(state)])
