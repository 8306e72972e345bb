"""Scratch is sized by what a call uses.  Host logic, no GPU."""
import ctypes as C

import pytest

from rwkv_quant_b200 import _lib

MB = 1 << 20


def _tensor(kind, bits, rows, cols, relayout=True):
    t = _lib.QTensorStruct(kind=_lib.KIND[kind], bits=bits, rows=rows, cols=cols, gs={"sb6": 32, "sym": 16}.get(kind, 0),
                           sb={"sb6": 8, "sym": 16}.get(kind, 0))
    t.codes = t.scale = 0x1000
    t.qsqm = t.d = t.dm = t.qs = 0x1000
    if relayout:
        t.dev_meta = t.dev_planes = 0x1000
    return t


def _model(D=2048, F=8192, V=65536, R=128, n_layer=24, relayout=True):
    layers = (_lib.LayerStruct * n_layer)()
    for L in layers:
        for n, shape in dict(Wr=(D, D), Wk=(D, D), Wv=(D, D), Wo=(D, D), Wfk=(F, D), Wfv=(D, F)).items():
            setattr(L, n, _tensor("sb6", 4, *shape, relayout))
    m = _lib.ModelStruct(n_layer=n_layer, n_embd=D, head_size=64, vocab_size=V, ffn_dim=F, max_rank=R)
    m.emb, m.head = _tensor("sb6", 5, V, D, relayout), _tensor("sb6", 5, V, D, relayout)
    m.layers = C.cast(layers, C.POINTER(_lib.LayerStruct))
    return m, layers


def test_gemm_holds_its_own_weights():
    lib = _lib.load()
    of = lambda t, m, rows: lib.rwkvq_gemm_workspace_bytes_of(C.byref(t), m, rows)
    small, head = _tensor("sb6", 4, 2048, 2048), _tensor("sym", 8, 65536, 2048)
    assert of(small, 128, 0) <= 2048 * 2048 * 2 + 4096
    assert of(small, 128, 1) <= 2048 * 2048 * 2 + 128 * (2048 + 64) * 2 + 4096
    assert 64 * MB <= of(head, 128, 0) <= 65 * MB                     # a chunk
    for t in (small, head, _tensor("sb6", 4, 300, 131328)):
        assert of(t, 500, 1) <= lib.rwkvq_gemm_workspace_bytes_for(500, t.cols) and of(t, 500, 0) <= lib.rwkvq_gemm_workspace_bytes_for(500, 0)


@pytest.mark.parametrize("tensor,n,pairs", [(("sb6", 4, 2048, 2048), 8, False), (("sb6", 4, 2048, 2048), 9, True),
                                            (("sb6", 4, 2048, 2048), 16, True), (("sb6", 4, 2048, 2048), 17, True),
                                            (("sb6", 4, 2048, 2048, False), 100, False), (("rtn", 8, 2048, 2048), 4096, False),
                                            (("sym", 8, 256, 16640), 100, False)])
def test_pairs_only_where_the_pipeline_reads_them(tensor, n, pairs):
    lib, t = _lib.load(), _tensor(*tensor)
    got = lib.rwkvq_gemv_batch_workspace_bytes_of(C.byref(t), n)
    rows = 256 + (4 * n + 255) // 256 * 256
    assert got <= lib.rwkvq_gemv_batch_workspace_bytes(n)
    assert got == rows if not pairs else rows < got <= rows + n * (4 * (2048 + 64) + 32 * 2048 // 256)


@pytest.mark.parametrize("B", [1, 2, 16, 64, 256])
def test_a_decode_step_has_no_room_for_kernels_it_does_not_use(B):
    m, _ = _model()
    lib = _lib.load()
    per_stream = 4 * (65536 + 8192 * 3 + 2048 * 40) + 64 * 1024
    assert lib.rwkvq_decode_workspace_bytes(C.byref(m), B) <= B * per_stream + 8 * MB
    assert lib.rwkvq_decode_workspace_bytes(C.byref(m), 300) >= 64 * MB
    bare, _ = _model(relayout=False)
    assert lib.rwkvq_decode_workspace_bytes(C.byref(bare), 64) >= 64 * MB


def test_logits_of_every_position_cost_the_head_gemm_only():
    m, _ = _model()
    size = lambda tail: _lib.load().rwkvq_forward_seq_workspace_bytes(C.byref(m), 16, 512, tail)
    n = 16 * 512
    assert size(512) - size(0) <= n * (2 * 2048 * 4 + (2048 + 64) * 2 + 4) + 64 * MB + 4096
    assert size(1) - size(0) <= 2 * MB
