"""Inputs at the edges of what the forward calls, the decode step and the linears take: non-finite values, tensors off
16-byte boundaries, states that share their storage, shapes beyond one kernel's range."""
import numpy as np
import pytest
import torch

from helpers import relmax
from test_gpu_dequant_gemv import _oracle_w, _synth_linear, _x

pytestmark = pytest.mark.gpu


def _model(recipe="compression", n_embd=256, ffn=1024, **kw):
    from rwkv_quant_b200 import synth
    from rwkv_quant_b200.backends.cuda import QuantRWKV7
    return QuantRWKV7(synth.build_checkpoint(dict(n_layer=2, vocab=512, n_embd=n_embd, ffn=ffn), recipe, seed=3, device="cuda"),
                      device="cuda", **kw)


def _states(model, B, offset=0):
    """States whose shift rows start ``offset`` floats behind a 16-byte boundary."""
    gen = torch.Generator(device="cuda").manual_seed(B)

    def draw(*shape, off=0):
        t = torch.empty(int(np.prod(shape)) + off, device="cuda")[off:].view(shape)
        return t.copy_(0.2 * torch.randn(shape, generator=gen, device="cuda"))
    D, H = model.n_embd, model.n_head
    return [(draw(B, H, 64, 64), draw(B, 1, D, off=offset), draw(B, 1, D, off=offset)) for _ in range(model.n_layer)]


def _idx(B, T):
    return torch.randint(1, 512, (B, T), generator=torch.Generator().manual_seed(100 * B + T)).cuda()


@pytest.mark.parametrize("B", [3, 20])
def test_shift_rows_off_16_byte_boundaries(cuda_lib, B):
    """Both regimes of a decode step and of short and long forward calls; a WKV state there is refused."""
    model = _model()
    for T in (1, 2, 17):
        idx = _idx(B, T)
        ref, rst = model.forward_stateful(idx, _states(model, B))
        got, gst = model.forward_stateful(idx, _states(model, B, offset=1))
        assert relmax(got.cpu().numpy(), ref.cpu().numpy()) <= 1e-4
        for s, r in zip(gst, rst):
            for a, b in zip(s, r):
                assert relmax(a.cpu().numpy(), b.cpu().numpy()) <= 1e-4
        off = [(torch.zeros(s[0].numel() + 1, device="cuda")[1:].view(s[0].shape), s[1], s[2]) for s in _states(model, B)]
        with pytest.raises(RuntimeError, match="16-byte"):
            model.forward_stateful(idx, off)


@pytest.mark.parametrize("bits", [6, 8])
@pytest.mark.parametrize("N", [8, 9, 16, 17, 64])
def test_block_scales_on_an_8_byte_boundary(cuda_lib, bits, N):
    """The int8 scale codes of a sym tensor may start on any boundary that suits the mma.sync kernel (8 bytes)."""
    from rwkv_quant_b200.backends.cuda import ops
    dq = ops.DeviceQT(_synth_linear("sym", bits, 256, 512, seed=bits))
    x = _x(N, 512, N)
    want = ops.gemv_batch(dq, x, check=True)
    i = ops._BUF_ORDER.index("qs")
    qs = dq.bufs[i]
    room = torch.empty(qs.numel() + 8, dtype=qs.dtype, device="cuda")
    assert room.data_ptr() % 16 == 0
    dq.bufs[i] = room[8:].view(qs.shape).copy_(qs)
    dq.struct = ops._descr(dq.bufs, dq.meta)
    got = ops.gemv_batch(dq, x, check=True)
    assert relmax(got.cpu().numpy(), want.cpu().numpy()) <= 4e-6       # another kernel from 9 rows on


@pytest.mark.parametrize("layout,bits,cols", [("sb6", 4, 33024), ("sym", 8, 33024), ("sb6", 5, 131328)])
def test_many_rows_through_a_wide_tensor(cuda_lib, layout, bits, cols):
    """More columns than a chunk of 256 converted rows leaves room for, and more than the norm table of the channel mix."""
    from rwkv_quant_b200.backends.cuda import ops
    qt = _synth_linear(layout, bits, 300, cols, seed=bits)
    x = _x(130, cols, bits)
    y = ops.gemm(ops.DeviceQT(qt), x, check=True)
    want = x.cpu().numpy().astype(np.float64) @ _oracle_w(qt).astype(np.float64).T
    assert relmax(y.cpu().numpy(), want) <= 1e-3


@pytest.mark.parametrize("layout,bits", [("sb6", 4), ("sb6", 6), ("sym", 6)])
@pytest.mark.parametrize("N", [3, 20, 70])
def test_wide_tensor_without_relayouted_streams(cuda_lib, layout, bits, N):
    """More columns than the pipeline's operand scratch holds: the kernel that reads the file buffers serves them."""
    from rwkv_quant_b200.backends.cuda import ops
    qt = _synth_linear(layout, bits, 160, 16640, seed=bits + N)
    x = _x(N, 16640, N)
    want = x.cpu().numpy().astype(np.float64) @ _oracle_w(qt).astype(np.float64).T
    for relayout in (False, True):
        y = ops.gemv_batch(ops.DeviceQT(qt, relayout=relayout), x, check=True)
        assert relmax(y.cpu().numpy(), want) <= 2e-5, relayout


@pytest.mark.parametrize("D,B", [(256, 70), (384, 70), (2048, 70), (256, 666), (256, 667), (2048, 74), (2048, 75), (2304, 75), (2560, 37),
                                 (2560, 38), (4096, 38)])
def test_shift_state_updated_in_place(cuda_lib, D, B):
    """One token a sequence: the row preparation may write the shift state over its input, whatever the width; streams on each side of
    the line from which one CTA makes all rows of a token."""
    import ctypes as C
    from rwkv_quant_b200 import _lib
    gen = torch.Generator(device="cuda").manual_seed(D)
    draw = lambda *s: torch.randn(s, generator=gen, device="cuda")
    x, w, b, mix, shift = draw(B, D), draw(D), draw(D), draw(6, D), draw(B, D)
    xn = torch.nn.functional.layer_norm(x.double(), (D,), w.double(), b.double())
    want = torch.stack([xn + (shift.double() - xn) * m.double() for m in mix])
    out = torch.empty(6, B, D, device="cuda")
    tab = (C.c_void_p * 6)(*[out[m].data_ptr() for m in range(6)])
    none = (C.c_void_p * 6)()
    _lib.check(cuda_lib.rwkvq_seq_ln_shift_mix_prep(x.data_ptr(), w.data_ptr(), b.data_ptr(), shift.data_ptr(), mix.data_ptr(), 6,
                                                    (C.c_int * 6)(*[4] * 6), none, none, none, tab, shift.data_ptr(), B, 1, D,
                                                    _lib.stream_ptr()), "prep")
    assert relmax(out.cpu().numpy(), want.cpu().numpy()) <= 1e-5
    assert relmax(shift.cpu().numpy(), xn.cpu().numpy()) <= 1e-5


@pytest.mark.parametrize("name", ["w0", "a0", "v0"])
@pytest.mark.parametrize("value", [float("nan"), float("inf"), -float("inf")])
@pytest.mark.parametrize("T", [15, 17])
def test_a_non_finite_gate_input_reaches_the_outputs(cuda_lib, name, value, T):
    """Both time-mix forms of calls of more than 64 rows (T on each side of the shortest chunked one) against the
    per-operator path: a NaN in front of a sigmoid stays a NaN, an infinity saturates it."""
    model = _model()
    getattr(model.blocks[1], name)[70] = value
    idx, st = _idx(5, T), _states(model, 5)
    got, gst = model.forward_stateful(idx, st)
    model.fused_prep = False
    ref, rst = model.forward_stateful(idx, st)
    for a, b in [(got, ref)] + [(x, y) for s, r in zip(gst, rst) for x, y in zip(s, r)]:
        assert torch.equal(a.isnan(), b.isnan())
        assert torch.equal(a.isnan(), torch.zeros_like(a.isnan())) or value != value
        ok = ~a.isnan()
        if ok.any():
            assert relmax(a[ok].cpu().numpy(), b[ok].cpu().numpy()) <= 1e-3
    assert value == value or got.isnan().any()


@pytest.mark.parametrize("B,t", [(3, 0), (3, 3), (3, 7), (3, 8), (3, 21), (30, 5), (40, 5)])      # one form of the scan each
def test_a_nan_token_leaves_earlier_positions_alone(cuda_lib, B, t):
    from rwkv_quant_b200.backends.cuda.ops import _BUF_ORDER
    model = _model()
    idx, st = _idx(B, 24), _states(model, B)
    idx[idx == 500] = 501
    idx[1, t] = 500
    clean, _ = model.forward_stateful(idx, st)
    model.emb.bufs[_BUF_ORDER.index("dm")][500] = float("nan")
    got, _ = model.forward_stateful(idx, st)
    assert got[1, t:].isnan().all()
    assert torch.equal(got[1, :t], clean[1, :t])
    others = [b for b in range(B) if b != 1]
    assert torch.equal(got[others], clean[others])


@pytest.mark.parametrize("tail", [1, 3, 5, 9, -2])
def test_tail_only_selects_as_a_slice_does(cuda_lib, tail):
    model = _model()
    idx, st = _idx(2, 5), _states(model, 2)
    full, _ = model.forward_stateful(idx, st)
    got, _ = model.forward_stateful(idx, st, tail_only=tail)
    want = full[:, -tail:] if 5 > tail else full
    assert got.shape == want.shape and relmax(got.cpu().numpy(), want.cpu().numpy()) <= 1e-5


@pytest.mark.parametrize("rows", [1, 2])
def test_an_operator_call_that_autograd_or_a_tracer_sees_is_not_bypassed(cuda_lib, rows):
    from torch.fx.experimental.proxy_tensor import make_fx
    from rwkv_quant_b200.backends.cuda import linear_for
    op = linear_for(_synth_linear("sb6", 4, 128, 256, seed=1))
    x = _x(rows, 256, 1)
    want = op(x)
    y = op(x.clone().requires_grad_())
    assert y.requires_grad and torch.equal(y.detach(), want)
    with pytest.raises(RuntimeError):                    # no gradient is defined: not a silent zero
        y.sum().backward()
    with torch.no_grad():
        assert not op(x.clone().requires_grad_()).requires_grad
    g = make_fx(lambda t: op(t))(x)
    assert any("rwkvq.gemv" in str(n.target) for n in g.graph.nodes)
    assert torch.equal(g(x), want)
    other = _x(rows, 256, 2)
    assert torch.equal(g(other), op(other))
    with pytest.raises(Exception):
        torch.func.jvp(op, (x,), (x,))


@pytest.mark.parametrize("rows", [1, 3, 200])
def test_cuda_rows_on_host_weights_are_refused(cuda_lib, rows):
    from rwkv_quant_b200.backends.cuda import linear_for
    op = linear_for(_synth_linear("sb6", 4, 128, 256, seed=1), "cpu")
    with pytest.raises(RuntimeError, match="CUDA tensors only"):
        op(_x(rows, 256, 1))


@pytest.mark.parametrize("B,T", [(1, 2), (1, 5), (1, 40), (5, 20)])      # every kind of head and of layer linear
def test_a_time_out_is_kept_until_it_is_asked_for(cuda_lib, B, T):
    """The kernels set one word of the model's by compare-and-swap; no later launch or call clears it."""
    from rwkv_quant_b200 import _lib
    model = _model()
    idx, st = _idx(B, T), _states(model, B)
    model.forward_stateful(idx, st)
    model.check()
    model._status.fill_(-9)                                       # as a kernel whose wait ran out leaves it
    model.forward_stateful(idx, st)
    with pytest.raises(_lib.RwkvqError, match="kernel status"):
        model.check()
    model.check()


def test_a_time_out_of_a_large_step_is_kept(cuda_lib):
    """More streams than the small-batch kernels take: the linears report to the step's own word."""
    from rwkv_quant_b200 import _lib
    model = _model()
    dec = model.decoder(260, use_graph=False)
    dec._ws[0][:4].view(torch.int32).fill_(-9)
    dec.step(torch.ones(260, dtype=torch.long, device="cuda"))
    with pytest.raises(_lib.RwkvqError, match="kernel status"):
        dec.check()


@pytest.mark.parametrize("B", [2, 13])
def test_an_error_behind_the_fork_joins_the_side_stream(cuda_lib, B):
    """A tensor of the last layer is refused when that layer is reached: what ran on the side stream until then must be
    ordered before the caller's later work (memory goes back to the allocator in that order).  Under capture an open
    side stream is an error of its own."""
    from rwkv_quant_b200 import _lib
    model = _model()
    dec = model.decoder(B, use_graph=False)
    dec.step(torch.ones(B, dtype=torch.long, device="cuda"))
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        dec.step(torch.ones(B, dtype=torch.long, device="cuda"))          # the stream has its side stream now
        torch.cuda.synchronize()
        layer = model._layers_c[1]
        codes = layer.w2.codes                                             # looked at behind the launch of r / k / v beside it
        graph = torch.cuda.CUDAGraph()
        graph.capture_begin()
        try:
            layer.w2.codes = None
            with pytest.raises(_lib.RwkvqError, match="null"):
                dec._run()
        finally:
            layer.w2.codes = codes
            graph.capture_end()
    torch.cuda.synchronize()
    ref = model.decoder(B, use_graph=False)
    dec = model.decoder(B)
    tok = torch.arange(1, B + 1, device="cuda")
    assert torch.equal(ref.step(tok), dec.step(tok))


@pytest.mark.parametrize("B", [1, 2, 9])
@pytest.mark.parametrize("name,field,value", [("w1", "gs", 0), ("g2", "rows", -4), ("Wk", "cols", 0)])
def test_a_tensor_that_a_later_layer_refuses_is_not_asked_for_before(cuda_lib, B, name, field, value):
    """The launches of a layer ask L2 for the tensors of the layer behind it, by their shapes and block sizes: descriptors that are
    refused at their turn must not be used (a block size of 0 divided, negative sizes reached beyond every buffer)."""
    from rwkv_quant_b200 import _lib
    model = _model()
    tok = torch.arange(1, B + 1, device="cuda")
    want = model.decoder(B, use_graph=False).step(tok).clone()
    dec = model.decoder(B, use_graph=False)
    t = getattr(model._layers_c[1], name)
    keep = getattr(t, field)
    try:
        setattr(t, field, value)
        with pytest.raises(_lib.RwkvqError):
            dec.step(tok)
    finally:
        setattr(t, field, keep)
    assert torch.equal(model.decoder(B, use_graph=False).step(tok), want)


@pytest.mark.parametrize("D", [128, 512, 768, 1024, 1280, 1536, 2048, 2304, 2560, 3072, 3584, 4096])
@pytest.mark.parametrize("N", [24, 49, 50, 199, 444, 1024])
def test_row_preparation_in_every_form(cuda_lib, D, N):
    """Widths and token counts on each side of the lines between the scalar, vector and group forms; the three row forms of a
    mix agree with the fp64 LayerNorm, shift and lerp: fp32 rows to rounding, pairs to 2^-20, scaled fp16 to half an ulp of 2^-10."""
    from rwkv_quant_b200.backends.cuda import ops
    gen = torch.Generator(device="cuda").manual_seed(D + N)
    draw = lambda *s: torch.randn(s, generator=gen, device="cuda")
    x, w, b, shift = draw(2, N // 2, D), draw(D), draw(D), draw(2, 1, D)
    xn = torch.nn.functional.layer_norm(x.double(), (D,), w.double(), b.double())
    prev = torch.cat([shift.double(), xn[:, :-1]], 1)
    for modes in ([1, 2, 4, 7, 2, 2], [7]):
        mix = draw(len(modes), D)
        rows, new = ops.seq_ln_shift_mix_prep(x, w, b, shift, mix, modes)
        assert relmax(new.cpu().numpy(), xn[:, -1:].cpu().numpy()) <= 2e-6
        for m, r in enumerate(rows):
            want = (xn + (prev - xn) * mix[m].double()).reshape(-1, D)
            top = want.abs().amax(1, keepdim=True)
            if r.f32 is not None:
                assert relmax(r.f32.cpu().numpy(), want.cpu().numpy()) <= 2e-6
            if r.split is not None:
                assert ((r.split[:, :D].double() + r.split[:, D:].double() - want).abs() <= top * 2.0 ** -20).all()
            if r.x16 is not None:
                got = r.x16[:, :D].double() / r.scale[:, None].double()
                assert ((got - want).abs() <= want.abs() * 2.0 ** -11 + top * 2.0 ** -20).all()
                assert (r.scale[:, None] * top <= 2.0 ** 14).all()


def test_two_streams_keep_their_precision_with_single_term_operands(cuda_lib):
    """RWKVQ_BATCH_FAST=1 (here by the library's profiling switch) selects single fp16 operands from three streams on."""
    import ctypes as C
    model = _model(n_embd=512, ffn=2048)
    hook = cuda_lib.rwkvq_profiling_batch_fast
    hook.restype, hook.argtypes = None, [C.c_int]
    out = {}
    try:
        for fast in (0, 1):
            hook(fast)
            for B in (2, 3):
                dec = model.decoder(B, states=_states(model, B), use_graph=False)
                dec.step(torch.arange(1, B + 1, device="cuda"))
                out[fast, B] = dec.logits.cpu().numpy()
    finally:
        hook(-1)
    assert relmax(out[1, 2], out[0, 2]) <= 2e-5
    assert relmax(out[1, 3], out[0, 3]) > 5e-5                    # the switch was on
