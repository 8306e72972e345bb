"""The one-call sequence forward and the one-stream decode step where their splits can go wrong: rows on each side of the
small-batch, tcgen05 and fp16-GEMM ranges, tokens on each side of the shortest chunked call and of a chunk of 8, heads on
each side of a half and a whole wave (one form of the scan each), and widths with a ragged last group of the LoRA and
LayerNorm threads.  Reference: the CPU oracle for the calls, the package's per-operator path for the steps.

Tolerances (of the largest value): calls of up to 64 rows and single steps are fp32 grade, some 1e-6 a linear and 2e-5
through two layers: 1e-4, a third of what one dropped half of an operand pair costs; longer calls have fp16 operands,
2^-11 a value and some 5e-4 through two layers: 1e-3."""
import hashlib

import pytest
import torch

from helpers import relmax

pytestmark = pytest.mark.gpu


def _checkpoint(recipe, **dims):
    from rwkv_quant_b200 import synth
    return synth.build_checkpoint(dict(n_layer=2, vocab=512, **dims), recipe, seed=3, device="cuda", keep_on_device=False)


def _model(recipe, **dims):
    from rwkv_quant_b200.backends.cuda import QuantRWKV7
    return QuantRWKV7(_checkpoint(recipe, **dims), device="cuda")


def _states(model, B):
    gen = torch.Generator(device="cuda").manual_seed(B)
    D, H = model.n_embd, model.n_head
    draw = lambda *shape: 0.2 * torch.randn(shape, generator=gen, device="cuda")
    return [(draw(B, H, 64, 64), draw(B, 1, D), draw(B, 1, D)) for _ in range(model.n_layer)]


def _same(a, b, tol):
    n = lambda t: t.cpu().numpy() if isinstance(t, torch.Tensor) else t
    assert relmax(n(a[0]), n(b[0])) <= tol
    for sa, sb in zip(a[1], b[1]):
        for x, y in zip(sa, sb):
            assert relmax(n(x), n(y).reshape(tuple(x.shape))) <= tol


@pytest.mark.parametrize("recipe", ["compression", "reduction"])
def test_forward_calls_match_the_oracle(cuda_lib, tmp_path, recipe):
    from oracle import codec_np as oc
    from oracle.model_np import OracleRWKV7
    from rwkv_quant_b200.backends.cuda import QuantRWKV7
    from rwkv_quant_b200.formats import save_rwkvq
    ck = _checkpoint(recipe, n_embd=256, ffn=1024)
    save_rwkvq(ck, str(tmp_path / "m.rwkvq"))
    model, oracle = QuantRWKV7(ck, device="cuda"), OracleRWKV7(*oc.open_rwkvq(str(tmp_path / "m.rwkvq")))
    for B, T in [(1, 2), (1, 16), (1, 17), (2, 32), (1, 65), (5, 15), (5, 16), (4, 17), (3, 23), (3, 24), (3, 25), (3, 31), (19, 15),
                 (18, 17), (19, 17), (37, 33), (38, 33), (400, 3), (401, 3)]:
        idx = torch.randint(1, 512, (B, T), generator=torch.Generator().manual_seed(B * 100 + T))
        st = _states(model, B)
        got = model.forward_stateful(idx.cuda(), st)
        model.check()
        ref = oracle.forward_stateful(idx.numpy(), [tuple(t.cpu().numpy() for t in s) for s in st])
        _same(got, ref, 1e-4 if B * T <= 64 else 1e-3)


def test_hidden_rows_far_below_their_bound(cuda_lib):
    """The channel mix of long calls scales its fp16 hidden rows by a bound on |W||x| instead of by their own maximum.  One row
    of W 2^9 times the others: tokens whose product with it is negative keep hidden rows some 2^11 below the bound (2^22
    squared), and lose nothing against the per-operator path, which scales by the maximum."""
    ck = _checkpoint("compression", n_embd=256, ffn=1024)
    for layer in (0, 1):
        t = ck.tensors[f"blocks.{layer}.ffn.key.weight"]
        t.gw_d[7] *= 2.0 ** 9
        t.gw_dm[7] *= 2.0 ** 9
    from rwkv_quant_b200.backends.cuda import QuantRWKV7
    model = QuantRWKV7(ck, device="cuda")
    idx = torch.randint(1, 512, (3, 40), generator=torch.Generator().manual_seed(1)).cuda()
    got, _ = model.forward_stateful(idx, _states(model, 3))
    model.fused_prep = False
    ref, _ = model.forward_stateful(idx, _states(model, 3))
    err = (got - ref).abs().amax(-1) / ref.abs().amax(-1)
    assert err.max() <= 2e-3 and err.median() <= 1e-3, (err.max(), err.median())


@pytest.mark.parametrize("recipe,D,F", [("compression", 256, 1024), ("reduction", 1280, 8192), ("compression_eh8", 2560, 10240),
                                        ("compression", 3328, 4096)])
def test_one_stream_steps_match_the_sequence(cuda_lib, recipe, D, F):
    model = _model(recipe, n_embd=D, ffn=F)
    idx = torch.randint(1, 512, (1, 9), generator=torch.Generator().manual_seed(D)).cuda()
    st = _states(model, 1)
    dec = model.decoder(1, states=[tuple(t.clone() for t in s) for s in st])
    steps = []
    for t in range(9):
        dec.step(idx[:, t])
        steps.append(dec.logits.clone())
    model.fused_prep = False
    ref, _ = model.forward_stateful(idx, st)
    assert relmax(torch.stack(steps, 1).cpu().numpy(), ref.cpu().numpy()) <= 1e-4


@pytest.mark.parametrize("B,T", [(1, 31), (1, 33), (1, 48), (1, 49), (1, 64), (2, 32), (20, 3)])
def test_time_mix_of_short_sequences_matches_its_steps(cuda_lib, B, T):
    """Chunks of 16 tokens, whole and ragged, against the step's kernel token by token; fresh and carried states."""
    model = _model("reduction", n_embd=256, ffn=1024)
    idx = torch.randint(1, 512, (B, T), generator=torch.Generator().manual_seed(T)).cuda()
    for st in (_states(model, B), model.init_state(B)):
        got = model.forward_stateful(idx, [tuple(t if t is None else t.clone() for t in s) for s in st])
        rows = []
        for t in range(T):
            lo, st = model.forward_stateful(idx[:, t:t + 1], st)
            rows.append(lo)
        _same(got, (torch.cat(rows, 1), st), 1e-4)


@pytest.mark.parametrize("recipe,D,B,T", [("compression", 256, 2, 3), ("compression", 768, 3, 3), ("reduction", 256, 16, 3),
                                          ("compression", 256, 17, 3), ("reduction", 768, 21, 3), ("compression", 2304, 37, 1),
                                          ("compression", 2304, 38, 1), ("reduction", 4096, 40, 1), ("compression", 256, 46, 1),
                                          # each side of the line from which a CTA normalises a token for all its mixes
                                          ("compression", 2048, 74, 1), ("compression", 2048, 75, 1), ("reduction", 2304, 75, 2),
                                          ("reduction", 2560, 37, 1), ("reduction", 2560, 38, 1)])
def test_steps_of_several_streams_match_the_sequence(cuda_lib, recipe, D, B, T):
    """The time mix and the LayerNorms of a step against the per-operator path (a few streams at a time: above 64 rows its linears have fp16
    operands): logits and all states after T tokens."""
    model = _model(recipe, n_embd=D, ffn=1024)
    idx = torch.randint(1, 512, (B, T), generator=torch.Generator().manual_seed(B)).cuda()
    st = _states(model, B)
    dec = model.decoder(B, states=[tuple(t.clone() for t in s) for s in st])
    steps = []
    for t in range(T):
        dec.step(idx[:, t])
        steps.append(dec.logits.clone())
    model.fused_prep = False
    few = 64 // T
    ref = [model.forward_stateful(idx[i:i + few], [tuple(t[i:i + few] for t in s) for s in st]) for i in range(0, B, few)]
    states = [tuple(torch.cat([r[1][l][k] for r in ref]) for k in range(3)) for l in range(model.n_layer)]
    _same((torch.stack(steps, 1), dec.states), (torch.cat([r[0] for r in ref]), states), 1e-4)


@pytest.mark.parametrize("B,T", [(1, 255), (1, 256), (2, 300), (37, 256), (38, 256)])
def test_weights_converted_beside_the_scan(cuda_lib, B, T):
    """Calls on each side of the lines from which the weights become fp16 on the side stream, against the per-operator path; a
    second call over the first one's buffers; and as a graph, whose forks are those of the captured stream."""
    model = _model("compression", n_embd=256, ffn=1024)
    idx = torch.randint(1, 512, (B, T), generator=torch.Generator().manual_seed(T)).cuda()
    model.fused_prep = False
    ref = model.forward_stateful(idx, _states(model, B), last_only=True)
    model.fused_prep = True
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        for _ in range(2):
            got = model.forward_stateful(idx, _states(model, B), last_only=True)
        stream.synchronize()
        _same(got, ref, 1e-3)
        st, g = _states(model, B), torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream):
            got = model.forward_stateful(idx, st, last_only=True)
        for _ in range(2):
            g.replay()
        stream.synchronize()
        _same(got, ref, 1e-3)
    model.check()


def _digest(D, recipe, B, T):
    model = _model(recipe, n_embd=D, ffn=4 * D)
    idx = torch.randint(1, 512, (B, T), generator=torch.Generator().manual_seed(T)).cuda()
    logits, states = model.forward_stateful(idx, _states(model, B), last_only=True)
    h = hashlib.sha256()
    for t in [logits] + [t for s in states for t in s]:
        h.update(t.contiguous().cpu().numpy().tobytes())
    return h.hexdigest()[:16]


LONG_CALLS = {
    (256, "reduction", 1, 300): "e1976a99397ced6b",
    (768, "reduction", 2, 77): "a0ec36bbdb59f446",
    (1024, "compression", 1, 256): "6a474cfdfd7c0077",
    (256, "compression", 5, 17): "9acecb7f95e80476",
}


@pytest.mark.parametrize("D,recipe,B,T", list(LONG_CALLS))
def test_long_calls_of_few_heads_keep_their_bits(cuda_lib, D, recipe, B, T):
    """Sums of the group norm in another order move fp16 roundings of the rows behind it: 7e-4 of the logits through 24 layers, where a
    call repeats itself exactly.  Digests of the seeded builds as first recorded; a change of them has to be meant."""
    assert _digest(D, recipe, B, T) == LONG_CALLS[D, recipe, B, T]
