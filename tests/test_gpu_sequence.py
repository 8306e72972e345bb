"""The one-call sequence forward and the one-stream decode step where their splits can go wrong: rows on each side of the
small-batch, tcgen05 and fp16-GEMM ranges, tokens on each side of a chunk of 16, heads on each side of a half and a whole
wave, and widths with a ragged last group of the LoRA and LayerNorm threads.  Reference: the package's own per-operator
sequence path, which the oracle tests cover."""
import pytest
import torch

from helpers import relmax

pytestmark = pytest.mark.gpu


def _model(recipe, **dims):
    from rwkv_quant_b200 import synth
    from rwkv_quant_b200.backends.cuda import QuantRWKV7
    return QuantRWKV7(synth.build_checkpoint(dict(n_layer=2, vocab=512, **dims), recipe, seed=3, device="cuda"), device="cuda")


def _states(model, B):
    gen = torch.Generator(device="cuda").manual_seed(B)
    D, H = model.n_embd, model.n_head
    draw = lambda *shape: 0.2 * torch.randn(shape, generator=gen, device="cuda")
    return [(draw(B, H, 64, 64), draw(B, 1, D), draw(B, 1, D)) for _ in range(model.n_layer)]


def _same(a, b):
    assert relmax(a[0].cpu().numpy(), b[0].cpu().numpy()) <= 1e-3
    for sa, sb in zip(a[1], b[1]):
        for x, y in zip(sa, sb):
            assert relmax(x.cpu().numpy(), y.cpu().numpy()) <= 1e-3


@pytest.mark.parametrize("recipe", ["compression", "reduction"])
@pytest.mark.parametrize("B,T", [(1, 16), (1, 17), (2, 32), (1, 65), (5, 16), (4, 17), (3, 31), (19, 15), (37, 33)])
def test_forward_call_matches_separate_passes(cuda_lib, recipe, B, T):
    model = _model(recipe, n_embd=256, ffn=1024)
    idx = torch.randint(1, 512, (B, T), generator=torch.Generator().manual_seed(B * 100 + T)).cuda()
    st = _states(model, B)
    one = model.forward_stateful(idx, st)
    model.fused_prep = False
    _same(one, model.forward_stateful(idx, st))


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
    assert relmax(torch.stack(steps, 1).cpu().numpy(), ref.cpu().numpy()) <= 1e-3
