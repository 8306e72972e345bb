"""The workloads this package's speed is judged on, as data and as calls of its public entry points.

A case is a dict of plain values; its ``path`` says which entry point it calls:

  decode    ``QuantRWKV7.decoder(B).step(tokens)``: one token for each of B concurrent streams, the
            serving loop (one stream: an interactive session)
  prefill   ``QuantRWKV7.forward_stateful(prompts [B, T], fresh states, last_only=True)``: prompts in,
            first logits and carried states out, the states written into a server's pool
  verify    ``QuantRWKV7.forward_stateful(drafts [1, T], states, tail_only=T)``: a speculative-decoding
            round, which keeps the old states until the drafts are accepted
  linear    one operator call of ``linear_for(tensor)``: what a program with its own model code uses
  quantize  ``quantize_sb6`` / ``quantize_sym``: packing one weight matrix of a checkpoint

Models are seeded random-init builds in the recipes and dimensions of ``rwkv_quant_b200.synth`` at full
depth: throughput does not depend on the weights' values.
"""
from __future__ import annotations

import math

import torch

from rwkv_quant_b200 import quantize as q
from rwkv_quant_b200 import synth
from rwkv_quant_b200.backends.cuda import QuantRWKV7, linear_for

# matrices of the two model sizes, [OUT, IN]: projections, channel-mix key and value, head
_SHAPES = [(d, d) for d in (2048, 2560)] + [(4 * d, d) for d in (2048, 2560)] + [(d, 4 * d) for d in (2048, 2560)]
_LAYOUTS = [("sb6", 4), ("sb6", 5), ("sb6", 6), ("sym", 6), ("sym", 8), ("rtn", 8)]


def listed():
    return [
        # one vector through one projection: an operator call is a few microseconds, mostly overhead
        dict(name="linear_1row", path="linear", layout="sb6", bits=5, out=2048, inp=2048, rows=1, dtype="bf16"),
        # a prompt chunk through a channel-mix value matrix, on the tensor-core side of the operator
        dict(name="linear_300rows", path="linear", layout="sym", bits=6, out=2048, inp=8192, rows=300, dtype="fp32"),
        # interactive decoding: one stream, both model sizes, both recipes
        dict(name="decode_1", path="decode", model="1.5b", recipe="compression", batch=1),
        dict(name="decode_1_large", path="decode", model="2.9b", recipe="reduction", batch=1),
        # a lightly loaded server: an odd number of streams
        dict(name="decode_13", path="decode", model="1.5b", recipe="reduction", batch=13),
        # the benchmark's serving load, and one beyond it
        dict(name="decode_64", path="decode", model="1.5b", recipe="compression", batch=64),
        dict(name="decode_100", path="decode", model="1.5b", recipe="compression_eh8", batch=100),
        # a pending token and four drafts
        dict(name="verify_5", path="verify", model="1.5b", recipe="compression", tokens=5),
        # prompts: the benchmark's pp512 alone and sixteen at once, and a few short ones of a ragged length
        dict(name="prefill_1x512", path="prefill", model="1.5b", recipe="reduction", batch=1, tokens=512),
        dict(name="prefill_3x77", path="prefill", model="1.5b", recipe="compression", batch=3, tokens=77),
        dict(name="prefill_16x512", path="prefill", model="1.5b", recipe="reduction", batch=16, tokens=512),
        # packing the largest matrix of a layer with the scale search
        dict(name="quantize_key", path="quantize", layout="sb6", bits=4, out=10240, inp=2560),
    ]


def draw(rng):
    """One more case of the same ranges."""
    def log_int(lo, hi):
        return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))

    path = rng.choice(["decode", "decode", "decode", "prefill", "prefill", "verify", "linear", "linear", "quantize"])
    if path == "linear":
        layout, bits = rng.choice(_LAYOUTS)
        out, inp = rng.choice(_SHAPES)
        return dict(path=path, layout=layout, bits=bits, out=out, inp=inp, rows=log_int(1, 1024),
                    dtype=rng.choice(["fp32", "fp16", "bf16"]))
    if path == "quantize":
        layout, bits = rng.choice([("sb6", 4), ("sb6", 5), ("sb6", 6), ("sym", 6), ("sym", 8)])
        return dict(path=path, layout=layout, bits=bits, out=log_int(512, 10240), inp=256 * rng.randint(4, 40))
    model = rng.choice(["1.5b", "1.5b", "2.9b"])
    recipe = rng.choice(["compression", "reduction", "compression_eh8"])
    if path == "decode":
        return dict(path=path, model=model, recipe=recipe, batch=log_int(1, 128))
    if path == "verify":
        return dict(path=path, model=model, recipe=recipe, tokens=rng.randint(2, 16))
    batch = log_int(1, 16)
    most = (8192 if model == "1.5b" else 4096) // batch
    return dict(path=path, model=model, recipe=recipe, batch=batch, tokens=log_int(17, min(1024, most)))


# ------------------------------------------------------------------------------------------- states

_DTYPES = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16}


def _pool(model, batch):
    """State storage of a server for ``batch`` streams: all layers' WKV states and shift rows."""
    L, H, S, D = model.n_layer, model.n_head, model.head_size, model.n_embd
    e = lambda *s: torch.zeros(s, device=model.device)
    return e(L, batch, H, S, S), e(L, batch, 1, D), e(L, batch, 1, D)


def _carried(pool, gen):
    """States as they stand in the middle of a text: WKV entries of a few tenths, normalised rows."""
    for t, std in zip(pool, (0.1, 1.0, 1.0)):
        t.normal_(0.0, std, generator=gen)
    return [tuple(t[i] for t in pool) for i in range(pool[0].shape[0])]


def prepare(case, seed):
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    if case["path"] in ("linear", "quantize"):
        w = torch.randn(case["out"], case["inp"], generator=gen, device=dev) * 0.02
        if case["path"] == "quantize":
            return dict(case=case, w=w)
        x = torch.randn(case["rows"], case["inp"], generator=gen, device=dev)
        if case["inp"] > case["out"]:                   # a channel-mix value matrix reads relu(.)^2
            x = torch.relu(x) ** 2
        qt = getattr(synth, "quant_" + case["layout"])("w", "proj", w, case["bits"])
        return dict(case=case, op=linear_for(qt, dev), x=x.to(_DTYPES[case["dtype"]]))

    model = QuantRWKV7(synth.build_checkpoint(case["model"], case["recipe"], seed=seed, device=dev), device=dev)
    batch, tokens = case.get("batch", 1), case.get("tokens", 1)
    idx = torch.randint(1, model.vocab_size, (batch, tokens), generator=gen, device=dev)
    pool = _pool(model, batch)
    if case["path"] == "prefill":
        return dict(case=case, model=model, idx=idx, pool=pool)
    states = _carried(pool, gen)
    if case["path"] == "verify":
        return dict(case=case, model=model, idx=idx, states=states, accepted=_pool(model, batch))
    return dict(case=case, dec=model.decoder(batch, states=states), idx=idx[:, 0].contiguous(), pool=pool)


def _store(states, pool):
    for k, t in enumerate(pool):
        torch.stack([st[k] for st in states], out=t)
    return pool


def run(state):
    case = state["case"]
    path = case["path"]
    if path == "decode":
        dec = state["dec"]
        nxt = dec.step(state["idx"])                    # states advance in place
        # the logits, the score of each greedy token (what a server reports beside it) and the states
        return dec.logits, dec.logits.gather(1, nxt[:, None]), state["pool"]
    if path == "prefill":
        m = state["model"]
        logits, states = m.forward_stateful(state["idx"], m.init_state(case["batch"]), last_only=True)
        return logits, _store(states, state["pool"])
    if path == "verify":
        logits, states = state["model"].forward_stateful(state["idx"], state["states"], tail_only=case["tokens"])
        return logits, _store(states, state["accepted"])
    if path == "linear":
        return state["op"](state["x"])
    if case["layout"] == "sb6":
        t = q.quantize_sb6("w", "proj", state["w"], case["bits"])
    else:
        t = q.quantize_sym("w", "proj", state["w"], case["bits"])
    bufs = (t.codes, t.codes_packed, t.gw_qh, t.gw_qh2, t.gw_qsqm, t.gw_qs, t.gw_d, t.gw_dm)
    return [b for b in bufs if b is not None]


# ------------------------------------------------------------------------------------------- floors

def _bytes_per_weight(layout, bits):
    """File-format bytes: codes, and block scales of half a bit (sb6) or 9/16 (sym) a weight."""
    return {"sb6": (bits + 0.5) / 8, "sym": (bits + 0.5625) / 8, "asym": 9 / 8, "rtn": bits / 8}[layout]


def _model_work(case, tokens_per_stream, head_rows):
    dims, rec = synth.MODEL_DIMS[case["model"]], synth.RECIPES[case["recipe"]]
    L, D, F, V = dims["n_layer"], dims["n_embd"], dims["ffn"], dims["vocab"]
    rk, batch = synth.lora_ranks(D), case.get("batch", 1)
    n = batch * tokens_per_stream
    groups = [("proj", 4 * D * D), ("cmix", 2 * D * F), ("wav_lora", 2 * D * (rk["w"] + rk["a"])), ("g_lora", 2 * D * rk["g"])]
    layers = [(g, L * k) for g, k in groups] + [("wav_lora", (L - 1) * 2 * D * rk["v"])]
    weights = sum(_bytes_per_weight(*rec[g]) * k for g, k in layers) + _bytes_per_weight(*rec["head"]) * V * D
    embedding = _bytes_per_weight(*rec["emb"]) * min(n, V) * D
    state = 4 * L * batch * (D * 64 + 2 * D)
    read = 1 if case["path"] == "prefill" else 2         # fresh states are not read
    wkv = 10 * 64 * D * L                                # S a, decay, two rank-1 updates, S r
    return {"bytes": weights + embedding + read * state + 4 * head_rows * V,
            "flops": 2 * n * sum(k for _, k in layers) + 2 * head_rows * V * D + n * wkv}


def work(case):
    path = case["path"]
    if path == "decode":
        return _model_work(case, 1, case["batch"])
    if path == "prefill":
        return _model_work(case, case["tokens"], case["batch"])
    if path == "verify":
        return _model_work(case, case["tokens"], case["tokens"])
    n = case["out"] * case["inp"]
    packed = _bytes_per_weight(case["layout"], case["bits"]) * n
    if path == "quantize":
        # the search visits 8 (sb6) or 19 (sym) scales, each some ten operations a weight
        return {"bytes": 4 * n + packed, "flops": (80 if case["layout"] == "sb6" else 190) * n}
    size = 4 if case["dtype"] == "fp32" else 2
    return {"bytes": packed + case["rows"] * (size * case["inp"] + 4 * case["out"]), "flops": 2 * case["rows"] * n}


def tolerance(case):
    path = case["path"]
    if path == "quantize":
        # a quotient on a rounding boundary may fall either way: sums run in no fixed order
        return {"rel": 1e-3, "differ": 1e-4}
    if path == "linear":
        # below 128 rows fp32-grade sums, from 128 rows on fp16 operands
        return {"rel": 1e-5 if case["rows"] < 128 else 5e-4}
    # up to 64 rows fp32-grade linears through all layers; longer calls have fp16 operands in every one
    rows = case.get("batch", 1) * case.get("tokens", 1)
    return {"rel": 1e-4} if path == "decode" or rows <= 64 else {"rel": 3e-3}
