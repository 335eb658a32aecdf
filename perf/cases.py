"""Performance cases of the Algebraic Transformer hot path: what users of this package run, through its public entry points.

``listed()`` names a dozen cases, ``draw(rng)`` gives further ones of the same ranges.  A case is a dict of plain values;
``prepare(case, seed)`` makes what a program holds before the call (inputs, parameters, caches), ``run(state)`` makes one
pass, ``work(case)`` says what that pass cannot do without and ``tolerance(case)`` how far two correct implementations at
the same precision may be apart.

Ranges
  attention    [B, H, T, D] with 1-16 sequences, 2-24 heads, 64-8192 tokens, D in {64, 128}; bfloat16, float16 (tensor
               cores) and float32 (smaller problems); forward + backward, or the forward alone without gradients;
               with and without a padding mask
  decode       one new token per sequence over a key/value cache of 64-8192 tokens, B*H from 4 to 256 pairs
  fused ops    16-16384 rows of 48-8192 columns, odd ones among them; bfloat16, float16, float32; forward + backward
  model        training steps of 128-8192 tokens (forward, loss, backward), and prompts of 16-1000 tokens followed by
               cached decode steps, d_model 512-1024, bfloat16
"""
import math

import torch

import fastalgebraictransformer_b200 as fat
from fastalgebraictransformer_b200 import ops

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
BYTES = {"bf16": 2, "fp16": 2, "fp32": 4}
DEVICE = "cuda"


def listed():
    return [
        # training attention at the size the benchmark quotes: long sequences, wide heads
        dict(name="attn_train_bf16_8x16x4096x128", kind="attn", grad=True, dtype="bf16", B=8, H=16, T=4096, D=128, mask=False),
        # float32 training of a small model's attention (research runs, gradient checks): twelve heads of 64, 512 tokens
        dict(name="attn_train_fp32_2x12x512x64", kind="attn", grad=True, dtype="fp32", B=2, H=12, T=512, D=64, mask=False),
        # a float16 batch of sequences of unequal length, right-padded to an odd length
        dict(name="attn_train_padded_fp16_4x12x777x64", kind="attn", grad=True, dtype="fp16", B=4, H=12, T=777, D=64, mask=True),
        # scoring or prompt processing of a single sequence, no gradients
        dict(name="attn_prefill_bf16_1x16x2000x128", kind="attn", grad=False, dtype="bf16", B=1, H=16, T=2000, D=128, mask=False),
        # one generation step's attention over long key/value caches
        dict(name="attn_decode_bf16_8x16x4096x128", kind="decode", dtype="bf16", B=8, H=16, T=4096, D=128),
        # the smallest call: residual addition + norm of a short sequence, where the fixed cost per call is everything
        dict(name="add_norm_bf16_64x768", kind="add_norm", dtype="bf16", rows=64, cols=768),
        # normalisation of a large batch at a large model's width
        dict(name="norm_bf16_16384x4096", kind="norm", dtype="bf16", rows=16384, cols=4096),
        # activation of a large feed-forward layer
        dict(name="swiglu_bf16_16384x8192", kind="swiglu", dtype="bf16", rows=16384, cols=8192, packed=False),
        # the medium model's activation: halves of a packed projection whose width (8/3 of 1024) is no multiple of 8
        dict(name="swiglu_packed_bf16_8192x2730", kind="swiglu", dtype="bf16", rows=8192, cols=2730, packed=True),
        # row softmax of square score matrices
        dict(name="softmax_bf16_4096x4096", kind="softmax", dtype="bf16", rows=4096, cols=4096),
        # a training step's forward, loss and backward: the small model's width, vocabulary and batch, eight layers
        dict(name="lm_train_bf16_8x1024", kind="lm_train", d_model=768, n_head=12, n_layers=8, vocab=32000, B=8, T=1024),
        # text generation with the small model: a prompt, then one cached step per token (the tokens are given, so that
        # the logits do not depend on a sampler)
        dict(name="lm_decode_bf16_8x512_32", kind="lm_decode", d_model=768, n_head=12, n_layers=12, vocab=32000, B=8, T=512, steps=32),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _columns(rng):
    """Row widths: mostly what models use (multiples of 64 or 8), some arbitrary."""
    n = _log_int(rng, 48, 8192)
    step = rng.choice([64, 64, 8, 1])
    return max(48, n // step * step)


def draw(rng):
    kind = rng.choice(["attn", "attn", "attn", "prefill", "decode", "add_norm", "norm", "swiglu", "softmax", "lm_train", "lm_decode"])
    if kind in ("attn", "prefill"):
        dtype = rng.choice(["bf16", "bf16", "fp16", "fp32"]) if kind == "attn" else rng.choice(["bf16", "fp16"])
        D = rng.choice([64, 128])
        H = rng.choice([2, 4, 8, 12, 16, 24])
        B = rng.choice([1, 2, 3, 4, 8, 16])
        T = _log_int(rng, 64, 8192 if dtype != "fp32" else 1024)
        if rng.random() < 0.5:
            T = max(64, T // 64 * 64)
        pairs = 8 * 16 * 4096 ** 2 * 128 if dtype != "fp32" else 6e9         # float32 problems are kept small
        while B > 1 and B * H * T * T * D > pairs:
            B //= 2
        while B * H * T * T * D > pairs:
            T = T * 3 // 4
        return dict(kind="attn", grad=kind == "attn", dtype=dtype, B=B, H=H, T=T, D=D, mask=rng.random() < 0.25)
    if kind == "decode":
        B, H, D = rng.choice([1, 2, 3, 4, 8, 16]), rng.choice([4, 8, 12, 16]), rng.choice([64, 128])
        return dict(kind="decode", dtype=rng.choice(["bf16", "bf16", "fp16", "fp32"]), B=B, H=H, T=_log_int(rng, 64, 8192), D=D)
    if kind in ("add_norm", "norm", "swiglu", "softmax"):
        c = dict(kind=kind, dtype=rng.choice(["bf16", "bf16", "fp16", "fp32"]), rows=_log_int(rng, 16, 16384), cols=_columns(rng))
        if kind == "swiglu":
            c["packed"] = rng.random() < 0.5
        return c
    d_model, n_head = rng.choice([(512, 8), (768, 12), (768, 6), (1024, 16), (1024, 8)])
    vocab = rng.choice([1000, 8000, 32000])
    if kind == "lm_train":
        B, T = rng.choice([1, 2, 4, 8]), _log_int(rng, 128, 1024)
        return dict(kind=kind, d_model=d_model, n_head=n_head, n_layers=rng.randint(2, 4), vocab=vocab, B=B, T=T)
    return dict(kind=kind, d_model=d_model, n_head=n_head, n_layers=rng.randint(2, 8), vocab=vocab, B=rng.choice([1, 2, 4, 8]),
                T=_log_int(rng, 16, 1000), steps=rng.choice([8, 16, 32]))


# ------------------------------------------------------------------------------------------------- inputs
def _leaf(gen, *shape, dtype, std=1.0):
    return (torch.randn(*shape, generator=gen, device=DEVICE) * std).to(dtype).requires_grad_(True)


def _model(case, seed):
    torch.manual_seed(seed)
    with torch.device(DEVICE):
        model = fat.AlgebraicTransformerLM(vocab_size=case["vocab"], d_model=case["d_model"], n_head=case["n_head"],
                                           n_layers=case["n_layers"], block_size=2048, dropout=0.0)
    return model.to(torch.bfloat16)


def prepare(case, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    kind = case["kind"]
    if kind == "attn":
        B, H, T, D, dtype = case["B"], case["H"], case["T"], case["D"], DTYPES[case["dtype"]]
        q, k, v = (_leaf(gen, B, H, T, D, dtype=dtype) for _ in range(3))
        state = dict(q=q, k=k, v=v, slopes=fat.compute_alibi_slopes(H, device=q.device), scale=1.0 / math.sqrt(D), mask=None)
        if case["grad"]:
            state["d_out"] = torch.randn(B, H, T, D, generator=gen, device=DEVICE).to(dtype)
        if case["mask"]:                                  # right padding: every sequence keeps at least half of its tokens
            keep = torch.randint((T + 1) // 2, T + 1, (B, 1), generator=gen, device=DEVICE)
            state["mask"] = (torch.arange(T, device=DEVICE)[None] < keep).to(torch.int64)
        return dict(case=case, **state)
    if kind == "decode":
        B, H, T, D, dtype = case["B"], case["H"], case["T"], case["D"], DTYPES[case["dtype"]]
        new = lambda *s: torch.randn(*s, generator=gen, device=DEVICE).to(dtype)          # noqa: E731
        return dict(case=case, q=new(B, H, D), k_new=new(B, H, D), v_new=new(B, H, D), k_cache=new(B, H, T, D), v_cache=new(B, H, T, D),
                    n_cached=torch.full((B,), T - 1, dtype=torch.int32, device=DEVICE),
                    slopes=fat.compute_alibi_slopes(H, device=torch.device(DEVICE)), scale=1.0 / math.sqrt(D))
    if kind in ("add_norm", "norm", "swiglu", "softmax"):
        R, C, dtype = case["rows"], case["cols"], DTYPES[case["dtype"]]
        state = dict(case=case, d_out=torch.randn(R, C, generator=gen, device=DEVICE).to(dtype))
        if kind == "swiglu" and case["packed"]:
            state["x"] = _leaf(gen, R, 2 * C, dtype=dtype)
        else:
            state["x"] = _leaf(gen, R, C, dtype=dtype, std=2.0 if kind == "softmax" else 1.0)
        if kind == "swiglu" and not case["packed"]:
            state["value"] = _leaf(gen, R, C, dtype=dtype)
        if kind in ("add_norm", "norm"):
            w = 1.0 + 0.1 * torch.randn(C, generator=gen, device=DEVICE)
            state["weight"] = w.to(dtype).requires_grad_(True)
        if kind == "add_norm":
            state["residual"] = _leaf(gen, R, C, dtype=dtype)
            state["d_h"] = torch.randn(R, C, generator=gen, device=DEVICE).to(dtype)
        return state
    model = _model(case, seed)
    if kind == "lm_train":
        ids = torch.randint(0, case["vocab"], (case["B"], case["T"]), generator=gen, device=DEVICE)
        return dict(case=case, model=model.train(), ids=ids)
    ids = torch.randint(0, case["vocab"], (case["B"], case["T"] + case["steps"]), generator=gen, device=DEVICE)
    return dict(case=case, model=model.eval(), prompt=ids[:, :case["T"]].contiguous(), tokens=ids[:, case["T"]:].contiguous())


# ------------------------------------------------------------------------------------------------- one pass
def _grads(outs, d_outs, leaves):
    for t in leaves:
        t.grad = None
    torch.autograd.backward(outs, d_outs)
    return [t.grad for t in leaves]


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "attn":
        if not case["grad"]:
            with torch.no_grad():
                return fat.rational_attention(s["q"], s["k"], s["v"], s["slopes"], s["scale"], key_mask=s["mask"])
        out = fat.rational_attention(s["q"], s["k"], s["v"], s["slopes"], s["scale"], key_mask=s["mask"])
        return [out.detach()] + _grads((out,), (s["d_out"],), (s["q"], s["k"], s["v"]))
    if kind == "decode":
        out = ops.attn_decode(s["q"], s["k_new"], s["v_new"], s["k_cache"], s["v_cache"], s["n_cached"], s["slopes"], s["scale"], fat.EPS)
        return [out, s["k_cache"], s["v_cache"]]          # (the step appends one row to each cache)
    if kind == "add_norm":
        h, y = fat.add_mean_error_norm(s["x"], s["residual"], s["weight"])
        return [h.detach(), y.detach()] + _grads((h, y), (s["d_h"], s["d_out"]), (s["x"], s["residual"], s["weight"]))
    if kind == "norm":
        y = fat.mean_error_norm(s["x"], s["weight"])
        return [y.detach()] + _grads((y,), (s["d_out"],), (s["x"], s["weight"]))
    if kind == "softmax":
        p = fat.rational_softmax(s["x"])
        return [p.detach()] + _grads((p,), (s["d_out"],), (s["x"],))
    if kind == "swiglu":
        if case["packed"]:
            out = fat.rational_swiglu(*s["x"].chunk(2, dim=-1))
            return [out.detach()] + _grads((out,), (s["d_out"],), (s["x"],))
        out = fat.rational_swiglu(s["x"], s["value"])
        return [out.detach()] + _grads((out,), (s["d_out"],), (s["x"], s["value"]))
    model = s["model"]
    if kind == "lm_train":
        model.zero_grad(set_to_none=True)
        logits, loss = model(s["ids"], labels=s["ids"])
        loss.backward()
        return [logits.detach(), loss.detach()] + [p.grad for p in model.parameters()]
    cache = model.new_cache(case["B"], case["T"] + case["steps"])
    logits = [model.forward_cached(s["prompt"], cache)]
    for i in range(case["steps"]):
        logits.append(model.forward_cached(s["tokens"][:, i:i + 1], cache))
    return logits + cache.k + cache.v


# ------------------------------------------------------------------------------------------------- work and tolerance
def work(case):
    kind = case["kind"]
    if kind == "attn":
        n, e = case["B"] * case["H"] * case["T"] * case["D"], BYTES[case["dtype"]]
        fwd = 2.0 * n * case["T"]                         # two contractions, causal half of the score matrix
        if not case["grad"]:
            return {"bytes": 4.0 * n * e, "flops": fwd}
        return {"bytes": 8.0 * n * e, "flops": 3.5 * fwd}                    # q, k, v, d_out in; out, dq, dk, dv out
    if kind == "decode":
        n = case["B"] * case["H"] * case["T"] * case["D"]
        return {"bytes": 2.0 * n * BYTES[case["dtype"]], "flops": 4.0 * n}
    if kind in ("add_norm", "norm", "swiglu", "softmax"):
        n, e = case["rows"] * case["cols"], BYTES[case["dtype"]]
        # tensors in + out of forward and backward, each forward input counted again where the backward needs it
        passes = {"add_norm": 8, "norm": 5, "swiglu": 8, "softmax": 5}[kind]
        return {"bytes": float(passes * n * e), "flops": 30.0 * n}
    C, L, V, B, T = case["d_model"], case["n_layers"], case["vocab"], case["B"], case["T"]
    ffn = int(C * 8 / 3)
    layer = 4 * C * C + 3 * C * ffn
    params = L * layer + V * C
    attn = 2.0 * B * L * C * T * T
    if kind == "lm_train":
        flops = 6.0 * B * T * params + 3.5 * attn
        # parameters twice, gradients once; the logits written once; per layer the tensors that have to be kept for the backward
        return {"bytes": 2.0 * (3 * params + B * T * V + L * B * T * (10 * C + 3 * ffn)), "flops": flops}
    steps = case["steps"]
    cached = sum(T + i + 1 for i in range(steps))
    flops = 2.0 * B * T * L * layer + attn + 2.0 * B * steps * params + 2.0 * B * V * C + 4.0 * B * L * C * cached
    return {"bytes": 2.0 * ((steps + 1) * params + 2.0 * B * L * C * (cached + T)), "flops": flops}


def tolerance(case):
    kind = case["kind"]
    if kind.startswith("lm_"):
        return {"rel": 2e-2}                              # bfloat16 roundings that pile up over the layers
    if case["dtype"] == "fp32":
        return {"rel": 1e-5}                              # float32 sums in another order
    return {"rel": 1e-2 if case["dtype"] == "bf16" else 2e-3}
