"""Decode step over a key/value cache (fat_attn_decode) and the cached ``generate`` (B200).

The reference has no cache: its generate() re-runs forward() over the whole prefix for every token
(algebraic_model.py:239-265).  The pin is therefore the causal attention itself: the decode step of the token at position
n must equal row n of the oracle's causal attention over the n+1 tokens, and the cached model must give the logits the
full forward gives at the same position.
"""
import ctypes
import os

import pytest
import torch

from conftest import bf16_violations, norm_max_err
from oracle import oracle

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _case(dtype, B, H, D, capacity, lengths, seed):
    g = torch.Generator().manual_seed(seed)
    q = torch.randn(B, H, D, generator=g).to(dtype)
    k_new = torch.randn(B, H, D, generator=g).to(dtype)
    v_new = torch.randn(B, H, D, generator=g).to(dtype)
    kc = torch.randn(B, H, capacity, D, generator=g).to(dtype)
    vc = torch.randn(B, H, capacity, D, generator=g).to(dtype)
    for b, n in enumerate(lengths):                 # rows that are not part of the sequence must never be read
        kc[b, :, n:] = float("nan")
        vc[b, :, n:] = float("nan")
    return q, k_new, v_new, kc, vc


def _oracle_rows(q, k_new, v_new, kc, vc, lengths, slopes, scale):
    rows = []
    for b, n in enumerate(lengths):
        k = torch.cat((kc[b, :, :n].float(), k_new[b].float()[:, None]), 1)[None]        # [1,H,n+1,D]
        v = torch.cat((vc[b, :, :n].float(), v_new[b].float()[:, None]), 1)[None]
        rows.append(oracle.rational_attention_last_row(q[b].float()[None], k, v, slopes, scale)[0])
    return torch.stack(rows)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,H,D,capacity,lengths", [
    (2, 4, 64, 300, (0, 299)),                      # an empty cache and one that the new row fills
    (3, 12, 64, 1024, (17, 511, 1000)),             # the small model's heads (non-power-of-two slopes)
    (2, 2, 128, 4096, (4095, 2500)),                # few (batch, head) pairs: the key range is split over 8 CTAs
    (1, 16, 128, 2048, (1234,)),                    # the XL model's heads
    (2, 3, 32, 96, (5, 64)),
])
def test_decode_step_equals_last_row_of_causal_attention(dtype, B, H, D, capacity, lengths):
    from fastalgebraictransformer_b200 import ops
    slopes = oracle.compute_alibi_slopes(H)
    scale = D ** -0.5
    q, k_new, v_new, kc, vc = _case(dtype, B, H, D, capacity, lengths, 7 + D + B)
    want = _oracle_rows(q, k_new, v_new, kc, vc, lengths, slopes, scale)
    kc_d, vc_d = kc.to(DEV), vc.to(DEV)
    n_cached = torch.tensor(lengths, dtype=torch.int32, device=DEV)
    got = ops.attn_decode(q.to(DEV), k_new.to(DEV), v_new.to(DEV), kc_d, vc_d, n_cached, slopes.to(DEV), scale, 1e-6)
    if dtype == torch.float32:
        assert norm_max_err(got, want) < 1e-5
    else:
        bad, _ = bf16_violations(got, want)
        assert bad == 0.0                            # every element inside |a-b| <= 1e-2 + 2e-2|b|
    for b, n in enumerate(lengths):                  # the new rows were appended, nothing else moved
        assert torch.equal(kc_d[b, :, n].cpu(), k_new[b]) and torch.equal(vc_d[b, :, n].cpu(), v_new[b])
        assert torch.equal(kc_d[b, :, :n].cpu(), kc[b, :, :n]) and torch.equal(vc_d[b, :, :n].cpu(), vc[b, :, :n])
        assert torch.isnan(kc_d[b, :, n + 1:]).all() and torch.isnan(vc_d[b, :, n + 1:]).all()
    # same arguments, same bits
    kc2, vc2 = kc.to(DEV), vc.to(DEV)
    again = ops.attn_decode(q.to(DEV), k_new.to(DEV), v_new.to(DEV), kc2, vc2, n_cached, slopes.to(DEV), scale, 1e-6)
    assert torch.equal(got, again)


def test_decode_reads_strided_views_of_the_packed_projection():
    """q, k_new, v_new as the model passes them: slices of one [B, 1, 3, H, D] projection output."""
    from fastalgebraictransformer_b200 import ops
    B, H, D, cap, n = 2, 4, 64, 128, 40
    g = torch.Generator().manual_seed(3)
    qkv = torch.randn(B, 1, 3, H, D, generator=g).to(torch.bfloat16)
    kc = torch.randn(B, H, cap, D, generator=g).to(torch.bfloat16)
    vc = torch.randn(B, H, cap, D, generator=g).to(torch.bfloat16)
    slopes = oracle.compute_alibi_slopes(H)
    want = _oracle_rows(qkv[:, 0, 0], qkv[:, 0, 1], qkv[:, 0, 2], kc, vc, (n, n), slopes, 0.125)
    qkv_d = qkv.to(DEV)
    got = ops.attn_decode(qkv_d[:, 0, 0], qkv_d[:, 0, 1], qkv_d[:, 0, 2], kc.to(DEV), vc.to(DEV),
                          torch.full((B,), n, dtype=torch.int32, device=DEV), slopes.to(DEV), 0.125, 1e-6)
    assert bf16_violations(got, want)[0] == 0.0


def test_decode_reports_a_full_cache_through_the_c_abi():
    """A sequence whose cache has no room gets zeros, nothing is written, and the status word says so."""
    from fastalgebraictransformer_b200 import _lib
    lib = _lib.lib()
    B, H, D, cap = 2, 2, 64, 16
    q = torch.randn(B, H, D, device=DEV)
    kc = torch.randn(B, H, cap, D, device=DEV)
    vc = torch.randn(B, H, cap, D, device=DEV)
    kc0, vc0 = kc.clone(), vc.clone()
    out = torch.full((B, H, D), 7.0, device=DEV)
    n_cached = torch.tensor([3, cap], dtype=torch.int32, device=DEV)      # the second sequence is full
    slopes = oracle.compute_alibi_slopes(H).to(DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    s2 = (ctypes.c_int64 * 2)(H * D, D)
    s3 = (ctypes.c_int64 * 3)(H * cap * D, cap * D, D)
    rc = lib.fat_attn_decode(q.data_ptr(), q.data_ptr(), q.data_ptr(), kc.data_ptr(), vc.data_ptr(), n_cached.data_ptr(),
                             slopes.data_ptr(), out.data_ptr(), B, H, cap, D, s2, s2, s2, s2, s3, s3, 0.125, 1e-6, _lib.F32,
                             status.data_ptr(), _lib.stream_ptr(q.device))
    assert rc == 0, lib.fat_last_error().decode()
    torch.cuda.synchronize()
    assert status.item() == 0x10000000
    assert torch.all(out[1] == 0) and torch.isfinite(out[0]).all() and not torch.all(out[0] == 0)
    assert torch.equal(kc[1], kc0[1]) and torch.equal(vc[1], vc0[1])
    assert torch.equal(kc[0, :, 3], q[0])                                 # the other sequence was served normally
    # refused on the host: a head size without a kernel, misaligned rows
    rc = lib.fat_attn_decode(q.data_ptr(), q.data_ptr(), q.data_ptr(), kc.data_ptr(), vc.data_ptr(), n_cached.data_ptr(),
                             slopes.data_ptr(), out.data_ptr(), B, H, cap, 48, s2, s2, s2, s2, s3, s3, 0.125, 1e-6, _lib.F32,
                             status.data_ptr(), None)
    assert rc == 3
    rc = lib.fat_attn_decode(q.data_ptr() + 4, q.data_ptr(), q.data_ptr(), kc.data_ptr(), vc.data_ptr(), n_cached.data_ptr(),
                             slopes.data_ptr(), out.data_ptr(), B, H, cap, D, s2, s2, s2, s2, s3, s3, 0.125, 1e-6, _lib.F32,
                             status.data_ptr(), None)
    assert rc == 4


def _tiny(dtype, d_model=64, n_head=2, n_layers=2, vocab=128, block_size=64):
    from fastalgebraictransformer_b200 import AlgebraicTransformerLM
    torch.manual_seed(11)
    model = AlgebraicTransformerLM(vocab_size=vocab, d_model=d_model, n_head=n_head, n_layers=n_layers, dropout=0.0,
                                   block_size=block_size)
    return model.to(DEV).to(dtype).eval()


@pytest.mark.parametrize("dtype,d_model,n_head", [(torch.float32, 64, 2), (torch.bfloat16, 256, 4), (torch.bfloat16, 256, 2)])
def test_cached_steps_give_the_logits_of_the_full_forward(dtype, d_model, n_head):
    """Prompt of 20 tokens, then 12 tokens one at a time: at every step the cached logits are the full forward's."""
    from fastalgebraictransformer_b200 import AlgebraicTransformerLM
    torch.manual_seed(11)
    model = AlgebraicTransformerLM(vocab_size=512, d_model=d_model, n_head=n_head, n_layers=2, dropout=0.0, block_size=64)
    ids = torch.randint(0, 512, (3, 32))
    # the pin: the reference's forward as the oracle restates it, in float32 on the (rounded) weights
    state = {k: v.detach().to(dtype).float() for k, v in model.state_dict().items()
             if k != "embed.weight" and not k.endswith("alibi_slopes")}
    want, _ = oracle.lm_forward(state, ids, n_head)
    model = model.to(DEV).to(dtype).eval()
    ids = ids.to(DEV)
    with torch.no_grad():
        full, _ = model(ids)
        cache = model.new_cache(3, 32)
        got = [model.forward_cached(ids[:, :20], cache)]
        for t in range(20, 32):
            got.append(model.forward_cached(ids[:, t:t + 1], cache))
    assert cache.seen == 32 and cache.lengths.tolist() == [32, 32, 32]
    # float32: the bar of the other float32 tests.  bfloat16: two layers of 16-bit operators and GEMMs in a row; the cached
    # steps must be as close to the float32 oracle as the full forward is (normalised error, like the model-level 16-bit test)
    tol = 1e-5 if dtype == torch.float32 else 3e-2
    assert norm_max_err(full[:, 19:], want[:, 19:]) < tol
    for i, t in enumerate(range(19, 32)):
        assert norm_max_err(got[i], want[:, t]) < tol, t
        if dtype == torch.float32:
            assert norm_max_err(got[i], full[:, t]) < 1e-5, t


def test_generate_with_cache_equals_the_reference_loop():
    """Greedy sampling (top_k=1 leaves one candidate) through the cache and through the reference's recompute loop."""
    model = _tiny(torch.float32, block_size=48)
    prompt = torch.randint(0, 128, (2, 9), device=DEV)
    a = model.generate(prompt.clone(), 24, top_k=1, use_cache=True)                      # decode steps replayed from a CUDA graph
    b = model.generate(prompt.clone(), 24, top_k=1, use_cache=False)
    e = model.generate(prompt.clone(), 24, top_k=1, use_cache=True, cuda_graph=False)    # every decode step launch by launch
    assert a.shape == (2, 33) and torch.equal(a, b) and torch.equal(e, b)
    fat_status = __import__("fastalgebraictransformer_b200").check_device_status
    fat_status()                                                                         # no cache overflow was reported
    # a run that would outgrow block_size falls back to the reference's loop (the window slides, positions shift)
    c = model.generate(prompt.clone(), 48, top_k=1, use_cache=True)
    d = model.generate(prompt.clone(), 48, top_k=1, use_cache=False)
    assert c.shape == (2, 57) and torch.equal(c, d)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_decode_first_token_of_an_empty_cache(dtype):
    """n_cached = 0 everywhere and a cache of one row: the token attends to itself only, out = v * f / (f + eps)."""
    from fastalgebraictransformer_b200 import ops
    B, H, D = 2, 3, 32
    g = torch.Generator().manual_seed(2)
    q, k_new, v_new = (torch.randn(B, H, D, generator=g).to(dtype) for _ in range(3))
    kc = torch.full((B, H, 1, D), float("nan"), dtype=dtype)
    vc = torch.full((B, H, 1, D), float("nan"), dtype=dtype)
    slopes = oracle.compute_alibi_slopes(H)
    want = oracle.rational_attention_last_row(q.float(), k_new.float()[:, :, None], v_new.float()[:, :, None], slopes, 0.2)
    kd, vd = kc.to(DEV), vc.to(DEV)
    got = ops.attn_decode(q.to(DEV), k_new.to(DEV), v_new.to(DEV), kd, vd, torch.zeros(B, dtype=torch.int32, device=DEV),
                          slopes.to(DEV), 0.2, 1e-6)
    if dtype == torch.float32:
        assert norm_max_err(got, want) < 1e-5
    else:
        assert bf16_violations(got, want)[0] == 0.0
    assert torch.equal(kd[:, :, 0].cpu(), k_new) and torch.equal(vd[:, :, 0].cpu(), v_new)


@pytest.mark.parametrize("dtype,d_model,n_head,d_ffn,vocab,B,prompt", [
    (torch.bfloat16, 256, 4, None, 1000, 8, 70),        # d_ffn 682: rows of the down projection only 4-byte aligned; keys shared by CTAs
    (torch.bfloat16, 512, 8, None, 509, 1, 300),        # d_ffn 1365: 2-byte aligned, ragged last units; many key shares
    (torch.float16, 768, 6, 2048, 1000, 9, 40),         # nine tokens: the second half of the MMA rows; heads of 128
    (torch.bfloat16, 768, 12, 2048, 777, 16, 33),       # more (batch, head) pairs than SMs
    (torch.float16, 64, 1, 40, 64, 2, 1),               # less than one unit per warp group
])
def test_fused_decode_step_equals_the_modules_and_the_oracle(dtype, d_model, n_head, d_ffn, vocab, B, prompt):
    """The whole step as one launch: logits, caches and lengths against the module-by-module step on the same caches, and
    the logits against the float32 oracle of the full forward."""
    from fastalgebraictransformer_b200 import AlgebraicTransformerLM, check_device_status
    torch.manual_seed(19)
    model = AlgebraicTransformerLM(vocab_size=vocab, d_model=d_model, n_head=n_head, n_layers=2, d_ffn=d_ffn, dropout=0.0, block_size=512)
    n = prompt + 4
    ids = torch.randint(0, vocab, (B, n))
    state = {k: v.detach().to(dtype).float() for k, v in model.state_dict().items() if k != "embed.weight" and not k.endswith("alibi_slopes")}
    want, _ = oracle.lm_forward(state, ids, n_head)
    model, ids = model.to(DEV).to(dtype).eval(), ids.to(DEV)
    caches, logits = [model.new_cache(B, n) for _ in range(2)], []
    for fused, cache in enumerate(caches):
        model.forward_cached(ids[:, :prompt], cache)
        if not fused:
            cache.step = False                          # module by module
        logits.append([model.forward_cached(ids[:, t:t + 1], cache) for t in range(prompt, n)])
    assert caches[1].step and not caches[0].step
    check_device_status()
    assert caches[1].lengths.tolist() == [n] * B and caches[1].seen == n
    # the two round at the same places and differ in the order of float32 sums: now and then a 16-bit rounding falls to the
    # other side (2^-9 or 2^-11 of one element), which two layers turn into a few times that of the largest logit
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    for a, b in zip(*logits):
        assert norm_max_err(b, a) < 4 * eps
    for t, got in enumerate(logits[1]):
        assert norm_max_err(got, want[:, prompt + t]) < 3e-2
    for side in ("k", "v"):
        for a, b in zip(getattr(caches[0], side), getattr(caches[1], side)):
            assert norm_max_err(b, a) < 4 * eps


def _both_ways(model, ids, prompt):
    """Logits of the steps after the prompt and the caches, operator by operator and as one launch."""
    B, n = ids.shape
    caches, logits = [model.new_cache(B, n) for _ in range(2)], []
    for fused, cache in enumerate(caches):
        model.forward_cached(ids[:, :prompt], cache)
        if not fused:
            cache.step = False
        logits.append([model.forward_cached(ids[:, t:t + 1], cache) for t in range(prompt, n)])
    assert caches[1].step and not caches[0].step
    return caches, logits


# more blocks than there are word buffers (two, used in turn).  The keys of a (batch, head) pair whole and shared out; heads of 128
# for up to eight sequences; 16 sequences at width 1024, which leave room for a ring of two chunks
@pytest.mark.parametrize("dtype,d_model,n_head,n_layers,vocab,B,prompt", [
    (torch.bfloat16, 768, 12, 5, 1000, 8, 150), (torch.bfloat16, 512, 8, 12, 509, 1, 300), (torch.float16, 768, 6, 3, 500, 4, 90),
    (torch.bfloat16, 1024, 16, 3, 300, 16, 40), (torch.float16, 512, 4, 4, 200, 3, 33),
])
def test_fused_decode_step_of_many_blocks(dtype, d_model, n_head, n_layers, vocab, B, prompt):
    """Two 16-bit evaluations drift apart with depth, so each is held against the 64-bit one: the fused step may be no further
    off than the operators are, up to the scatter of such errors (2-norms over thousands of elements: 3-4 % here, 15 % allowed)."""
    from fastalgebraictransformer_b200 import AlgebraicTransformerLM, check_device_status
    torch.manual_seed(23)
    model = AlgebraicTransformerLM(vocab_size=vocab, d_model=d_model, n_head=n_head, n_layers=n_layers, dropout=0.0, block_size=512)
    ids = torch.randint(0, vocab, (B, prompt + 6))
    state = {k: v.detach().to(dtype).double() for k, v in model.state_dict().items() if k != "embed.weight" and not k.endswith("alibi_slopes")}
    exact, _ = oracle.lm_forward(state, ids, n_head)
    model, ids = model.to(DEV).to(dtype).eval(), ids.to(DEV)
    caches, logits = _both_ways(model, ids, prompt)
    check_device_status()
    exact = exact[:, prompt:]
    off = [((torch.stack(x, 1).double().cpu() - exact).norm() / exact.norm()).item() for x in logits]
    assert off[1] < 1.15 * off[0], f"{off[1]:.5f} from the exact logits, the operators {off[0]:.5f}"
    assert off[0] < 3e-2
    for side in ("k", "v"):
        for a, b in zip(*(getattr(c, side) for c in caches)):
            assert norm_max_err(b, a) < 3e-2


# a chunk of the ring: 256 (heads of 64) or 128 (of 128) cached rows, 1024 or 2048 elements of weight rows
@pytest.mark.parametrize("dtype,d_model,n_head,d_ffn,vocab,B,prompt,strided", [
    (torch.bfloat16, 768, 12, 1000, 640, 8, 254, False),     # the last rows of a chunk and the first of the next; down rows end inside a block of 32
    (torch.float16, 768, 6, 2730, 320, 13, 126, True),       # two chunks of down rows off 16-byte boundaries; cached rows apart in memory
    (torch.bfloat16, 1280, 10, 2048, 200, 2, 17, False),     # a width that is not compiled in, two chunks per row
    (torch.bfloat16, 320, 5, 2049, 333, 16, 15, True),       # odd rows, two chunks; act rows with a word to spare
    (torch.float16, 512, 4, 2056, 64, 1, 513, False),        # one chunk and eight elements; shares of the keys
    (torch.bfloat16, 512, 8, 1000, 64, 8, 1789, False),      # cached rows go round the ring; the last chunk is not whole
    (torch.bfloat16, 512, 8, 1000, 64, 8, 1789, True),       # and fetched row by row
    (torch.float16, 768, 6, 1000, 64, 2, 1789, True),
])
def test_fused_decode_step_at_the_edges_of_chunks(dtype, d_model, n_head, d_ffn, vocab, B, prompt, strided):
    """Against the operators, on the same bound as above (two blocks: a rounding that tips moves a few 16-bit steps)."""
    from fastalgebraictransformer_b200 import AlgebraicTransformerLM, check_device_status
    torch.manual_seed(29)
    model = AlgebraicTransformerLM(vocab_size=vocab, d_model=d_model, n_head=n_head, n_layers=2, d_ffn=d_ffn, dropout=0.0, block_size=2048)
    model, ids = model.to(DEV).to(dtype).eval(), torch.randint(0, vocab, (B, prompt + 5), device=DEV)
    make = model.new_cache

    def new_cache(batch, capacity):
        cache = make(batch, capacity)
        if strided:
            cache.k, cache.v = ([torch.cat([t, t], -1)[..., :t.shape[-1]] for t in side] for side in (cache.k, cache.v))
        return cache
    model.new_cache = new_cache
    caches, logits = _both_ways(model, ids, prompt)
    check_device_status()
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    for a, b in zip(*logits):
        assert norm_max_err(b, a) < 4 * eps
    for side in ("k", "v"):
        for a, b in zip(*(getattr(c, side) for c in caches)):
            assert norm_max_err(b, a) < 4 * eps


def _fill_shared(value):
    """Every 32-bit word of every SM's shared memory."""
    from fastalgebraictransformer_b200.build import FILL_SHARED_LIB
    if not os.path.exists(FILL_SHARED_LIB):
        pytest.skip("tests/_build/libfill_shared.so has not been built")
    fill = ctypes.CDLL(FILL_SHARED_LIB).test_fill_shared
    assert fill(ctypes.c_uint32(value), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0


# what the ring's stages hold where nothing is copied to: rows of the matrix beyond its last one, the ends of rows, cached rows beyond the
# last.  Odd feed-forward widths, whose last unit is in the second half of a chunk (1365) or in the first (3413, 2389), and an even one
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("d_model,n_head,d_ffn,B", [(*m, B) for m in ((512, 8, 1365), (512, 4, 1365), (768, 12, 1042)) for B in (1, 8, 16)] +
                         [(*m, B) for m in ((1280, 20, 3413), (1280, 10, 3413)) for B in (1, 8)] + [(896, 14, 2389, 16), (896, 7, 2389, 16)])
def test_fused_decode_step_uses_nothing_that_it_has_not_written(dtype, d_model, n_head, d_ffn, B):
    """Shared memory full of NaN before every step, and one sequence whose cached rows are NaN: what the others get is to the bit what
    they get from finite leftovers, and stays as close to the operators as in the tests above."""
    from fastalgebraictransformer_b200 import AlgebraicTransformerLM, check_device_status
    torch.manual_seed(31)
    model = AlgebraicTransformerLM(vocab_size=203, d_model=d_model, n_head=n_head, n_layers=2, d_ffn=d_ffn, dropout=0.0, block_size=512)
    model = model.to(DEV).to(dtype).eval()
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    for prompt in (3, 300):
        n = prompt + 3
        ids = torch.randint(0, 203, (B, n), device=DEV)
        start = model.new_cache(B, n)
        model.forward_cached(ids[:, :prompt], start)
        out = {}
        for how in ("operators", "zeros", "nan", "nan rows"):
            cache = model.new_cache(B, n)
            for mine, its in zip(cache.k + cache.v, start.k + start.v):
                mine.copy_(its)
                if how == "nan rows":
                    mine[0, :, :prompt] = float("nan")
            cache.lengths.copy_(start.lengths)
            cache.seen = start.seen
            if how == "operators":
                cache.step = False
            steps = []
            for t in range(prompt, n):
                _fill_shared(0xffffffff if how == "nan" else 0)
                steps.append(model.forward_cached(ids[:, t:t + 1], cache))
            assert (how == "operators") != bool(cache.step)
            out[how] = steps + [c[:, :, prompt:n] for c in cache.k + cache.v]
        check_device_status()
        for want, zeros, nan, rows in zip(*out.values()):
            assert norm_max_err(zeros, want) < 4 * eps
            assert torch.equal(nan, zeros)
            assert torch.equal(rows[1:], zeros[1:])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("n_head", [1, 2])
def test_fused_decode_step_rounds_where_the_operators_round(dtype, n_head):
    """Weights with one power of two per row make every contraction exact, so the order of sums does not matter and both ways
    have to agree to the bit, in every block: the residual stream, whose sums are rounded block by block, included."""
    from fastalgebraictransformer_b200 import AlgebraicTransformerLM
    torch.manual_seed(5)
    C, n_layers = 128, 6
    model = AlgebraicTransformerLM(vocab_size=96, d_model=C, n_head=n_head, n_layers=n_layers, d_ffn=192, dropout=0.0, block_size=64)
    with torch.no_grad():
        for block in model.blocks:
            for w in (block.attn.qkv.weight, block.attn.out.weight, block.ffn.w_gate_val.weight, block.ffn.w_out.weight):
                col = torch.randint(0, w.shape[1], (w.shape[0], 1))
                w.zero_().scatter_(1, col, (2.0 ** torch.randint(-2, 2, col.shape)) * (1 - 2 * torch.randint(0, 2, col.shape)))
        model.head.weight.copy_(torch.randint(1, 9, (96, C)) / 8.0 * (1 - 2 * torch.randint(0, 2, (96, C))))
    model = model.to(DEV).to(dtype).eval()
    caches, logits = _both_ways(model, torch.randint(0, 96, (3, 8), device=DEV), 1)
    for side in ("k", "v"):
        for i, (a, b) in enumerate(zip(*(getattr(c, side) for c in caches))):
            assert torch.equal(a, b), f"{side} of block {i}"
    for a, b in zip(*logits):                         # (the head's weights are dense: its sums may still round either way)
        assert norm_max_err(b, a) < (2.0 ** -7 if dtype == torch.bfloat16 else 2.0 ** -10)


def _half_model(n_layers=2, d_model=128, n_head=2, vocab=64, **kw):
    from fastalgebraictransformer_b200 import AlgebraicTransformerLM
    torch.manual_seed(3)
    kw = {"dropout": 0.0, "block_size": 64, **kw}
    return AlgebraicTransformerLM(vocab_size=vocab, d_model=d_model, n_head=n_head, n_layers=n_layers, **kw).to(DEV).to(torch.bfloat16).eval()


@pytest.mark.parametrize("what", ["ids", "lengths", "workspace", "slopes", "k", "v", "workspace dtype", "lengths dtype"])
def test_decode_step_operator_refuses_tensors_from_elsewhere(what):
    """Every tensor of the step has to be on the model's GPU (here: one on the host); refused before anything is launched."""
    model = _half_model()
    cache = model.new_cache(2, 12)
    ids = torch.randint(0, 64, (2, 5), device=DEV)
    model.forward_cached(ids[:, :4], cache)
    model.forward_cached(ids[:, 4:], cache)
    blocks = model.blocks
    args = dict(ids=ids[:, :1], embed=model.embed.weight, norm=model.norm.weight, head=model.head.weight,
                params=[w for b in blocks for w in (b.norm1.weight, b.attn.qkv.weight, b.attn.out.weight, b.norm2.weight, b.ffn.w_gate_val.weight, b.ffn.w_out.weight)],
                slopes=[b.attn.alibi_slopes for b in blocks], k=list(cache.k), v=list(cache.v), lengths=cache.lengths.clone(),
                workspace=torch.zeros(1 << 20, dtype=torch.uint8, device=DEV))
    step = lambda: torch.ops.algebraic.lm_decode_step(*args.values(), 0.125, 1e-6, 1e-6)          # noqa: E731
    assert step().shape == (2, 64)
    torch.cuda.synchronize()
    if what.endswith("dtype"):
        name = what.split()[0]
        args[name] = args[name].to(torch.int64)
    elif isinstance(args[what], list):
        args[what][1] = args[what][1].cpu()
    else:
        args[what] = args[what].cpu()
    with pytest.raises(RuntimeError, match="model's GPU"):
        step()


def _unaligned(t):
    """The same values in memory that starts two bytes after a 16-byte boundary."""
    return torch.empty(t.numel() + 8, dtype=t.dtype, device=t.device)[1:t.numel() + 1].view(t.shape).copy_(t)


@pytest.mark.parametrize("late", [False, True])
@pytest.mark.parametrize("what", ["embedding rows", "embedding rows fewer", "parameter", "head", "slopes dtype", "cache layout", "cache alignment"])
def test_what_the_fused_step_does_not_take_runs_module_by_module(what, late):
    """Models and caches that the operators take and the single launch does not: same result as without it, whether they
    differ from the start or (late) come to differ after the first fused step."""
    results = []
    for fused in (False, True):
        model = _half_model(vocab=64)
        cache = model.new_cache(2, 16)
        ids = torch.randint(0, 60, (2, 9), generator=torch.Generator().manual_seed(4)).to(DEV)
        model.forward_cached(ids[:, :4], cache)
        if late:
            if fused:
                model.forward_cached(ids[:, 4:5], cache)
                assert cache.step
            else:                                    # (the same rows in the cache as the fused step leaves)
                model.forward_cached(ids[:, 4:5], cache)
        cache.step = None if fused else False
        with torch.no_grad():
            if what.startswith("embedding"):
                rows = 60 if what.endswith("fewer") else 80
                model.embed = torch.nn.Embedding(rows, 128).to(DEV).to(torch.bfloat16)
                model.embed.weight.copy_(torch.randn(rows, 128, generator=torch.Generator().manual_seed(6)))
            elif what == "parameter":
                w = model.blocks[1].ffn.w_out.weight
                w.data = _unaligned(w)
            elif what == "head":
                model.head.weight.data = _unaligned(model.head.weight)
            elif what == "slopes dtype":
                model.blocks[1].attn.alibi_slopes = model.blocks[1].attn.alibi_slopes.double()
            elif what == "cache layout":
                cache.k[1] = cache.k[1].permute(0, 2, 1, 3).contiguous().permute(0, 2, 1, 3)
            else:                                    # rows of 8 extra elements: aligned, but not alike
                cache.v[0] = torch.cat((cache.v[0], cache.v[0][..., :8]), -1)[..., :64]
        results.append([model.forward_cached(ids[:, t:t + 1], cache) for t in range(5 if late else 4, 9)] + [cache.lengths, *cache.k, *cache.v])
        assert not cache.step
    for got, want in zip(*results):
        assert torch.equal(got[..., :9, :] if got.dim() == 4 else got, want[..., :9, :] if want.dim() == 4 else want)


@pytest.mark.parametrize("B,new,fused", [(2, 12, True), (1, 12, False), (9, 12, False), (1, 4, True)])
def test_generate_replays_the_faster_way(B, new, fused, monkeypatch):
    """A captured step is the single launch only where its replay wins (width 768: up to 8 sequences; width 128: more than one); a
    few tokens are stepped without a capture, where it always does."""
    from fastalgebraictransformer_b200.algebraic_model import _DecodeStep
    calls, stock = [], _DecodeStep.__call__
    monkeypatch.setattr(_DecodeStep, "__call__", lambda self, *a: calls.append(1) or stock(self, *a))
    model = _half_model(d_model=768, n_head=12) if B == 9 else _half_model()
    prompt = torch.randint(0, 64, (B, 7), device=DEV)
    assert model.generate(prompt, new, top_k=1).shape == (B, 7 + new)
    assert bool(calls) == fused


@pytest.mark.parametrize("new", [3, 12])
def test_generate_inside_a_callers_capture(new, monkeypatch):
    """A caller may capture the whole call (no capture of its own then): nothing of generate's own waits for the GPU (the sampler is
    a stand-in, since torch may check its probabilities on the host)."""
    monkeypatch.setattr(torch, "multinomial", lambda probs, num_samples: probs.argmax(-1, keepdim=True))
    model = _half_model()
    prompt = torch.randint(0, 64, (2, 7), device=DEV)
    want = model.generate(prompt, new, cuda_graph=False)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = model.generate(prompt, new, cuda_graph=False)
    for _ in range(2):
        got.zero_()
        graph.replay()
        assert torch.equal(got, want)


def test_workspace_outlives_its_last_launch_on_another_stream():
    """A step dropped while its launch still waits on a side stream: its workspace must not be handed out again yet."""
    model = _half_model()
    cache = model.new_cache(2, 12)
    ids = torch.randint(0, 64, (2, 8), device=DEV)
    model.forward_cached(ids[:, :4], cache)
    model.forward_cached(ids[:, 4:5], cache)
    address, nbytes = cache.step.rest[0].data_ptr(), cache.step.rest[0].numel()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        torch.cuda._sleep(100_000_000)               # about 50 ms
        model.forward_cached(ids[:, 5:6], cache)
    cache.step = None
    taken = [torch.empty(nbytes, dtype=torch.uint8, device=DEV) for _ in range(4)]
    still_waiting = not side.query()
    assert still_waiting and address not in [t.data_ptr() for t in taken]
    torch.cuda.current_stream().wait_stream(side)


def test_fused_decode_step_yields_to_hooks_and_replaced_modules():
    from fastalgebraictransformer_b200 import AlgebraicTransformerLM
    torch.manual_seed(3)
    model = AlgebraicTransformerLM(vocab_size=64, d_model=128, n_head=2, n_layers=2, dropout=0.0, block_size=64).to(DEV).to(torch.bfloat16).eval()
    ids = torch.randint(0, 64, (2, 12), device=DEV)
    cache = model.new_cache(2, 12)
    model.forward_cached(ids[:, :4], cache)
    model.forward_cached(ids[:, 4:5], cache)
    assert cache.step
    calls = []
    handle = model.blocks[1].attn.qkv.register_forward_hook(lambda *a: calls.append(1))
    model.forward_cached(ids[:, 5:6], cache)
    assert calls == [1]
    handle.remove()
    model.blocks[0].ffn.w_out = torch.nn.Sequential(model.blocks[0].ffn.w_out)
    model.forward_cached(ids[:, 6:7], cache)
    assert cache.step is False and cache.lengths.tolist() == [7, 7] and cache.seen == 7
