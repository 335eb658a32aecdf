"""The give-up path of the bounded waits, run once in the allowed form.

Every wait inside the tcgen05 kernels is bounded: when the bound is hit the kernel records a status word, raises a CTA-wide
flag that makes all later waits fall through, and runs to its normal teardown (named barriers, TMEM release).  Nothing in
normal operation makes a wait run out, so a TEST-ONLY build of the library (tests/_build/libfat_b200_waittest.so, made by
`python -m fastalgebraictransformer_b200.build`; the package never loads it) compiles the attention forward with a
producer that leaves out one V tile and with waits that give up after ~3 ms.  One single-CTA launch of it must return by
itself with the status word set; an ordinary launch of the shipped library right after must be correct, which also shows
that the tensor memory of the SM was released.  No trap, no faulting access, no unbounded loop is involved.
"""
import ctypes
import math
import os

import pytest
import torch

from conftest import ROOT, bf16_violations
from oracle import oracle

pytestmark = pytest.mark.gpu
LIB = os.path.join(ROOT, "tests", "_build", "libfat_b200_waittest.so")


def test_a_wait_that_runs_out_ends_in_a_status_word_and_a_usable_gpu():
    if not os.path.exists(LIB):
        pytest.skip("tests/_build/libfat_b200_waittest.so has not been built")
    import fastalgebraictransformer_b200 as fat
    from fastalgebraictransformer_b200 import _lib
    dev = torch.device("cuda", 0)
    B, H, T, D = 1, 1, 128, 64
    g = torch.Generator().manual_seed(71)
    q, k, v, go = (torch.randn(B, H, T, D, generator=g).to(torch.bfloat16) for _ in range(4))
    slopes = oracle.compute_alibi_slopes(H)
    qd, kd, vd, sd = (t.to(dev) for t in (q, k, v, slopes))
    out = torch.empty_like(qd)
    out_lo = torch.empty_like(qd)
    L = torch.empty(B, H, T, dtype=torch.float32, device=dev)
    status = torch.zeros(1, dtype=torch.int32, device=dev)

    test_lib = ctypes.CDLL(LIB)                                # its own handle: the symbols stay local to it
    fn = test_lib.fat_attn_fwd
    fn.restype, fn.argtypes = _lib.PROTOTYPES["fat_attn_fwd"]
    rc = fn(qd.data_ptr(), kd.data_ptr(), vd.data_ptr(), sd.data_ptr(), out.data_ptr(), out_lo.data_ptr(), L.data_ptr(),
            B, H, T, D, _lib.strides3(qd), _lib.strides3(kd), _lib.strides3(vd), _lib.strides3(out), 1.0 / math.sqrt(D), 1e-6,
            1, _lib.BF16, _lib.PATH_TENSOR, status.data_ptr(), _lib.stream_ptr(dev))
    assert rc == 0
    torch.cuda.synchronize()                                   # returns: the kernel ended by itself
    word = int(status.item())
    assert (word >> 24) & 0x1f == 1, f"status word 0x{word:08x}: expected the wait-timeout code"
    assert word & 0xffffff in (22, 23, 30, 31, 40, 10, 11), f"status word 0x{word:08x}: unexpected wait site"

    # the shipped library on the same GPU, right after: correct results (and no kernel stuck waiting for tensor memory)
    leaves = [t.to(dev).requires_grad_(True) for t in (q, k, v)]
    res = fat.rational_attention(*leaves, sd, 1.0 / math.sqrt(D))
    res.backward(go.to(dev))
    fat.check_device_status()
    want = oracle.rational_attention_grads(q.float(), k.float(), v.float(), go.float(), slopes, 1.0 / math.sqrt(D))
    for got, w in zip((res, leaves[0].grad, leaves[1].grad, leaves[2].grad), want):
        bad, _ = bf16_violations(got.float(), w)
        assert bad == 0.0


def test_a_copy_that_never_arrives_ends_in_nan_losses_and_a_usable_gpu():
    """The staged loss kernel: in the test build the first block never requests the copy of its fifth row.  The wait for
    it runs out (~3 ms), the block marks its rows with NaN losses, every block returns, and the shipped library gives the
    right loss on the same GPU right after."""
    if not os.path.exists(LIB):
        pytest.skip("tests/_build/libfat_b200_waittest.so has not been built")
    import fastalgebraictransformer_b200 as fat
    from fastalgebraictransformer_b200 import _lib
    dev = torch.device("cuda", 0)
    n_sm = torch.cuda.get_device_properties(dev).multi_processor_count
    B, T, V = 4, 2 * n_sm, 4096                                # 8 rows per block: enough for the staged kernel, and for row 4 of block 0
    g = torch.Generator().manual_seed(5)
    logits = torch.randn(B, T, V, generator=g).to(torch.bfloat16)
    labels = torch.randint(0, V, (B, T), generator=g)
    ld, lab = logits.to(dev), labels.to(dev)
    n_valid = torch.tensor([float(B * (T - 1))], device=dev)
    row_loss = torch.zeros(B * T, device=dev)
    d_logits = torch.empty_like(ld)

    test_lib = ctypes.CDLL(LIB)
    fn = test_lib.fat_shifted_ce_fwd
    fn.restype, fn.argtypes = _lib.PROTOTYPES["fat_shifted_ce_fwd"]
    rc = fn(ld.data_ptr(), lab.data_ptr(), n_valid.data_ptr(), row_loss.data_ptr(), d_logits.data_ptr(), B, T, V, ld.stride(0), ld.stride(1),
            lab.stride(0), lab.stride(1), -100, _lib.BF16, _lib.stream_ptr(dev))
    assert rc == 0
    torch.cuda.synchronize()                                   # returns: every block ended by itself
    bad = torch.isnan(row_loss)
    mine = torch.arange(B * T, device=dev) % n_sm == 0         # the rows of block 0
    assert bad[mine].all() and not bad[~mine].any()

    want = oracle.shifted_cross_entropy(logits.float(), labels)
    got = fat.shifted_cross_entropy(ld, lab)
    assert abs(got.item() - want.item()) < 4e-2               # (the loss comes back in the logits' dtype: bfloat16 near 8.8 has steps of 0.06)


class LmLayer(ctypes.Structure):
    _fields_ = [(n, ctypes.c_void_p) for n in ("norm1", "qkv", "out", "norm2", "gate_val", "down", "k_cache", "v_cache", "slopes")]


def _lm_step(lib, model, cache, ids, workspace, lengths, logits, status):
    """fat_lm_decode_step of `lib` on a model's parameters and a cache."""
    from fastalgebraictransformer_b200 import _lib
    fn = lib.fat_lm_decode_step
    fn.restype, fn.argtypes = _lib.PROTOTYPES["fat_lm_decode_step"]
    layers = (LmLayer * len(model.blocks))()
    for i, b in enumerate(model.blocks):
        layers[i] = LmLayer(*[t.data_ptr() for t in (b.norm1.weight, b.attn.qkv.weight, b.attn.out.weight, b.norm2.weight, b.ffn.w_gate_val.weight,
                                                     b.ffn.w_out.weight, cache.k[i], cache.v[i], b.attn.alibi_slopes)])
    B, H, capacity, D = cache.k[0].shape
    w = model.head.weight
    return fn(ctypes.addressof(layers), len(model.blocks), ids.data_ptr(), ids.stride(0), model.embed.weight.data_ptr(), model.norm.weight.data_ptr(),
              w.data_ptr(), logits.data_ptr(), lengths.data_ptr(), _lib.strides3(cache.k[0]), int(model.blocks[0].attn.alibi_slopes.dtype == torch.float32),
              workspace.data_ptr(), workspace.numel(), B, w.shape[1], H, D, model.blocks[0].ffn.w_out.weight.shape[1], w.shape[0], capacity, D ** -0.5,
              1e-6, 1e-6, _lib.BF16, status.data_ptr(), _lib.stream_ptr(w.device))


def _lm_case(B=2, n=9, vocab=300):
    import fastalgebraictransformer_b200 as fat
    torch.manual_seed(9)
    model = fat.AlgebraicTransformerLM(vocab_size=vocab, d_model=256, n_head=4, n_layers=3, dropout=0.0, block_size=64).to("cuda").to(torch.bfloat16).eval()
    ids = torch.randint(0, vocab, (B, n), device="cuda")
    cache = model.new_cache(B, n)
    model.forward_cached(ids[:, :n - 1].contiguous(), cache)
    w = model.head.weight
    nbytes = torch.ops.algebraic.lm_decode_workspace_bytes(B, 256, 4, 64, model.blocks[0].ffn.w_out.weight.shape[1], vocab, 3, n, w.dtype)
    return model, cache, ids[:, n - 1:].contiguous(), torch.zeros(nbytes, dtype=torch.uint8, device="cuda")


@pytest.mark.parametrize("vocab", [300, 301])
def test_words_that_never_arrive_end_in_nan_logits_and_a_usable_step(vocab):
    """The decode step of the language model: in the test build one unit of the first projection is never handed on.  The CTAs
    that need it give up after ~3 ms, all return, the logits are NaN, no length moves; the shipped library then takes the same
    step in the same workspace and gives the module-by-module logits.  With a vocabulary of 301 the computing warps of the test build
    wait for none of their weights either, so that they are done while copies are on their way: the loading warp waits for those."""
    if not os.path.exists(LIB):
        pytest.skip("tests/_build/libfat_b200_waittest.so has not been built")
    from fastalgebraictransformer_b200 import _lib
    model, cache, ids, workspace = _lm_case(vocab=vocab)
    logits = torch.zeros(2, vocab, dtype=torch.bfloat16, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    lengths = cache.lengths.clone()
    assert _lm_step(ctypes.CDLL(LIB), model, cache, ids, workspace, lengths, logits, status) == 0
    torch.cuda.synchronize()
    assert (status.item() >> 24) & 0xf == 1 and status.item() & 0xffffff == 300, f"status word 0x{status.item():08x}"
    assert torch.isnan(logits).all()
    assert torch.equal(lengths, cache.lengths)
    assert workspace[12].item() == 1                                           # what generate looks at before it samples

    status.zero_()
    assert _lm_step(_lib.lib(), model, cache, ids, workspace, lengths, logits, status) == 0
    torch.cuda.synchronize()
    assert status.item() == 0 and lengths.tolist() == [9, 9]
    cache.step = False
    want = model.forward_cached(ids, cache)
    assert ((logits.float() - want.float()).abs().max() / want.float().abs().max()).item() < 4 * 2.0 ** -8      # (as the fused step's tests)


def test_a_sequence_without_room_keeps_its_length():
    from fastalgebraictransformer_b200 import _lib
    model, cache, ids, workspace = _lm_case()
    lengths = torch.tensor([8, 9], dtype=torch.int32, device="cuda")           # the second sequence's cache is full
    logits = torch.zeros(2, 300, dtype=torch.bfloat16, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    for t in cache.k + cache.v:
        t[:, :, 8] = 0.0
    before = [t.clone() for t in cache.k + cache.v]
    assert _lm_step(_lib.lib(), model, cache, ids, workspace, lengths, logits, status) == 0
    torch.cuda.synchronize()
    assert status.item() == 0x10000000 and lengths.tolist() == [9, 9]
    assert torch.isfinite(logits).all()
    for t, b in zip(cache.k + cache.v, before):
        assert torch.equal(t[1], b[1]) and not torch.equal(t[0, :, 8], b[0, :, 8])


def test_generate_reports_a_step_that_gave_up():
    """The status word is read once at the end; another report in it is left for check_device_status."""
    import fastalgebraictransformer_b200 as fat
    from fastalgebraictransformer_b200 import _lib
    model, _, ids, _ = _lm_case()
    word = _lib.device_status(torch.device("cuda", 0))
    word.fill_(1 << 24 | 300)
    with pytest.raises(RuntimeError, match="ran out"):
        model.generate(ids, 4, top_k=1)
    assert word.item() == 0
    word.fill_(0x10000000)
    assert model.generate(ids, 4, top_k=1).shape == (2, 5)
    with pytest.raises(RuntimeError, match="without room"):
        fat.check_device_status()


@pytest.mark.parametrize("gave_up", [True, False])
def test_generate_does_not_sample_from_a_step_that_gave_up(gave_up, monkeypatch):
    """NaN probabilities are a device assert in multinomial, so a given-up step's logits are replaced before it; a model's own
    NaN are not.  (The step and multinomial are stand-ins here: no NaN reaches the sampler whatever generate does.)"""
    from fastalgebraictransformer_b200.algebraic_model import _DecodeStep
    model, _, ids, _ = _lm_case()
    seen = []

    def step(self, input_ids, cache):
        self.rest[0][12] = int(gave_up)
        return torch.full((2, 300), float("nan"), dtype=torch.bfloat16, device="cuda")

    def multinomial(probs, num_samples):
        seen.append(bool(torch.isfinite(probs).all()))
        return torch.zeros(2, 1, dtype=torch.int64, device="cuda")

    monkeypatch.setattr(_DecodeStep, "__call__", step)
    monkeypatch.setattr(torch, "multinomial", multinomial)
    model.generate(ids, 4, top_k=1)
    assert seen == [True] + [gave_up] * 3
