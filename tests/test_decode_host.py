"""When a cached step may run as one launch: the host's side of the decision (no GPU: fake tensors stand for the devices)."""
import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode


class Taken(Exception):
    pass


class Step:
    """Stands for a fused step that covers whatever it is asked."""
    def stands(self, model):
        return True

    def __call__(self, ids, cache):
        raise Taken


def model_and_cache(device="cuda:0"):
    from fastalgebraictransformer_b200 import AlgebraicTransformerLM
    torch.set_default_dtype(torch.bfloat16)         # (fake parameters cannot be converted)
    try:
        with torch.device(device):
            model = AlgebraicTransformerLM(vocab_size=64, d_model=128, n_head=2, n_layers=2, dropout=0.0, block_size=64).eval()
    finally:
        torch.set_default_dtype(torch.float32)
    cache = model.new_cache(2, 12)
    cache.seen, cache.step = 4, Step()
    return model, cache


def test_ids_of_another_gpu_never_reach_the_launch():
    with FakeTensorMode():
        model, cache = model_and_cache()
        with pytest.raises(Taken):
            model.forward_cached(torch.zeros(2, 1, dtype=torch.int64, device="cuda:0"), cache)
        with pytest.raises(RuntimeError, match="cuda:1"):           # (the embedding's refusal)
            model.forward_cached(torch.zeros(2, 1, dtype=torch.int64, device="cuda:1"), cache)


def test_a_head_without_a_weight_of_its_own_is_asked_for_nothing():
    """A wrapped head (an adapter, say) makes no fused step; the cached step runs module by module."""
    with FakeTensorMode():
        model, cache = model_and_cache()
        cache.step = None
        model.head = torch.nn.Sequential(model.head)
        assert model.forward_cached(torch.zeros(2, 1, dtype=torch.int64, device="cuda:0"), cache).shape == (2, 64)
        assert cache.step is False and cache.seen == 5


@pytest.mark.parametrize("what", ["k", "v", "lengths", "slopes"])
def test_a_cache_or_slopes_of_another_gpu_make_no_fused_step(what):
    from fastalgebraictransformer_b200.algebraic_model import _DecodeStep
    with FakeTensorMode():
        model, cache = model_and_cache()
        assert _DecodeStep.make(model, cache) is not None
        if what == "lengths":
            cache.lengths = cache.lengths.to("cuda:1")
        elif what == "slopes":
            model.blocks[1].attn.alibi_slopes = model.blocks[1].attn.alibi_slopes.to("cuda:1")
        else:
            getattr(cache, what)[1] = getattr(cache, what)[1].to("cuda:1")
        assert _DecodeStep.make(model, cache) is None


def _scale(model):
    model.blocks[1].attn.scale = 0.5


def _heads(model):
    model.blocks[0].attn.n_head = 4


def _eps_of_a_block(model):
    model.blocks[0].norm2.eps = 1e-3


def _eps_of_the_last_norm(model):
    model.norm.eps = 1e-3


def _forward_of_an_instance(model):
    attn = model.blocks[1].attn
    attn.forward = lambda *a, **k: type(attn).forward(attn, *a, **k)


def _deferred_forward_of_a_block(model):
    block = model.blocks[0]
    block.forward_deferred = lambda *a, **k: type(block).forward_deferred(block, *a, **k)


def _forward_of_the_embedding(model):
    embed = model.embed
    embed.forward = lambda x: type(embed).forward(embed, x)


def _clipped_embedding(model):
    model.embed.max_norm = 1.0


CHANGES = [_scale, _heads, _eps_of_a_block, _eps_of_the_last_norm, _forward_of_an_instance, _deferred_forward_of_a_block,
           _forward_of_the_embedding, _clipped_embedding]


@pytest.mark.parametrize("change", CHANGES)
def test_a_changed_constant_or_method_ends_the_fused_step(change):
    """What the step was made of no longer holds: it must not stand, however the change came about."""
    from fastalgebraictransformer_b200.algebraic_model import _DecodeStep
    with FakeTensorMode():
        model, cache = model_and_cache()
        step = _DecodeStep.make(model, cache)
        assert step.stands(model)
        change(model)
        assert not step.stands(model)


@pytest.mark.parametrize("change", CHANGES)
def test_a_step_is_not_made_of_a_model_that_differs(change):
    from fastalgebraictransformer_b200.algebraic_model import _DecodeStep
    with FakeTensorMode():
        model, cache = model_and_cache()
        change(model)
        assert _DecodeStep.make(model, cache) is None           # (scale and eps: one value for all blocks and norms)


def test_a_method_replaced_on_the_class_ends_the_fused_step(monkeypatch):
    from fastalgebraictransformer_b200 import algebraic_model
    with FakeTensorMode():
        model, cache = model_and_cache()
        step = algebraic_model._DecodeStep.make(model, cache)
        stock = algebraic_model.AlgebraicAttention.forward
        monkeypatch.setattr(algebraic_model.AlgebraicAttention, "forward", lambda self, *a, **k: stock(self, *a, **k))
        assert not step.stands(model) and algebraic_model._DecodeStep.make(model, cache) is None


def test_heads_that_are_not_the_caches_make_no_fused_step():
    from fastalgebraictransformer_b200.algebraic_model import _DecodeStep
    with FakeTensorMode():
        model, cache = model_and_cache()
        for block in model.blocks:
            block.attn.n_head, block.attn.d_head = 1, 128
        assert _DecodeStep.make(model, cache) is None


def test_constants_changed_everywhere_are_taken_over():
    from fastalgebraictransformer_b200.algebraic_model import _DecodeStep
    with FakeTensorMode():
        model, cache = model_and_cache()
        for block in model.blocks:
            block.attn.scale = 0.5
        for norm in [model.norm] + [n for b in model.blocks for n in (b.norm1, b.norm2)]:
            norm.eps = 1e-3
        assert _DecodeStep.make(model, cache).rest[1:3] == (0.5, 1e-3)


def test_decode_step_operator_declares_what_it_writes_and_its_shape():
    """The caches' rows, the lengths and the workspace; the result is [B, V] of the head's dtype."""
    from fastalgebraictransformer_b200.algebraic_model import _DecodeStep
    schema = torch.ops.algebraic.lm_decode_step.default._schema
    written = {a.name for a in schema.arguments if a.alias_info is not None and a.alias_info.is_write}
    assert written == {"k", "v", "lengths", "workspace"}
    with FakeTensorMode():
        model, cache = model_and_cache()
        logits = _DecodeStep.make(model, cache)(torch.zeros(2, 1, dtype=torch.int64, device="cuda:0"), cache)
        assert logits.shape == (2, 64) and logits.dtype == torch.bfloat16


@pytest.mark.parametrize("B,d_model,d_ffn,fused", [
    (8, 768, 2048, True), (8, 1024, 2730, True), (16, 512, 1365, True), (1, 768, 2048, True), (1, 1024, 2730, True), (2, 512, 1365, True),
    (9, 768, 2048, False), (16, 1024, 2730, False), (1, 512, 1365, False), (1, 896, 2389, False), (4, 1280, 3413, False), (1, 1536, 4096, False),
])
def test_which_way_a_captured_step_goes(B, d_model, d_ffn, fused):
    """Both sides of the line (which is on the safe side: beyond it the launch is the faster way at some of these sizes too)."""
    from fastalgebraictransformer_b200.algebraic_model import _DecodeStep
    assert _DecodeStep.beats_replayed_operators(B, d_ffn, d_model) == fused


def test_copies_of_a_cache_leave_the_step_behind():
    """A step's workspace serves one cache at a time, and a saved cache must not carry the model."""
    import copy
    import pickle
    from fastalgebraictransformer_b200.algebraic_model import KVCache
    cache = KVCache(2, 1, 2, 8, 64, torch.float32, "cpu")
    cache.step, cache.seen = Step(), 3
    for other in (copy.copy(cache), copy.deepcopy(cache), pickle.loads(pickle.dumps(cache))):
        assert other.step is None and other.seen == 3 and torch.equal(other.lengths, cache.lengths)
    assert isinstance(cache.step, Step)


@pytest.mark.parametrize("C,D,widest", [(1280, 64, {8: 8384, 16: 2368}), (1024, 128, {8: 8896, 16: 2880}), (768, 64, {8: 9408, 16: 3392}), (2048, 128, {8: 6848, 16: 0})])
def test_the_widest_feed_forward_row_that_the_step_takes(C, D, widest):
    """What the launch refuses goes module by module: the line at which the tokens' rows are too large for it (1280 wide with 16 sequences and the
    default d_ffn of 3413 is beyond it), on both of its sides."""
    from fastalgebraictransformer_b200 import _lib
    need = _lib.lib().fat_lm_decode_workspace_bytes
    need.restype, need.argtypes = _lib.PROTOTYPES["fat_lm_decode_workspace_bytes"]
    for rows, F in widest.items():
        for B in (rows, rows - 7):
            assert F == 0 or need(B, C, C // D, D, F, 100, 2, 64, _lib.BF16) > 0
            assert need(B, C, C // D, D, max(F, C) + 1, 100, 2, 64, _lib.BF16) == 0
