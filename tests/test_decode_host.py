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
