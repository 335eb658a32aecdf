"""The operators' C++ autograd nodes under the machinery that plain Python autograd Functions work with (B200)."""
import pytest
import torch

from oracle import oracle

pytestmark = pytest.mark.gpu
DEV = "cuda"


def fat():
    import fastalgebraictransformer_b200 as m
    return m


def _packed(qkv, slopes):
    from fastalgebraictransformer_b200.backward import rational_attention_packed
    return rational_attention_packed(qkv, slopes, 0.125)


def _masked(q, k, v, slopes):
    keep = (torch.arange(q.size(2), device=q.device)[None] < torch.tensor([[20], [33]], device=q.device)).to(torch.int64)
    return fat().rational_attention(q, k, v, slopes, 0.125, key_mask=keep)


# name: (call, shapes of its differentiable inputs); the last entry of a shape list that is a number adds ALiBi slopes for that many heads
CALLS = {
    "softmax": (lambda x: fat().rational_softmax(x), [(5, 48)]),
    "swiglu": (lambda g, v: fat().rational_swiglu(g, v), [(5, 48), (5, 48)]),
    "swiglu_halves": (lambda x: fat().rational_swiglu(*x.chunk(2, -1)), [(5, 96)]),
    "norm": (lambda x, w: fat().mean_error_norm(x, w), [(5, 48), (48,)]),
    "add_norm": (lambda x, r, w: fat().add_mean_error_norm(x, r, w), [(5, 48), (5, 48), (48,)]),
    "add_norm_sum_only": (lambda x, r, w: fat().add_mean_error_norm(x, r, w)[0], [(5, 48), (5, 48), (48,)]),
    "attention": (lambda q, k, v, s: fat().rational_attention(q, k, v, s, 0.125), [(2, 3, 33, 64)] * 3 + [3]),
    "attention_masked": (_masked, [(2, 3, 33, 64)] * 3 + [3]),
    "attention_packed": (_packed, [(2, 33, 3, 2, 64), 2]),
}


def case(name, dtype=torch.float32):
    """(call, differentiable inputs, constants), the same numbers every time."""
    fn, shapes = CALLS[name]
    g = torch.Generator().manual_seed(71)
    leaves = [torch.randn(s, generator=g).to(dtype).to(DEV).requires_grad_(True) for s in shapes if isinstance(s, tuple)]
    return fn, leaves, [oracle.compute_alibi_slopes(s).to(DEV) for s in shapes if not isinstance(s, tuple)]


def loss_of(out):
    return sum((o * torch.linspace(0.5, 1.5, o.numel(), device=DEV).view(o.shape).to(o.dtype)).sum() for o in (out if isinstance(out, tuple) else (out,)))


def plain_grads(name, dtype=torch.float32):
    fn, leaves, constants = case(name, dtype)
    loss_of(fn(*leaves, *constants)).backward()
    return [t.grad for t in leaves]


def same(got, want):
    return all((a is None and b is None) or torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("name", CALLS)
def test_compiled_autograd_over_an_eager_forward(name):
    """The backward of an eager forward traced as a whole: the nodes show what they depend on and run on the tracer's tensors."""
    from torch._dynamo import compiled_autograd
    fn, leaves, constants = case(name)
    for _ in range(2):                                  # (the second pass finds the first one's trace)
        for t in leaves:
            t.grad = None
        loss = loss_of(fn(*leaves, *constants))
        with compiled_autograd._enable(lambda graph: graph):
            loss.backward()
        assert same([t.grad for t in leaves], plain_grads(name))
