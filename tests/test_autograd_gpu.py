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


OPERATORS = {"softmax": "softmax_fwd", "swiglu": "swiglu_fwd", "norm": "norm_fwd", "add_norm": "add_norm_fwd", "attention": "attn_fwd",
             "attention_packed": "attn_fwd"}


@pytest.mark.parametrize("name", OPERATORS)
def test_torch_function_modes_see_the_operators(name):
    seen = []

    class Mode(torch.overrides.TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))

    fn, leaves, constants = case(name)
    with Mode():
        out = fn(*leaves, *constants)
    assert f"algebraic.{OPERATORS[name]}" in seen
    loss_of(out).backward()
    assert same([t.grad for t in leaves], plain_grads(name))


@pytest.mark.parametrize("name", OPERATORS)
def test_torch_function_of_a_subclass_is_asked(name):
    seen = []

    class Marked(torch.Tensor):
        @classmethod
        def __torch_function__(cls, func, types, args=(), kwargs=None):
            seen.append(getattr(func, "__name__", str(func)))
            return super().__torch_function__(func, types, args, kwargs or {})

    fn, leaves, constants = case(name)
    out = fn(*[t.detach().as_subclass(Marked) for t in leaves], *constants)
    assert OPERATORS[name] in seen
    assert type(out[0] if isinstance(out, tuple) else out) is Marked


@pytest.mark.parametrize("name", OPERATORS)
@pytest.mark.parametrize("transform", ["vmap", "grad"])
def test_functorch_transforms_stay_refused(name, transform):
    """The operators have no functorch rules; a call under a transform raises, as their autograd Functions always did."""
    fn, leaves, constants = case(name)
    args = [t.detach() for t in leaves]
    with pytest.raises(RuntimeError, match="functorch"):
        if transform == "vmap":
            torch.vmap(lambda x: loss_of(fn(x, *args[1:], *constants)))(torch.stack([args[0]] * 2))
        else:
            torch.func.grad(lambda x: loss_of(fn(x, *args[1:], *constants)))(args[0])


@pytest.mark.parametrize("name", OPERATORS)
def test_forward_mode_is_refused(name):
    import torch.autograd.forward_ad as forward_ad
    fn, leaves, constants = case(name)
    with forward_ad.dual_level(), pytest.raises(NotImplementedError):
        fn(forward_ad.make_dual(leaves[0], torch.ones_like(leaves[0])), *leaves[1:], *constants)


def test_a_graph_of_gradients_keeps_the_packed_gradient():
    """create_graph: the halves' projection still gets one packed gradient, not a concatenation (the profiler's view of it)."""
    x = torch.randn(64, 512, device=DEV, requires_grad=True)
    results = []
    for create in (False, True):
        out = fat().rational_swiglu(*x.chunk(2, -1))
        with torch.profiler.profile() as prof:
            results.append(torch.autograd.grad(out, x, torch.ones_like(out), create_graph=create)[0].detach())
        names = {e.name for e in prof.events()}
        assert "algebraic::swiglu_bwd_packed" in names and "aten::cat" not in names, create
    assert torch.equal(*results)


def test_a_traced_feed_forward_block_keeps_the_packed_gradient():
    """torch.compile of the block: the traced backward holds the packed operator and no concatenation; same gradients."""
    from torch._dynamo.backends.common import aot_autograd
    graphs = []

    def keep(graph, inputs):
        graphs.append({str(n.target) for n in graph.graph.nodes})
        return graph.forward

    torch.manual_seed(8)
    block = fat().algebraic_model.RationalSwiGLU(64, 96).to(DEV)
    x = torch.randn(2, 17, 64, device=DEV, requires_grad=True)
    want = torch.autograd.grad(block(x).sum(), [x, *block.parameters()])
    got = torch.autograd.grad(torch.compile(block, backend=aot_autograd(fw_compiler=keep, bw_compiler=keep))(x).sum(), [x, *block.parameters()])
    assert same(got, want)
    names = set().union(*graphs)
    assert any("swiglu_bwd_packed" in n for n in names) and not any("aten.cat" in n for n in names)


@pytest.mark.parametrize("name", ["attention", "attention_packed"])
@pytest.mark.parametrize("inputs", [False, True])
def test_slopes_that_ask_for_a_gradient(name, inputs):
    """They have none (the operator's slopes are constants), but the result belongs to their graph, as with the Functions."""
    fn, leaves, (slopes,) = case(name)
    slopes.requires_grad_(True)
    leaves = [t.requires_grad_(inputs) for t in (x.detach() for x in leaves)]
    out = fn(*leaves, slopes)
    assert out.requires_grad
    loss_of(out).backward()
    assert slopes.grad is None
    assert same([t.grad for t in leaves], plain_grads(name) if inputs else [None] * len(leaves))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("head", [False, True])
def test_traced_loss_has_the_eager_gradients(head, dtype):
    """torch.compile of the loss: its gradients are formed in the forward and scaled in the backward, in place when it is eager."""
    g = torch.Generator().manual_seed(9)
    x, w = torch.randn(2, 17, 64, generator=g).to(dtype).to(DEV), torch.randn(40, 64, generator=g).to(dtype).to(DEV)
    labels = torch.randint(0, 40, (2, 17), generator=g).to(DEV)

    def loss(x, w):
        out = fat().head_shifted_cross_entropy(x, w, labels, -100) if head else fat().shifted_cross_entropy(x, labels, -100)
        return out * 3.0

    results = []
    for fn in (loss, torch.compile(loss, backend="aot_eager")):
        leaves = [x.clone().requires_grad_(True), w.clone().requires_grad_(True)]
        fn(*leaves).backward()
        results.append([t.grad for t in leaves])
    assert (results[0][1] is not None) == head
    # eager: one product with 3 in float32, rounded; traced: the same product
    for got, want in zip(*results[::-1]):
        assert (got is None and want is None) or torch.allclose(got, want, rtol=2.0 ** -7 if dtype == torch.bfloat16 else 1e-6, atol=0)


@pytest.mark.parametrize("name", CALLS)
def test_traced_calls_have_the_eager_gradients(name):
    """torch.compile follows the Function classes instead of the C++ nodes: same formulas, same kernels, same bits."""
    fn, leaves, constants = case(name)
    loss_of(torch.compile(fn, backend="aot_eager")(*leaves, *constants)).backward()
    want = [torch.zeros_like(t) if g is None else g for t, g in zip(leaves, plain_grads(name))]      # (a traced graph fills in zeros)
    assert same([t.grad for t in leaves], want)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("name", CALLS)
def test_saved_tensor_hooks_and_checkpointing(name, dtype):
    """What the nodes save passes through the hooks (here: to the host and back), and a checkpointed call is run again."""
    from torch.utils.checkpoint import checkpoint
    want = plain_grads(name, dtype)
    fn, leaves, constants = case(name, dtype)
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t.shape) or t.cpu(), lambda t: t.to(DEV)):
        out = fn(*leaves, *constants)
    loss_of(out).backward()
    assert packed and close(dtype, [t.grad for t in leaves], want)
    fn, leaves, constants = case(name, dtype)
    loss_of(checkpoint(fn, *leaves, *constants, use_reentrant=False)).backward()
    assert close(dtype, [t.grad for t in leaves], want)


def close(dtype, got, want):
    """The same bits, but for the d_q of the 16-bit attention backward, whose sums land in no fixed order (float32 sums rounded to 16 bits)."""
    if dtype == torch.float32:
        return same(got, want)
    return all((a is None and b is None) or torch.allclose(a, b, rtol=2.0 ** -7, atol=2.0 ** -7 * float(b.abs().max())) for a, b in zip(got, want))


@pytest.mark.parametrize("name", CALLS)
def test_a_graph_kept_for_a_second_backward(name):
    fn, leaves, constants = case(name)
    loss = loss_of(fn(*leaves, *constants))
    loss.backward(retain_graph=True)
    first = [t.grad.clone() if t.grad is not None else None for t in leaves]
    loss.backward()
    assert all((t.grad is None and f is None) or torch.equal(t.grad, 2 * f) for t, f in zip(leaves, first))
    with pytest.raises(RuntimeError, match="second time"):
        loss.backward()
