"""A block as one native autograd node against the node written in Python: the same kernels on the same numbers, so equal bit
for bit, and the same answers to what autograd may ask of a node."""
import pytest
import torch

from warpstate_ai_b200 import WarpStateConfig
from warpstate_ai_b200.models.warpstate import WarpStateCore
from warpstate_ai_b200.ops import fused
from warpstate_ai_b200.optim import ParamArena


def block(seed=0):
    torch.manual_seed(seed)
    cfg = WarpStateConfig(vocab_size=64, d_model=256, n_heads=4, n_cores=1, logical_depth=2, ffn_hidden=192, chunk_size=128,
                          gradient_checkpointing=False, parallel_memory=True)
    with torch.device("cuda"):
        return WarpStateCore(cfg)


def autocast():
    return torch.autocast("cuda", dtype=torch.bfloat16, cache_enabled=False)


def run(core, x, modulation, dy, passes=1, hooks=None):
    for p in core.parameters():
        if p.grad is not None:
            p.grad.zero_()
    leaves = [t.detach().clone().requires_grad_(t.requires_grad) if t is not None else None for t in (x, *modulation)]
    with autocast(), hooks or torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: t):
        y = core(*leaves)
    for i in range(passes):
        y.backward(dy, retain_graph=i + 1 < passes)
    return [y.detach()] + [None if t is None or t.grad is None else t.grad.clone() for t in leaves] + \
        [None if p.grad is None else p.grad.clone() for p in core.parameters()]


@pytest.mark.gpu
@pytest.mark.parametrize("modulated,input_grad,frozen", [(True, True, ()), (False, True, ()), (True, False, ()),
                                                         (True, True, ("norm1.weight", "in_proj.weight", "fast_decay_logit"))])
def test_native_node_equals_the_python_one(monkeypatch, modulated, input_grad, frozen):
    core = block()
    ParamArena(core)
    for name, p in core.named_parameters():
        p.requires_grad_(name not in frozen)
    x = torch.randn(3, 256, 256, device="cuda").requires_grad_(input_grad)
    modulation = [torch.randn(256, device="cuda").mul_(0.1).requires_grad_(True) if modulated else None for _ in range(2)]
    dy = torch.randn(3, 256, 256, device="cuda")
    seen = []
    native = run(core, x, modulation, dy)
    twice = run(core, x, modulation, dy, passes=2)
    hooked = run(core, x, modulation, dy, hooks=torch.autograd.graph.saved_tensors_hooks(
        lambda t: (seen.append(t.shape), t.cpu())[1], lambda t: t.cuda()))
    assert seen
    monkeypatch.setattr(fused, "_block_node", lambda *a: None)
    python = run(core, x, modulation, dy)
    python_twice = run(core, x, modulation, dy, passes=2)
    for a, b, c in ((native, python, hooked), (twice, python_twice, python_twice)):
        for p, q, r in zip(a, b, c):
            assert (p is None) == (q is None) == (r is None)
            assert p is None or (torch.equal(p, q) and torch.equal(p, r))


@pytest.mark.gpu
def test_scoring_pass_and_transposed_input(monkeypatch):
    core = block(1)                                        # no arena: cached casts
    x = torch.randn(256, 2, 256, device="cuda").transpose(0, 1)
    scale, bias = torch.randn(2, 256, device="cuda").mul_(0.1).unbind(0)
    with torch.no_grad(), autocast():
        native = core(x, scale, bias)
        assert not native.requires_grad
        monkeypatch.setattr(fused, "_block_node", lambda *a: None)
        assert torch.equal(native, core(x, scale, bias))
    monkeypatch.undo()
    with autocast():                                       # gradients that autograd holds: the Python node
        assert fused._block_node(core, x, scale, bias, True) is None
        assert type(core(x, scale, bias).grad_fn).__name__ == "CoreFnBackward"
        ParamArena(core)                                   # gradients that the arena holds: the native one
        assert "BlockFn" in core(x, scale, bias).grad_fn.name()


@pytest.mark.gpu
def test_transforms_that_the_node_does_not_support_are_refused():
    core = block(2)
    ParamArena(core)
    x = torch.randn(1, 128, 256, device="cuda")
    with autocast():
        with pytest.raises(RuntimeError):
            torch.func.grad(lambda t: core(t).sum())(x)
        with pytest.raises(RuntimeError):
            torch.func.vmap(core)(x[None])
        with pytest.raises((RuntimeError, NotImplementedError)):
            with torch.autograd.forward_ad.dual_level():
                core(torch.autograd.forward_ad.make_dual(x, torch.ones_like(x)))


@pytest.mark.gpu
def test_a_hook_on_finished_gradients_takes_the_python_node(monkeypatch):
    core, called = block(3), []
    ParamArena(core)
    x = torch.randn(1, 128, 256, device="cuda", requires_grad=True)
    monkeypatch.setattr(fused, "_core_grad_hook", called.append)
    with autocast():
        core(x).sum().backward()
    assert called == [core]


@pytest.mark.gpu
@pytest.mark.parametrize("train", [False, True])
def test_a_bias_without_a_scale_is_no_modulation(monkeypatch, train):
    """Every form of a block takes such a call: the modulation is its scale's to ask for."""
    core = block(4)
    ParamArena(core)
    x, bias = torch.randn(2, 128, 256, device="cuda"), torch.randn(256, device="cuda")
    with torch.set_grad_enabled(train), autocast():
        native = core(x, None, bias)
        assert torch.equal(native, core(x))
        monkeypatch.setattr(fused, "_block_node", lambda *a: None)
        assert torch.equal(native, core(x, None, bias))
        with fused.disabled():
            plain = core(x, None, bias)
        assert torch.allclose(native, plain.float(), rtol=0.1, atol=0.1)


@pytest.mark.gpu
def test_scoring_in_inference_mode():
    core = block(5)
    x = torch.randn(1, 256, 256, device="cuda")
    with autocast(), torch.no_grad():
        want = core(x)
    with autocast(), torch.inference_mode():
        assert torch.equal(core(x), want) and torch.equal(core(x.clone()), want)


@pytest.mark.gpu
@pytest.mark.parametrize("arena", [True, False])
def test_a_compiled_caller(arena):
    """`torch.compile` around a block, or around the code that calls one, runs the block as it is."""
    core = block(6)
    if arena:
        ParamArena(core)
    x = torch.randn(2, 128, 256, device="cuda")
    dy = torch.randn(2, 128, 256, device="cuda")
    want = run(core, x.requires_grad_(True), (None, None), dy)
    got = run(torch.compile(core, backend="eager"), x, (None, None), dy)
    for a, b in zip(want, got):
        assert (a is None) == (b is None) and (a is None or torch.equal(a, b))
    with torch.no_grad(), autocast():
        assert torch.equal(torch.compile(lambda t: core(t) * 2.0, backend="eager")(x), want[0] * 2.0)
    torch._dynamo.reset()


@pytest.mark.gpu
@pytest.mark.filterwarnings("ignore:.*autograd kernel was not registered")
@pytest.mark.parametrize("native", [True, False])
def test_create_graph_gives_gradients_without_a_second_derivative(monkeypatch, native):
    core = block(7)
    ParamArena(core)
    if not native:
        monkeypatch.setattr(fused, "_block_node", lambda *a: None)
    x, dy = (torch.randn(1, 128, 256, device="cuda", requires_grad=True) for _ in range(2))
    with autocast():
        y = core(x)
    plain, = torch.autograd.grad(y, [x], dy, retain_graph=True)
    gradient, = torch.autograd.grad(y, [x], dy, create_graph=True)
    assert gradient.requires_grad and torch.equal(gradient, plain)
    assert torch.autograd.grad(gradient.sum(), [x, dy], allow_unused=True) == (None, None)
