"""The hook on a core's finished gradients: set for the backward pass alone or for both, it fires once per core and finds every
gradient of the core final, also where several depths share the core (their norms' and logits' gradients would otherwise be
added after it, to a bucket that is already being reduced)."""
import gc
import os
import subprocess
import sys
import weakref
from pathlib import Path

import pytest
import torch
import torch.distributed as dist

from warpstate_ai_b200 import WarpStateConfig, WarpStateLM
from warpstate_ai_b200.ops import attention, fused, gemm
from warpstate_ai_b200.optim import ParamArena


def model(device, cores, depth):
    torch.manual_seed(cores + depth)
    cfg = WarpStateConfig(vocab_size=64, d_model=256, n_heads=4, n_cores=cores, logical_depth=depth, ffn_hidden=192, chunk_size=128,
                          gradient_checkpointing=False, parallel_memory=True)
    with torch.device(device):
        return WarpStateLM(cfg)


def gradients(core):
    return {name: p.main_grad.clone() for name, p in core.named_parameters()}


@pytest.fixture(autouse=True)
def no_hook_afterwards():
    yield
    fused.set_core_grad_hook(None)


def check(forward, backward, arena, cores, hook_in_forward):
    """Gradients with the hook set equal those without it; when it fires they are what they are at the end."""
    arena.zero_grad()
    backward(forward())
    want = [gradients(core) for core in cores]
    seen = []
    arena.zero_grad()
    hook = lambda core: seen.append((core, gradients(core)))
    if hook_in_forward:
        fused.set_core_grad_hook(hook)
    y = forward()
    fused.set_core_grad_hook(hook)
    backward(y)
    fused.set_core_grad_hook(None)
    assert [core for core, _ in seen] == list(reversed(cores))
    for core, found in seen:
        final = gradients(core)
        assert all(torch.equal(found[name], final[name]) for name in final), [n for n in final if not torch.equal(found[n], final[n])]
    for core, values in zip(cores, want):
        for name, g in gradients(core).items():
            assert g.abs().sum() > 0 and torch.equal(g, values[name]), name


class Node(torch.autograd.Function):
    """Stands for the native block: a gradient for each of its arguments, and the question that the native node asks."""

    @staticmethod
    def forward(ctx, x, scale, bias, n1, n2, fast, slow, mix, main, hooked, core, notify):
        ctx.main, ctx.hook, ctx.factor = main, (hooked, core, notify), float(x.flatten()[0])
        ctx.shapes = [None if t is None else t.shape for t in (scale, bias, n1, n2)] + [t.shape for t in (fast, slow, mix)]
        return x * 2.0

    @staticmethod
    def backward(ctx, dy):
        for m in ctx.main:
            m += 1.0
        scale, bias, n1, n2, fast, slow, mix = (None if s is None else torch.full(s, ctx.factor * (i + 1)) for i, s in enumerate(ctx.shapes))
        hooked, core, notify = ctx.hook
        if int(hooked) and fused._core_finished(core, notify, [n1, n2, fast, slow, mix]):
            n1 = n2 = fast = slow = mix = None
        return dy * 2.0, scale, bias, n1, n2, fast, slow, mix, None, None, None, None


def stand_ins(replace):
    def block(x, scale, bias, n1, n2, weights, bf16, main, fast, slow, mix, rope, eps, heads, flag, hooked, core, notify):
        return Node.apply(x, scale, bias, n1, n2, fast, slow, mix, main, hooked, core, notify)
    replace(fused, "_native_block", lambda: block)
    replace(attention, "kernels_ready", lambda core: True)
    replace(gemm, "error_flag", lambda device: None)


def blocks_forward(net, value=1.0):
    x = torch.full((1, 128, 256), value)
    for depth, (scale, bias) in enumerate(zip(net.depth_scale.unbind(0), net.depth_bias.unbind(0))):
        x = fused.core_forward(net.cores[depth % len(net.cores)], x, scale, bias, notify=depth < len(net.cores))
    return x


@pytest.mark.parametrize("cores,depth", [(1, 1), (2, 4), (2, 3)])
def test_a_native_node_leaves_nothing_behind_the_hook(monkeypatch, cores, depth):
    stand_ins(monkeypatch.setattr)
    net = model("cpu", cores, depth)
    arena = ParamArena(net, bf16_mirror=True)
    check(lambda: blocks_forward(net), lambda y: y.sum().backward(), arena, list(net.cores), False)


def worker(rank, world, folder):
    """Gradients reduced from the hook on, against the average of every rank's own."""
    from warpstate_ai_b200.parallel.grad_sync import CollectiveGradSync
    dist.init_process_group("gloo", init_method=(folder / "rendezvous").as_uri(), rank=rank, world_size=world)
    stand_ins(setattr)
    net = model("cpu", 2, 4)
    arena = ParamArena(net, bf16_mirror=True)
    sync = CollectiveGradSync(torch.device("cpu"), world, rank)
    sync.attach(arena, net)
    blocks_forward(net, 1.0 + rank).sum().backward()
    want = arena.grad.clone()
    dist.all_reduce(want)
    arena.zero_grad()
    sync.begin_update()
    y = blocks_forward(net, 1.0 + rank)
    with sync.last_micro_batch():
        y.sum().backward()
        assert len(sync.reduced) == 2                       # both cores' buckets, ahead of the tail
    sync.finish_update()
    assert arena.grad.abs().sum() > 0 and torch.equal(arena.grad, want / world)
    dist.destroy_process_group()


def test_two_ranks_with_shared_cores_hold_the_average(tmp_path):
    env = dict(os.environ, PYTHONPATH=str(Path(__file__).resolve().parents[1]) + os.pathsep + os.environ.get("PYTHONPATH", ""))
    ranks = [subprocess.Popen([sys.executable, __file__, str(rank), "2", str(tmp_path)], env=env, stdout=subprocess.PIPE,
                              stderr=subprocess.STDOUT, text=True) for rank in range(2)]
    try:
        for rank in ranks:
            out, _ = rank.communicate(timeout=240)
            assert rank.returncode == 0, out[-3000:]
    finally:
        for rank in ranks:
            rank.kill()


@pytest.mark.gpu
@pytest.mark.parametrize("hook_in_forward", [False, True])
@pytest.mark.parametrize("native", [True, False])
@pytest.mark.parametrize("checkpoint", [False, True])
@pytest.mark.parametrize("cores,depth", [(2, 2), (2, 4)])
def test_shared_cores_on_the_device(monkeypatch, cores, depth, native, checkpoint, hook_in_forward):
    net = model("cuda", cores, depth).train()
    net.cfg.gradient_checkpointing = checkpoint
    arena = ParamArena(net)
    if not native:
        monkeypatch.setattr(fused, "_block_node", lambda *a: None)
    ids = torch.randint(0, 64, (2, 256), device="cuda")
    def forward():
        with torch.autocast("cuda", dtype=torch.bfloat16, cache_enabled=False):
            return net(ids, ids, return_logits=False)[1]
    check(forward, lambda loss: loss.backward(), arena, list(net.cores), hook_in_forward)


def native_forward(net):
    with torch.autocast("cuda", dtype=torch.bfloat16, cache_enabled=False):
        return net.cores[0](torch.ones(1, 128, 256, device="cuda"))


@pytest.mark.gpu
def test_an_error_in_the_hook_ends_the_backward_pass():
    net = model("cuda", 1, 1).train()
    ParamArena(net)
    y = native_forward(net)
    def refuse(core):
        raise KeyError("refused")
    fused.set_core_grad_hook(refuse)
    with pytest.raises(KeyError, match="refused"):
        y.sum().backward()


@pytest.mark.gpu
def test_a_core_that_nobody_holds_any_more():
    net = model("cuda", 1, 1).train()
    ParamArena(net)
    y, norm, core = native_forward(net), net.cores[0].norm1.weight, weakref.ref(net.cores[0])
    del net
    gc.collect()
    assert core() is None
    called = []
    fused.set_core_grad_hook(called.append)
    y.sum().backward()
    assert called == [] and norm.grad.abs().sum() > 0


if __name__ == "__main__":
    worker(int(sys.argv[1]), int(sys.argv[2]), Path(sys.argv[3]))
