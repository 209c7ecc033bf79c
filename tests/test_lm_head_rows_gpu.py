"""The LM head over the labelled rows only: selections at the edges of tiles, k-blocks and row blocks, against the FP32
head; unlabelled rows must not reach the loss or a gradient, whatever they hold."""
import pytest
import torch

from warpstate_ai_b200.ops import _ext, lmhead
from warpstate_ai_b200.ops import reference as R
from warpstate_ai_b200.ops.gemm import check_device_errors

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-9))


def labels_with(kind, rows, vocab):
    labels = torch.randint(0, vocab, (rows,), device="cuda")
    keep = torch.zeros(rows, dtype=torch.bool, device="cuda")
    if kind == "span":
        keep[rows // 8:rows // 2 + 3] = True
    elif kind == "random":
        keep = torch.rand(rows, device="cuda") < 0.3
    else:                                   # a count: that many rows, spread over the batch
        keep[torch.randperm(rows, device="cuda")[:kind]] = True
    labels[~keep] = -100
    return labels, keep


@pytest.mark.parametrize("rows,d,vocab,kind", [
    (512, 256, 1000, 0), (512, 256, 1000, 1), (600, 256, 1000, 64), (600, 256, 1000, 65), (777, 256, 1000, 255),
    (777, 256, 1000, 256), (777, 256, 1000, 257), (777, 256, 1000, 776), (777, 256, 1000, 777), (2048, 512, 32768, "span"),
    (17000, 128, 520, "random"), (17000, 128, 520, 8192), (17000, 128, 520, 8193), (17000, 128, 520, 16500),
    (17000, 128, 520, 17000)])
def test_head_over_labelled_rows(rows, d, vocab, kind):
    # BF16 logits and logit gradients (2^-9 each, independent per element) against FP32 ones: as in the dense test
    _ext.require()
    torch.manual_seed(rows + vocab)
    hidden = torch.randn(rows, d, device="cuda").bfloat16()
    labels, keep = labels_with(kind, rows, vocab)
    hidden[~keep] = float("nan")
    hidden.requires_grad_(True)
    weight = (torch.randn(vocab, d, device="cuda") * 0.05).requires_grad_(True)
    coef = torch.randn(rows, device="cuda")
    assert rows >= lmhead.SELECT_FROM and lmhead.kernels_ready(hidden, weight)
    logp = lmhead.token_logps(hidden, weight, labels)
    (logp * coef).sum().backward()
    check_device_errors()
    h32 = hidden.detach()[keep].float().requires_grad_(True)
    w32 = weight.detach().bfloat16().float().requires_grad_(True)
    want = R.lm_head_token_logps(h32, w32, labels[keep])
    (want * coef[keep]).sum().backward()
    assert torch.count_nonzero(logp[~keep]) == 0 and torch.count_nonzero(hidden.grad[~keep]) == 0
    assert torch.isfinite(hidden.grad).all() and torch.isfinite(weight.grad).all()
    if keep.any():
        assert rel(logp[keep], want) < 5e-3
        assert rel(hidden.grad[keep], h32.grad) < 0.02
        assert rel(weight.grad, w32.grad) < 0.02
    else:
        assert torch.count_nonzero(weight.grad) == 0
    # a second pass accumulates into the tied gradient and changes nothing else
    first = hidden.grad.clone()
    hidden.grad = None
    (lmhead.token_logps(hidden, weight, labels) * coef).sum().backward()
    assert torch.equal(hidden.grad, first) and rel(weight.grad, 2 * w32.grad if keep.any() else weight.grad) < 0.02


@pytest.mark.parametrize("rows,kept,kind", [(777, 777, 777), (777, 777, 300), (777, 256, 777), (777, 512, 257), (9000, 256, "random"),
                                            (9000, 0, "random")])
def test_kept_logits_give_the_bits_of_recomputed_ones(monkeypatch, rows, kept, kind):
    """Logit gradients from kept logits, from recomputed ones, and from both in one pass; a second backward over the same
    graph recomputes what the first consumed."""
    _ext.require()
    torch.manual_seed(rows + kept)
    d, vocab = 256, 1000
    hidden = torch.randn(rows, d, device="cuda").bfloat16()
    labels, keep = labels_with(kind, rows, vocab)
    weight = torch.randn(vocab, d, device="cuda") * 0.05
    coef = torch.randn(rows, device="cuda")

    def gradients(keep_bytes, passes=1):
        monkeypatch.setattr(lmhead, "KEEP_BYTES", keep_bytes)
        h, w = hidden.clone().requires_grad_(True), weight.clone().requires_grad_(True)
        value = (lmhead.token_logps(h, w, labels) * coef).sum()
        for index in range(passes):
            h.grad = w.grad = None
            value.backward(retain_graph=index + 1 < passes)
        check_device_errors()
        return h.grad, w.grad

    assert lmhead.kept_rows(rows, vocab) == rows
    recomputed = gradients(0)
    monkeypatch.setattr(lmhead, "KEEP_BYTES", 2 * vocab * kept)
    assert lmhead.kept_rows(rows, vocab) == kept
    mine, twice = gradients(2 * vocab * kept), gradients(2 * vocab * kept, passes=2)
    assert torch.equal(mine[0], recomputed[0]) and torch.equal(twice[0], recomputed[0])
    # the weight gradient is added up over blocks of rows, which end elsewhere: FP32 additions in another order
    assert rel(mine[1], recomputed[1]) < 1e-5 and rel(twice[1], recomputed[1]) < 1e-5


def test_scratch_of_the_recomputed_rows_has_their_number(monkeypatch):
    """A few rows past the kept ones take a few rows of logits beside them, not a whole block."""
    _ext.require()
    torch.manual_seed(0)
    rows, kept, d, vocab = 4096 + 40, 4096, 64, 8192
    monkeypatch.setattr(lmhead, "KEEP_BYTES", 2 * vocab * kept)
    hidden = torch.randn(rows, d, device="cuda").bfloat16().requires_grad_(True)
    weight = (torch.randn(vocab, d, device="cuda") * 0.05).requires_grad_(True)
    labels = torch.randint(0, vocab, (rows,), device="cuda")
    peak = None
    for _ in range(2):                                       # once to have casts, flags and cached gradients in place
        hidden.grad = weight.grad = None
        value = lmhead.token_logps(hidden, weight, labels).sum()
        torch.cuda.synchronize()
        before = torch.cuda.memory_allocated()
        torch.cuda.reset_peak_memory_stats()
        value.backward()
        peak = torch.cuda.max_memory_allocated() - before
    check_device_errors()
    small = rows * d * 2 + 2 * vocab * d * 4 + rows * 16     # dhidden, the FP32 weight gradient (once more as autograd's), vectors
    assert peak < small + 40 * vocab * 2 + (1 << 20), peak


def head_problem(rows=777, d=256, vocab=1000):
    torch.manual_seed(rows)
    hidden = torch.randn(rows, d, device="cuda").bfloat16()
    labels, _ = labels_with("random", rows, vocab)
    return hidden, torch.randn(vocab, d, device="cuda") * 0.05, labels, torch.randn(rows, device="cuda")


def test_kept_logits_are_saved_tensors():
    """Hooks on saved tensors (offload, checkpointing) see all that the head holds between its passes, and what they
    give back is what the backward pass uses."""
    _ext.require()
    hidden, weight, labels, coef = head_problem()
    plain_h, plain_w = hidden.clone().requires_grad_(True), weight.clone().requires_grad_(True)
    (lmhead.token_logps(plain_h, plain_w, labels) * coef).sum().backward()
    packed_shapes = []

    def pack(t):
        packed_shapes.append((t.dtype, tuple(t.shape)))
        return t.cpu()

    h, w = hidden.clone().requires_grad_(True), weight.clone().requires_grad_(True)
    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t.cuda()):
        value = (lmhead.token_logps(h, w, labels) * coef).sum()
    assert (torch.bfloat16, (777, 1000)) in packed_shapes
    for index in range(2):                                   # the second time the hooks give fresh logits back
        h.grad = w.grad = None
        value.backward(retain_graph=index == 0)
        assert torch.equal(h.grad, plain_h.grad) and torch.equal(w.grad, plain_w.grad)


def test_checkpointing_the_head_holds_no_logits():
    _ext.require()
    from torch.utils.checkpoint import checkpoint
    hidden, weight, labels, coef = head_problem(rows=2048, d=64, vocab=8192)
    plain_h, plain_w = hidden.clone().requires_grad_(True), weight.clone().requires_grad_(True)
    (lmhead.token_logps(plain_h, plain_w, labels) * coef).sum().backward()
    h, w = hidden.clone().requires_grad_(True), weight.clone().requires_grad_(True)
    before = torch.cuda.memory_allocated()
    value = (checkpoint(lmhead.token_logps, h, w, labels, use_reentrant=False) * coef).sum()
    assert torch.cuda.memory_allocated() - before < 2 * 2048 * 8192 // 4     # the logits are 32 MiB
    value.backward()
    check_device_errors()
    assert torch.equal(h.grad, plain_h.grad) and rel(w.grad, plain_w.grad) < 1e-6


@pytest.mark.parametrize("checkpointing,holds", [(False, True), (True, False)])
def test_a_model_that_checkpoints_its_blocks_keeps_no_logits(checkpointing, holds):
    _ext.require()
    from warpstate_ai_b200 import WarpStateConfig, WarpStateLM
    cfg = WarpStateConfig(vocab_size=8192, d_model=128, n_heads=2, n_cores=1, logical_depth=1, ffn_hidden=192, chunk_size=128,
                          gradient_checkpointing=checkpointing, parallel_memory=True)
    with torch.device("cuda"):
        model = WarpStateLM(cfg).train()
    hidden = torch.randn(2, 1024, 128, device="cuda", dtype=torch.bfloat16).requires_grad_(True)
    targets = torch.randint(0, 8192, (2, 1024), device="cuda")
    for _ in range(2):
        before = torch.cuda.memory_allocated()
        with torch.autocast("cuda", dtype=torch.bfloat16):
            loss = model.loss_from_hidden(hidden, targets)
        held = torch.cuda.memory_allocated() - before
        loss.backward()
        del loss
    assert (held > 2048 * 8192 * 2) is holds                 # 32 MiB of logits


# at most 1536 rows and at least four rounds of tiles: the weight gradient fetches its old sums, adds to them and stores them, for as many
# k-blocks as the selection has rows
@pytest.mark.parametrize("rows,d,kind", [(1200, 1024, 0), (1200, 1024, 1), (1200, 1024, 64), (1536, 768, 65), (1200, 1024, "span"), (1531, 1024, "random"),
                                         (1536, 768, 1536)])
def test_fetched_sums_of_a_selection(rows, d, kind):
    _ext.require()
    torch.manual_seed(rows + d)
    vocab = 32768
    hidden = torch.randn(rows, d, device="cuda").bfloat16()
    labels, keep = labels_with(kind, rows, vocab)
    hidden[~keep] = float("nan")
    hidden.requires_grad_(True)
    weight = (torch.randn(vocab, d, device="cuda") * 0.05).requires_grad_(True)
    coef = torch.randn(rows, device="cuda")
    before = torch.randn(vocab, d, device="cuda") * 0.01
    weight.main_grad = before.clone()
    logp = lmhead.token_logps(hidden, weight, labels)
    (logp * coef).sum().backward()
    check_device_errors()
    if not keep.any():
        assert torch.equal(weight.main_grad, before)
        return
    w32 = weight.detach().bfloat16().float().requires_grad_(True)
    (R.lm_head_token_logps(hidden.detach()[keep].float(), w32, labels[keep]) * coef[keep]).sum().backward()
    # the product as above; the sum and the difference here round once each
    assert rel(weight.main_grad.double() - before.double(), w32.grad) < 0.02 + 2.0 ** -23 * float(before.norm() / w32.grad.norm())
