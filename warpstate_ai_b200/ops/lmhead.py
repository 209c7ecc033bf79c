"""Fused LM-head cross-entropy (front-end of the WS_EPI_CE_* GEMM epilogues and lmhead.cu).

Forward: one tcgen05 GEMM over the tied embedding matrix whose epilogue folds each 128-column
slice of the logits into (max, sum exp) and records the label's logit; where no backward pass
follows, the ``[tokens, vocab]`` logits are not written.  Backward: the logit gradients
``(softmax - onehot) * row_weight`` in BF16 feed the dX GEMM (gradient of the hidden states) and
the dW GEMM (FP32 accumulation into the tied embedding's gradient).

An unlabelled row (-100: prompts and padding, most of a post-training batch) adds nothing to either pass, so from
`SELECT_FROM` rows on the labelled rows are packed together on the device and the GEMMs run over them alone; their
number is read by the kernels, not by the host.  Where every row is labelled nothing is copied.  When a backward pass
will follow, the forward pass leaves the BF16 logits of up to `KEEP_BYTES` worth of rows behind, from which the logit
gradients are formed in place; for the rows past them, and below `SELECT_FROM` rows, the backward pass computes the
logits again, block by block, and the gradients come out of that product's epilogue.

`loss_sum` is the summed cross-entropy over labels != -100 (reference warpstate/model.py:316-334,
ops/loss_experiment.py:14-19); `token_logps` is the per-row label log-probability used for
per-sequence sums in DPO (reference dpo.py:150-161).
"""
from __future__ import annotations

import torch

from . import _ext
from . import gemm as G

IGNORE = -100
# Two tiles of the CTA-pair GEMM.  Below, at most one tile of rows could be left out, and the passes over the weight and its
# gradient are what the head costs (d 2048, vocabulary 32768, forward + backward with every row labelled: 0.56 ms over all
# 256 rows, 0.52 selected; 30 % labelled 0.54 and 0.52).  At 512 rows 0.58 and 0.53, at 2048 with 30 % labelled 0.89 and 0.59.
SELECT_FROM = 512
ROWS_PER_BLOCK = 8192  # bounds the BF16 dlogits scratch to 512 MiB at vocab 32768
# Logits kept between the passes of one call, unless it says otherwise: 16384 rows at vocab 32768, the micro-batch of the
# production run.  They live as long as the call's graph, in a training step from the head's forward to its backward, which
# follows at once, and there they are the logit gradients' buffer.  They count every row, labelled or not (how many are
# labelled is known on the device only).  Peak of a backward pass: the kept bytes and, for rows past them, the logits of
# min(`ROWS_PER_BLOCK`, those rows); with 0 kept bytes the latter alone, at most 512 MiB at vocab 32768.
KEEP_BYTES = 1 << 30


def kept_rows(rows: int, vocab: int, keep_bytes: int | None = None) -> int:
    """Rows whose logits are kept: all of them, or as many whole tiles of 256 as ``keep_bytes`` (`KEEP_BYTES`) hold."""
    most = (KEEP_BYTES if keep_bytes is None else keep_bytes) // (2 * vocab)
    return rows if rows <= most else most // 256 * 256


def kernels_ready(hidden: torch.Tensor, weight: torch.Tensor) -> bool:
    return (hidden.is_cuda and hidden.dim() == 2 and weight.shape[0] % 8 == 0 and hidden.shape[1] % 8 == 0
            and _ext.available())


class _TokenLogps(torch.autograd.Function):
    """per-row log p(label) (0 where the label is -100); differentiable w.r.t. hidden and weight."""

    @staticmethod
    def forward(ctx, hidden, weight, labels, keep_bytes):
        from .fused import bf16_weight
        ops = torch.ops.ws_b200
        hidden = hidden.contiguous()
        labels = labels.contiguous()
        wb = bf16_weight(weight)
        flag = G.error_flag(hidden.device)
        ctx.weight = weight
        ctx.selected = hidden.shape[0] >= SELECT_FROM and ops.gemm_pair_available()
        if ctx.selected:
            keep = kept_rows(hidden.shape[0], wb.shape[0], keep_bytes)
            logp, *rest = ops.lm_head_fwd_labelled(hidden, wb, labels, IGNORE, keep, flag)
            ctx.save_for_backward(hidden, labels, *rest)
            ctx.spent = False
            return logp
        lse, logp = ops.lm_head_fwd(hidden, wb, labels, IGNORE, flag)
        ctx.save_for_backward(hidden, labels, lse)
        return logp

    @staticmethod
    def backward(ctx, grad_logp):
        from .fused import bf16_weight
        ops = torch.ops.ws_b200
        hidden, labels, lse, *selection = ctx.saved_tensors
        weight = ctx.weight
        wb = bf16_weight(weight)
        flag = G.error_flag(hidden.device)
        # d logp / d logits = onehot - softmax  ->  dlogits = (softmax - onehot) * (-grad), masked rows 0
        row_weight = (-grad_logp.float() * labels.ne(IGNORE)).contiguous()
        dh = torch.empty_like(hidden)
        main = getattr(weight, "main_grad", None)
        grad_w = main if main is not None else torch.zeros(weight.shape, dtype=torch.float32, device=weight.device)
        if ctx.selected:
            index, count, packed, labels_sel, logits = selection
            # the logits become their own gradients: another backward over the same graph computes them again
            if ctx.spent:
                logits = logits.new_empty(0)
            ctx.spent = True
            ops.lm_head_bwd_labelled(hidden, packed, wb, labels, labels_sel, index, count, lse, row_weight, IGNORE,
                                     ROWS_PER_BLOCK, logits, dh, grad_w, flag)
            return dh, (None if main is not None else grad_w.to(weight.dtype)), None, None
        for start in range(0, hidden.shape[0], ROWS_PER_BLOCK):
            stop = min(start + ROWS_PER_BLOCK, hidden.shape[0])
            h = hidden[start:stop]
            dlogits = ops.lm_head_dlogits(h, wb, labels[start:stop], lse[start:stop], row_weight[start:stop], flag)
            G.grad_input(dlogits, wb, out=dh[start:stop])
            G.grad_weight_accumulate(dlogits, h, grad_w, accumulate=True)
        return dh, (None if main is not None else grad_w.to(weight.dtype)), None, None


def token_logps(hidden: torch.Tensor, weight: torch.Tensor, labels: torch.Tensor,
                keep_bytes: int | None = None) -> torch.Tensor:
    """``keep_bytes``: how much of the logits may be held for the backward pass (None: `KEEP_BYTES`; 0 where memory counts
    more than the product that makes them again)."""
    if not (torch.is_grad_enabled() and (hidden.requires_grad or weight.requires_grad)):
        keep_bytes = 0
    return _TokenLogps.apply(hidden, weight, labels, keep_bytes)


def loss_sum(hidden: torch.Tensor, weight: torch.Tensor, labels: torch.Tensor, keep_bytes: int | None = None) -> torch.Tensor:
    return -token_logps(hidden, weight, labels, keep_bytes).sum()
