"""RMSNorm backward behind a depth modulation: the gradients of scale and bias from the same pass, against FP64 and
against the separate column sums they replace for the FP32 stream."""
import pytest
import torch

from warpstate_ai_b200.ops import _ext

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float((a.double() - b).norm() / b.norm().clamp_min(1e-30))


@pytest.mark.parametrize("rows,d", [(1, 128), (2, 256), (3, 1280), (591, 2048), (593, 1280), (4096, 2048)])
def test_modulation_gradients_of_the_norm_pass(rows, d):
    _ext.require()
    ops = torch.ops.ws_b200
    torch.manual_seed(rows + d)
    x = torch.randn(rows, d, device="cuda") * 0.3
    scale, bias = torch.randn(d, device="cuda") * 0.2, torch.randn(d, device="cuda") * 0.2
    scale[::37] = -1.0                                       # a column the modulation switches off
    w = 1.0 + 0.1 * torch.randn(d, device="cuda")
    dz, dres = torch.randn(rows, d, device="cuda").bfloat16(), torch.randn(rows, d, device="cuda")
    _, rstd, xmod = ops.rmsnorm_fwd(x, scale, bias, w, 1e-5, True)
    dx, grads = ops.rmsnorm_bwd_mod(dz, xmod, rstd, w, dres, scale, bias)
    plain_dx, _, plain_dw = ops.rmsnorm_bwd(dz, xmod, rstd, w, dres, scale, False)
    plain_db, plain_ds = ops.colsum2(plain_dx, x, scale)
    leaves = [t.double().requires_grad_(True) for t in (x, scale, bias, w)]
    wide = leaves[0] * (1.0 + leaves[1]) + leaves[2]
    z = wide * torch.rsqrt(wide.square().mean(-1, keepdim=True) + 1e-5) * leaves[3]
    ((z * dz.double()).sum() + (wide * dres.double()).sum()).backward()
    want_dx, want_ds, want_db, want_dw = (t.grad for t in leaves)
    on = scale != -1.0
    # sums of `rows` FP32 products of rounded factors: a few 2^-24 each, growing at most with the root of the count; dx of
    # the two kernels is the same formula with other contractions and xmod rounded once more, a few 2^-24 apart
    assert rel(dx, plain_dx.double()) < 1e-6 and rel(dx, want_dx) < 1e-5
    assert rel(grads[0], want_dw) < 1e-5 and rel(grads[1], want_db) < 1e-5
    assert rel(grads[2][on], want_ds[on]) < 1e-5
    assert torch.count_nonzero(grads[2][~on]) == 0
    # no further from FP64 than the separate pass, up to the noise of the last bits
    assert rel(grads[1][on], want_db[on]) <= 1.5 * rel(plain_db[on], want_db[on]) + 2e-7
    assert rel(grads[2][on], want_ds[on]) <= 1.5 * rel(plain_ds[on], want_ds[on]) + 2e-7
    assert rel(grads[0], want_dw) <= 1.5 * rel(plain_dw, want_dw) + 2e-7


@pytest.mark.parametrize("rows,d,near", [(5, 128, 1e-3), (593, 1280, 1e-3), (1024, 2048, 1e-5)])
def test_modulation_gradients_under_a_bias_that_hides_the_input(rows, d, near):
    """1 + scale down to ``near`` of 1 and biases of 1: xmod - bias keeps few bits of x * (1 + scale), x itself keeps all."""
    _ext.require()
    ops = torch.ops.ws_b200
    torch.manual_seed(rows + d)
    x = torch.randn(rows, d, device="cuda") * 0.3
    scale = near * (1.0 + torch.rand(d, device="cuda")) - 1.0
    scale[::5] = -1.0
    bias = 1.0 + torch.rand(d, device="cuda")
    w = 1.0 + 0.1 * torch.randn(d, device="cuda")
    dz, dres = torch.randn(rows, d, device="cuda").bfloat16(), torch.randn(rows, d, device="cuda")
    _, rstd, xmod = ops.rmsnorm_fwd(x, scale, bias, w, 1e-5, True)
    dx, grads = ops.rmsnorm_bwd_mod(dz, None, rstd, w, dres, scale, bias, x)
    plain_dx, _, _ = ops.rmsnorm_bwd(dz, xmod, rstd, w, dres, scale, False)
    _, plain_ds = ops.colsum2(plain_dx, x, scale)
    leaves = [t.double().requires_grad_(True) for t in (x, scale, bias, w)]
    wide = leaves[0] * (1.0 + leaves[1]) + leaves[2]
    z = wide * torch.rsqrt(wide.square().mean(-1, keepdim=True) + 1e-5) * leaves[3]
    ((z * dz.double()).sum() + (wide * dres.double()).sum()).backward()
    want_dx, want_ds, want_db, want_dw = (t.grad for t in leaves)
    # sums of FP32 products of rounded factors, as in the test above; a column that is switched off has its gradient, too
    assert rel(dx, want_dx) < 1e-5 and rel(grads[0], want_dw) < 1e-5 and rel(grads[1], want_db) < 1e-5
    assert rel(grads[2], want_ds) < 1e-5
    on = scale != -1.0                                       # the separate pass divides by 1 + scale
    assert rel(grads[2][on], want_ds[on]) <= 1.5 * rel(plain_ds[on], want_ds[on]) + 2e-7


def test_modulation_gradients_of_a_block_under_such_a_bias():
    """The whole block hands its input to the norm pass: the scale's gradient against the FP32 composite, column by column
    where 1 + scale is small."""
    from warpstate_ai_b200 import WarpStateConfig
    from warpstate_ai_b200.models.warpstate import WarpStateCore
    from warpstate_ai_b200.ops import fused
    torch.manual_seed(0)
    cfg = WarpStateConfig(vocab_size=64, d_model=128, n_heads=2, n_cores=1, logical_depth=1, ffn_hidden=192, chunk_size=128,
                          gradient_checkpointing=False, parallel_memory=True)
    with torch.device("cuda"):
        core = WarpStateCore(cfg)
    x, dy = torch.randn(2, 256, 128, device="cuda") * 0.3, torch.randn(2, 256, 128, device="cuda")
    scale, bias = torch.full((128,), 1e-5 - 1.0, device="cuda"), torch.ones(128, device="cuda")
    scale[:64] = 0.1

    def gradient(checkpoint):
        leaves = [t.clone().requires_grad_(True) for t in (x, scale, bias)]
        with torch.autocast("cuda", dtype=torch.bfloat16):
            out = fused.core_forward(core, *leaves, checkpoint=checkpoint)
        out.backward(dy)
        return leaves[1].grad

    leaves = [t.clone().requires_grad_(True) for t in (x, scale, bias)]
    with fused.disabled():
        core(*leaves).backward(dy)
    for checkpoint in (False, True):
        for part in (slice(0, 64), slice(64, 128)):
            # BF16 products inside the block: 2 % as for its other gradients; xmod - bias alone would be off by 1e-7 / 3e-6
            assert rel(gradient(checkpoint)[part], leaves[1].grad[part].double()) < 0.02, (checkpoint, part)
