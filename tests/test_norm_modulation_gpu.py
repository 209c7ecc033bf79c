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
    # sums of `rows` FP32 products of rounded factors: a few 2^-24 each, growing at most with the root of the count
    assert rel(dx, plain_dx.double()) < 1e-6 and rel(dx, want_dx) < 1e-5
    assert rel(grads[0], want_dw) < 1e-5 and rel(grads[1], want_db) < 1e-5
    assert rel(grads[2][on], want_ds[on]) < 1e-5
    assert torch.count_nonzero(grads[2][~on]) == 0
    # no further from FP64 than the separate pass, up to the noise of the last bits
    assert rel(grads[1][on], want_db[on]) <= 1.5 * rel(plain_db[on], want_db[on]) + 2e-7
    assert rel(grads[2][on], want_ds[on]) <= 1.5 * rel(plain_ds[on], want_ds[on]) + 2e-7
    assert rel(grads[0], want_dw) <= 1.5 * rel(plain_dw, want_dw) + 2e-7
