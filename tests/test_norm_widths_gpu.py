"""RMSNorm forward by each of its kernels (a block per row where rows are few, a warp that holds the row in registers past that,
for every width up to 2048, and the general one for wider rows), which agree bit for bit, and column sums of many partial rows."""
import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("modulated", [False, True])
@pytest.mark.parametrize("rows,d", [(1, 256), (9, 1280), (1792, 1280), (513, 256), (7, 384), (300, 2048), (1184, 1920), (1185, 256),
                                    (1300, 384), (1185, 2048), (10000, 128), (3, 2176), (1300, 2176), (9600, 4096)])
def test_forward(rows, d, modulated, dtype):
    from warpstate_ai_b200.ops import _ext
    _ext.require()
    torch.manual_seed(rows)
    x = torch.randn(rows, d, device="cuda").to(dtype)
    scale, bias, w = (torch.randn(d, device="cuda") * 0.2 for _ in range(3))
    w += 1
    z, rstd, xmod = torch.ops.ws_b200.rmsnorm_fwd(x, scale if modulated else None, bias if modulated else None, w, 1e-5, True)
    want = x.double() * (1 + scale.double()) + bias.double() if modulated else x.double()
    if dtype is torch.bfloat16 and modulated:
        want = xmod.double()                                   # rounded to the stream's type first
    assert torch.allclose(xmod.double(), want, rtol=2e-6, atol=2e-6)
    factor = torch.rsqrt(want.square().mean(-1, keepdim=True) + 1e-5)
    assert torch.allclose(rstd.double()[:, None], factor, rtol=1e-5)
    # FP32 stream: one rounding to BF16; BF16 stream: the normalised value, the weight and their product are rounded
    roundings = 1 if dtype is torch.float32 else 3
    assert ((z.double() - want * factor * w.double()).abs() <= roundings * 2.0 ** -8 * (want * factor * w.double()).abs() + 1e-6).all()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("modulated", [False, True])
@pytest.mark.parametrize("d", range(128, 2049, 128))
def test_few_rows_and_many_give_the_same(d, modulated, dtype):
    from warpstate_ai_b200.ops import _ext
    _ext.require()
    torch.manual_seed(d)
    x = torch.randn(1185, d, device="cuda").to(dtype)
    scale, bias, w = (torch.randn(d, device="cuda") * 0.2 for _ in range(3))
    mod = (scale, bias) if modulated else (None, None)
    many = torch.ops.ws_b200.rmsnorm_fwd(x, *mod, w, 1e-5, True)
    for rows in (1184, 297, 296, 1):
        few = torch.ops.ws_b200.rmsnorm_fwd(x[-rows:], *mod, w, 1e-5, True)
        for a, b in zip(many, few):
            assert torch.equal(a[-rows:], b)


@pytest.mark.gpu
@pytest.mark.parametrize("rows,d", [(1, 256), (31, 1280), (129, 2048), (5000, 1280)])
def test_weight_gradient_sums(rows, d):
    from warpstate_ai_b200.ops import _ext
    _ext.require()
    torch.manual_seed(rows)
    x, dres = torch.randn(rows, d, device="cuda"), torch.randn(rows, d, device="cuda")
    dz, w = torch.randn(rows, d, device="cuda").bfloat16(), torch.randn(d, device="cuda")
    rstd = torch.rsqrt(x.square().mean(-1) + 1e-5)
    _, _, dw = torch.ops.ws_b200.rmsnorm_bwd(dz, x, rstd, w, dres, None, True)
    terms = dz.double() * x.double() * rstd.double()[:, None]
    assert ((dw.double() - terms.sum(0)).abs() <= rows * 2.0 ** -23 * terms.abs().sum(0) + 1e-6).all()
