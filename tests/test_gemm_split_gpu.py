"""Products that are cut along the contraction, and few-row products on the CTA-pair kernel, against FP32: the pieces'
edges (a ragged last piece, k not a multiple of the k-block), ragged rows and every epilogue that can be cut."""
import pytest
import torch

from warpstate_ai_b200.ops import _ext, gemm as G

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float((a.float() - b).norm() / b.norm().clamp_min(1e-12))


@pytest.mark.parametrize("m", [96, 128, 129, 255, 300, 777, 1792])
@pytest.mark.parametrize("n,k", [(256, 7168), (2048, 7168), (1280, 8960), (264, 4104), (520, 6400)])
def test_long_contractions(m, n, k):
    # FP32 accumulation in another order than the oracle's: 1e-4 as for the uncut product; BF16 outputs round once more
    _ext.require()
    torch.manual_seed(m + n + k)
    x, w = torch.randn(m, k, device="cuda").bfloat16(), (torch.randn(n, k, device="cuda") * 0.05).bfloat16()
    ref = x.float() @ w.float().T
    scale = torch.rand(m, device="cuda") + 0.5
    resid = torch.randn(m, n, device="cuda") * 10
    assert rel(G.linear(x, w), ref) < 0.004
    assert rel(G.linear(x, w, row_scale=scale), ref * scale[:, None]) < 0.004
    assert rel(G.linear_f32(x, w), ref) < 1e-4
    assert rel(G.linear_residual(x, w, resid), ref + resid) < 1e-4
    assert rel(G.linear_residual(x, w, resid.bfloat16()), ref + resid.bfloat16().float()) < 0.008
    wt = (torch.randn(k, n, device="cuda") * 0.05).bfloat16()
    assert rel(G.grad_input(x, wt), x.float() @ wt.float()) < 0.004
    out = torch.full((m + 2, n), float("nan"), device="cuda", dtype=torch.bfloat16)      # nothing past the rows asked for
    G.linear(x, w, out=out[1:m + 1])
    G.check_device_errors()
    assert torch.isnan(out[0].float()).all() and torch.isnan(out[m + 1].float()).all() and rel(out[1:m + 1], ref) < 0.004


def test_runs_agree_bit_for_bit():
    _ext.require()
    torch.manual_seed(0)
    x, w = torch.randn(300, 7168, device="cuda").bfloat16(), torch.randn(2048, 7168, device="cuda").bfloat16()
    first = G.linear(x, w)
    assert all(torch.equal(G.linear(x, w), first) for _ in range(3))


BF16, RESID_F32, SWIGLU, ACC_F32, SWIGLU_BWD, F32, RESID_BF16, CE_FWD = range(8)


@pytest.mark.parametrize("m,n,k,epilogue,pieces", [
    (300, 2048, 7168, BF16, 4), (300, 2048, 7168, RESID_F32, 4), (777, 1280, 8960, BF16, 3), (1792, 1280, 8960, BF16, 2),
    (129, 264, 4104, BF16, 4), (128, 2048, 2048, RESID_BF16, 4),       # long contractions of few tiles
    (2048, 2048, 7168, BF16, 1), (1792, 2048, 7168, BF16, 1),          # two pieces would take a second round
    (300, 2048, 1024, BF16, 1), (300, 2048, 7168, F32, 1)])
def test_which_products_are_cut(m, n, k, epilogue, pieces):
    """The plan, and that the launches follow it: a cut product is the grouped launch and the one that adds its pieces."""
    _ext.require()
    assert _ext.cdll().ws_gemm_plan(m, n, k, 0, epilogue, 1, 148) == pieces
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the launches below are those of 148 SMs")
    x, w = torch.randn(m, k, device="cuda").bfloat16(), torch.randn(n, k, device="cuda").bfloat16()
    resid = torch.randn(m, n, device="cuda")
    before = _ext.launch_count()
    if epilogue == BF16:
        G.linear(x, w)
    elif epilogue == F32:
        G.linear_f32(x, w)
    else:
        G.linear_residual(x, w, resid if epilogue == RESID_F32 else resid.bfloat16())
    assert _ext.launch_count() - before == (2 if pieces > 1 else 1)
    G.check_device_errors()
