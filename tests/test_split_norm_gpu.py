"""A block whose out_proj is cut along k: the kernel that adds the pieces does the second norm as well, with the results of the
two launches it replaces, bit for bit."""
import pytest
import torch

from warpstate_ai_b200 import WarpStateConfig
from warpstate_ai_b200.models.warpstate import WarpStateCore
from warpstate_ai_b200.ops import _ext, fused, gemm


@pytest.mark.gpu
@pytest.mark.parametrize("batch,d,ffn", [(1, 2048, 192), (3, 2048, 320), (1, 1024, 64)])
def test_block_with_a_cut_out_proj(monkeypatch, batch, d, ffn):
    torch.manual_seed(d + batch)
    cfg = WarpStateConfig(vocab_size=64, d_model=d, n_heads=d // 64, n_cores=1, logical_depth=1, ffn_hidden=ffn, chunk_size=128,
                          gradient_checkpointing=False, parallel_memory=True)
    with torch.device("cuda"):
        core = WarpStateCore(cfg)
        x = torch.randn(batch, 128, d)
        scale, bias = torch.randn(2, d).mul_(0.1).unbind(0)
        core.norm2.weight.data.normal_(1, 0.2)
    _ext.require()
    cut = _ext.cdll().ws_gemm_plan(128 * batch, d, d, 0, gemm.EPI_RESID_F32, 1, torch.cuda.get_device_properties(0).multi_processor_count) > 1
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        core(x, scale, bias)
        before = _ext.launch_count()
        one = core(x, scale, bias)
        launched = _ext.launch_count() - before
        monkeypatch.setattr(gemm, "_policy", {"fwd:0x0x0": {"kernel": "pair", "sm_limit": 0}})   # launch by launch, from Python
        before = _ext.launch_count()
        many = fused.core_forward(core, x, scale, bias)
        assert launched == _ext.launch_count() - before - (1 if cut else 0)
    gemm.check_device_errors()
    assert torch.equal(one, many)


@pytest.mark.gpu
@pytest.mark.parametrize("tokens,d", [(128, 2048), (256, 2048), (384, 2048), (128, 1280), (128, 1024)])
def test_the_second_norm_is_that_of_the_norm_kernel(tokens, d):
    """The factor is FP32, so an ulp of the sum of squares shows in it."""
    from warpstate_ai_b200.ops import attention
    torch.manual_seed(d + tokens)
    _ext.require()
    heads, ffn = d // 64, 64
    x, scale, bias = torch.randn(tokens, d, device="cuda"), *torch.randn(2, d, device="cuda").mul_(0.1).unbind(0)
    n1, n2 = torch.randn(2, d, device="cuda").mul_(0.2).add_(1).unbind(0)
    w_in, w_out, w_ug, w_down = ((torch.randn(n, k, device="cuda") * 0.03).bfloat16()
                                 for n, k in ((5 * d, d), (d, d), (2 * ffn, d), (d, ffn)))
    logits = torch.randn(3, heads, device="cuda").unbind(0)
    def block(w_out):
        return torch.ops.ws_b200.block_fwd(x, scale, bias, n1, w_in, w_out, n2, w_ug, w_down, *logits,
                                           attention.rope_table(x.device, pair_major=True), 1e-5, 1, tokens, heads, False, True,
                                           gemm.error_flag(x.device))
    x2, rstd2, z2 = block(w_out)[6:9]
    gemm.check_device_errors()
    with pytest.raises(RuntimeError, match="CUDA"):      # refused on the host, as by the two launches
        block(w_out.cpu())
    z, rstd, _ = torch.ops.ws_b200.rmsnorm_fwd(x2, None, None, n2, 1e-5, False)
    assert torch.equal(rstd2, rstd) and torch.equal(z2, z)
