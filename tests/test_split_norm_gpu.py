"""A block whose out_proj is cut along k: the kernel that adds the pieces does the second norm as well, with the results of the
two launches it replaces."""
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
    assert float((one - many).norm() / many.norm()) < 1e-6
