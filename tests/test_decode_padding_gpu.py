"""The decode projections pad a batch to the next of 16, 32, 48 and 64 rows: what a row gives does not depend on it."""
import pytest
import torch

from warpstate_ai_b200.ops import gemm


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [16, 17, 32, 33, 48, 49, 64])
@pytest.mark.parametrize("epilogue", [0, 1, 2, 3])
def test_what_rows_are_padded_to_changes_no_bit(rows, epilogue):
    from warpstate_ai_b200.ops import _ext
    _ext.require()
    torch.manual_seed(rows)
    ops, n, k = torch.ops.ws_b200, 640, 1088
    w = (torch.randn(2 * n if epilogue == 2 else n, k, device="cuda") * 0.05).bfloat16()
    x = torch.randn(rows, k, device="cuda").bfloat16()

    def product(part):
        shape = (ops.decode_gemm_splits(n, k), part.shape[0], n) if epilogue == 1 else (part.shape[0], n)
        out = torch.full(shape, float("nan"), device="cuda", dtype=torch.float32 if epilogue % 2 else torch.bfloat16)
        ops.decode_gemm(w, part.contiguous(), n, epilogue, out, gemm.error_flag(x.device))
        return out

    together, dim = product(x), 1 if epilogue == 1 else 0
    assert torch.equal(together, torch.cat([product(x[i:i + 9]) for i in range(0, rows, 9)], dim=dim))
    gemm.check_device_errors()
