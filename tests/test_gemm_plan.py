"""Which GEMM kernel a product takes (`ws_gemm_plan`), a function of its sizes that needs no GPU: on 148 SMs, at the edges of
each rule."""
import pytest

from warpstate_ai_b200.ops import _ext

BF16, RESID_F32, SWIGLU, ACC_F32, SWIGLU_BWD, F32, RESID_BF16, CE_FWD, CE_BWD = range(9)


@pytest.mark.parametrize("m,n,k,a_mn,epilogue,packed,plan", [
    (95, 2048, 2048, 0, RESID_F32, 1, 0), (255, 2048, 16384, 1, ACC_F32, 1, 0), (256, 2048, 16384, 1, ACC_F32, 1, 1),
    # short contractions: the single-CTA kernel, except for the epilogues that leave through shared memory
    (128, 1280, 256, 0, BF16, 1, 0), (128, 688, 256, 0, SWIGLU, 1, 0), (255, 32768, 256, 0, CE_FWD, 1, 0),
    (96, 256, 256, 0, RESID_F32, 1, 1), (96, 256, 256, 0, F32, 1, 1), (96, 688, 256, 0, SWIGLU_BWD, 1, 1),
    (128, 4480, 1280, 0, SWIGLU, 1, 1), (128, 4480, 1280, 0, SWIGLU, 0, 0), (128, 7168, 2048, 0, SWIGLU, 0, 1),
    (96, 10240, 2048, 0, BF16, 1, 1), (128, 6400, 1024, 0, BF16, 1, 1), (128, 6400, 1016, 0, BF16, 1, 0),
    # rounds over the chip: 74 tiles fit the pairs, 75 fit the SMs only; past 128 rows both kernels need two rounds
    (128, 74 * 256, 2048, 0, CE_FWD, 1, 1), (128, 74 * 256 + 8, 2048, 0, CE_FWD, 1, 0), (128, 32768, 2048, 0, CE_BWD, 1, 0),
    (129, 32768, 2048, 0, CE_BWD, 1, 1), (129, 32768, 2048, 0, BF16, 1, 1),
    # from 256 rows on always the pair kernel; cut along k where the pieces fit one round
    (256, 32768, 256, 0, BF16, 1, 1), (256, 688, 256, 0, SWIGLU, 0, 1), (300, 2048, 7168, 0, BF16, 1, 4),
    (128, 2048, 14336, 0, BF16, 1, 4), (300, 2048, 7168, 0, SWIGLU_BWD, 1, 1)])
def test_plan(m, n, k, a_mn, epilogue, packed, plan):
    if not _ext.load():
        pytest.skip("the kernel library cannot be built here")
    lib = _ext.cdll()
    assert lib.ws_gemm_plan(m, n, k, a_mn, epilogue, packed, 148) == plan
    assert lib.ws_gemm_plan(m, n, k, a_mn, epilogue, packed, 1) == 0
