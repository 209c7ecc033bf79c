"""Products of few tokens with the weights in the MMA's rows: which products take the kernel (CPU), and its results at the
edges of its tiles, against the products themselves."""
import pytest
import torch

from warpstate_ai_b200.ops import _ext

BF16, RESID_F32, SWIGLU = 0, 1, 2


@pytest.mark.parametrize("m,n,k,epilogue,packed,takes", [
    (95, 10240, 2048, BF16, 1, 0), (96, 10240, 2048, BF16, 1, 1), (128, 10240, 2048, BF16, 1, 1), (224, 10240, 2048, BF16, 1, 1), (256, 10240, 2048, BF16, 1, 0),
    (257, 10240, 2048, BF16, 1, 1), (300, 10240, 2048, BF16, 1, 1), (384, 10240, 2048, BF16, 1, 1), (448, 10240, 2048, BF16, 1, 1), (512, 10240, 2048, BF16, 1, 0),
    (513, 10240, 2048, BF16, 1, 0), (300, 7168, 2048, SWIGLU, 0, 1), (300, 7168, 2048, SWIGLU, 1, 0), (300, 6400, 1280, BF16, 1, 0),
    (128, 6400, 1280, BF16, 1, 1), (128, 4480, 1280, SWIGLU, 0, 1), (160, 4480, 1280, SWIGLU, 0, 0), (192, 7168, 2048, SWIGLU, 0, 1), (224, 7168, 2048, SWIGLU, 0, 0), (128, 10240, 1016, BF16, 1, 0), (128, 10240, 2048, RESID_F32, 1, 0),
    (129, 264, 4104, BF16, 1, 0),          # cut along k instead
    # twice the rounds of the single-CTA kernel; less than that; as many
    (128, 32768, 2048, BF16, 1, 0), (96, 20480, 4096, BF16, 1, 0), (128, 10752, 3072, SWIGLU, 0, 0), (128, 37888, 2048, BF16, 1, 0),
    (128, 37896, 2048, BF16, 1, 1), (96, 60000, 2048, BF16, 1, 0), (160, 32768, 2048, BF16, 1, 1), (128, 18944, 2048, BF16, 1, 1), (128, 18952, 2048, BF16, 1, 0)])
def test_which_products_take_it(m, n, k, epilogue, packed, takes):
    if not _ext.load():
        pytest.skip("the kernel library cannot be built here")
    lib = _ext.cdll()
    assert lib.ws_gemm_rows_takes(m, n, k, epilogue, packed, 148) == takes
    assert lib.ws_gemm_rows_takes(m, n, k, epilogue, packed, 1) == 0


def product(m, n, k, epilogue):
    torch.manual_seed(m + n)
    x = torch.randn(m, k, device="cuda").bfloat16()
    w = (torch.randn((2 if epilogue == SWIGLU else 1) * n, k, device="cuda") / k ** 0.5).bfloat16()
    return x, w, x.double() @ w.double().T, k * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(96, 10240, 1024), (128, 6400, 1088), (129, 4104, 1280), (257, 9480, 2048), (300, 10240, 2048),
                                   (320, 10008, 1032), (321, 10248, 1024), (160, 19208, 1024)])
def test_bf16_results(m, n, k):
    from warpstate_ai_b200.ops import gemm
    _ext.require()
    assert _ext.cdll().ws_gemm_rows_takes(m, n, k, BF16, 1, torch.cuda.get_device_properties(0).multi_processor_count)
    x, w, want, error = product(m, n, k, BF16)
    wide = torch.randn(m, n + 24, device="cuda").bfloat16()
    before = wide.clone()
    torch.ops.ws_b200.gemm(x, w, False, False, BF16, m, n, k, wide[:, :n], None, None, None, 1.0, 0.0, gemm.error_flag(x.device))
    gemm.check_device_errors()
    assert ((wide[:, :n].double() - want).abs() <= 2.0 ** -8 * want.abs() + error).all()
    assert torch.equal(wide[:, n:], before[:, n:])


@pytest.mark.gpu
@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("m,h,k", [(96, 4480, 1280), (160, 7168, 2048), (290, 7168, 2048), (384, 7240, 1088)])
def test_swiglu_without_up_and_gate(m, h, k, wide):
    """One BF16 rounding of silu(gate) up behind FP32 arithmetic (2^-10 of it: the sigmoid's approximation), and of up and
    gate before where they are rounded."""
    from warpstate_ai_b200.ops import gemm
    _ext.require()
    assert _ext.cdll().ws_gemm_rows_takes(m, h, k, SWIGLU, 0, torch.cuda.get_device_properties(0).multi_processor_count)
    x, w, both, _ = product(m, h, k, SWIGLU)
    act = torch.full((m, h), float("nan"), device="cuda", dtype=torch.bfloat16)
    torch.ops.ws_b200.gemm(x, w, False, False, SWIGLU, m, h, k, None, act, None, None, 1.0, 0.0, gemm.error_flag(x.device), wide)
    gemm.check_device_errors()
    up, gate = both[:, :h], both[:, h:]
    want = up * gate * torch.sigmoid(gate)
    slope = 1.1 * (up.abs() + 1)                       # of silu, and what an error of gate's sum does to the product
    bound = (2.0 ** -8 * (1 if wide else 3) + 2.0 ** -9) * want.abs() + slope * (2.0 ** -9 * gate.abs() * (0 if wide else 1) + 1e-5)
    assert ((act.double() - want).abs() <= bound + 2.0 ** -10 * up.abs()).all()


@pytest.fixture
def settings():
    """(SM limit, CTA pairs or not) of the library, put back afterwards."""
    lib = _ext.cdll()
    def set_to(sms=0, pairs=-1):
        lib.ws_gemm_set_sm_limit(sms)
        lib.ws_gemm_set_pair_mode(pairs)
    yield set_to
    set_to()


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k,epilogue,sms", [
    (300, 32768, 2048, BF16, 148), (320, 19208, 1024, BF16, 148), (128, 40000, 1024, BF16, 148), (300, 9600, 2048, SWIGLU, 148),
    (300, 4104, 1024, BF16, 20), (160, 1288, 1024, BF16, 4), (257, 1288, 1088, BF16, 2), (300, 2056, 2048, SWIGLU, 8), (160, 2056, 2048, SWIGLU, 4)])
def test_several_tiles_to_a_pair(settings, m, n, k, epilogue, sms):
    """One accumulator (above 256 tokens) or two are filled again, and the SwiGLU warps' exchange goes on from tile to tile.  The
    results are those of the single-CTA kernel, which has the tokens in its rows and stores row by row, bit for bit."""
    from warpstate_ai_b200.ops import gemm
    lib = _ext.cdll()
    sms = min(sms, torch.cuda.get_device_properties(0).multi_processor_count)
    settings(sms=sms)
    assert lib.ws_gemm_rows_takes(m, n, k, epilogue, 0, sms)
    assert (n + (255 if epilogue == BF16 else 127)) // (256 if epilogue == BF16 else 128) > sms // 2
    x, w, want, error = product(m, n, k, epilogue)
    def run():
        return gemm.linear(x, w) if epilogue == BF16 else gemm.linear_swiglu(x, w, want_packed=False, wide=True)[1]
    got = run()
    settings(pairs=0)
    assert torch.equal(got, run())
    gemm.check_device_errors()
    if epilogue == BF16:
        assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + error).all()
