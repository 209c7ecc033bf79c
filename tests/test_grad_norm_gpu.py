"""The gradient norm of an arena: finite sums against FP64, and what it reports where a sum leaves FP32."""
import math

import pytest
import torch

from warpstate_ai_b200.ops import _ext

pytestmark = pytest.mark.gpu

BLOCKS = 148 * 8


def stats_of(g):
    _ext.require()
    return torch.ops.ws_b200.grad_norm_clip(g, 1.0, None, None).tolist()[:4]


@pytest.mark.parametrize("n", [4, 4 * BLOCKS - 4, 4 * BLOCKS + 4, 1 << 22])
def test_finite_norm(n):
    torch.manual_seed(n)
    g = torch.randn(n, device="cuda") * 0.01
    norm, coef, square, skip = stats_of(g)
    want = float(g.double().norm())
    # four squares in FP32, the rest in FP64, one rounding of the sum and one of the root
    assert abs(norm - want) <= 2 ** -22 * want and abs(square - want * want) <= 2 ** -22 * want * want and skip == 0.0
    assert coef == pytest.approx(min(1.0, 1.0 / (want + 1e-6)), rel=1e-6)


@pytest.mark.parametrize("values", [{0: 2e19}, {0: math.inf}, {0: 1e19, 4: 1e19, 8: 1e19, 12: 1e19, 16: 1e19},
                                    {0: 1.5e19, 1 << 21: 1.5e19, (1 << 22) - 1: 1.5e19}])
def test_a_sum_past_fp32_is_reported_as_infinite(values):
    """One square, a block's sum (its remainder is inf - inf or -inf), or only the sum of the blocks."""
    g = torch.full((1 << 22,), 1e-3, device="cuda")
    for index, value in values.items():
        g[index] = value
    norm, coef, square, skip = stats_of(g)
    assert norm == math.inf and square == math.inf and coef == 0.0 and skip == 1.0


def test_a_nan_stays_one():
    g = torch.zeros(1 << 16, device="cuda")
    g[12345] = math.nan
    norm, coef, square, skip = stats_of(g)
    assert math.isnan(norm) and math.isnan(square) and coef == 0.0 and skip == 1.0
