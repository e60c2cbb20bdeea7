"""The gate function of the MoE layer's kernels against the compiler's division and against float64."""
import pytest
import torch

from open_cake_ir_b200 import _lib

pytestmark = pytest.mark.gpu


def silu(x):
    y, by_division = torch.empty_like(x), torch.empty_like(x)
    assert _lib.library().cake_b200_test_silu(x.data_ptr(), y.data_ptr(), by_division.data_ptr(), x.numel(), torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    return y, by_division


def test_within_an_ulp_of_the_division():
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.cat([torch.randn(1 << 20, device="cuda", generator=g) * s for s in (1e-30, 1e-6, 1e-2, 1.0, 8.0, 30.0, 1e6, 1e30)])
    x = x[x > -80]                     # the quotient is a normal number
    y, by_division = silu(x)
    ulps = (y.view(torch.int32).long() - by_division.view(torch.int32).long()).abs()
    assert int(ulps.max()) <= 1
    # the exponential's own error: 2 + |1.16 x| ulp of exp(-x), which enters the quotient at most in full; and the roundings of the sum and the quotient
    exact = x.double() / (1 + torch.exp(-x.double()))
    bound = (2 + 1.16 * x.double().abs().clamp(max=88) + 2) * 2.0 ** -23
    assert bool(((y.double() - exact).abs() <= bound * exact.abs() + 1e-44).all())


def test_ends_of_the_range():
    x = torch.tensor([0.0, -0.0, 88.0, 3e38, float("inf"), -87.0, -88.0, -200.0, -1e30, float("nan")], device="cuda")
    y, _ = silu(x)
    assert y[:2].tolist() == [0.0, 0.0] and y[2:5].tolist() == x[2:5].tolist() and bool(torch.isnan(y[9]))
    assert bool((y[5:9] <= 0).all()) and bool((y[5:9] >= x[5:9] * 1.7e-38).all())        # x e^-87 and smaller in place of what vanishes
