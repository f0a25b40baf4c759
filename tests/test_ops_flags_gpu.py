"""Switches of the operators may be any number: numpy's truth values, as comparisons of arrays give them, and plain 0 and 1."""
import numpy as np
import pytest
import torch

from spiraltorch_b200.ops import elementwise as E
from spiraltorch_b200.ops import gemm as G
from spiraltorch_b200.ops import norm as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flag", [np.bool_, int, float, np.float32, torch.tensor])
@pytest.mark.parametrize("on", [False, True])
def test_any_truth_value(flag, on):
    torch.manual_seed(0)
    a, b = torch.randn(64, 64, device="cuda").bfloat16(), torch.randn(64, 64, device="cuda").bfloat16()
    gamma = torch.randn(64, device="cuda").bfloat16()

    def run(x):
        y, _, mean, rstd = N.norm_forward(a, gamma, None, 1e-5, x)
        dgamma, dbeta = torch.ones(64, device="cuda"), torch.ones(64, device="cuda")
        dx = N.norm_backward(b, a, gamma, mean, rstd, x, dgamma, dbeta, x)
        return (G.gemm(a, b, a_mn=x, b_mn=x), E.rope_(a.clone(), 4, 16, 8, backward=x), y, dx, dgamma)

    for got, want in zip(run(flag(on)), run(on)):
        assert torch.equal(got, want)
