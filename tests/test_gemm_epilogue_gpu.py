"""Epilogues of the plain product at the edges of its tiles: outputs and operands through the copy engine, and the element-wise
accesses that stay where a leading dimension or an address does not allow it."""
import pytest
import torch

from spiraltorch_b200.ops import gemm as G
from spiraltorch_b200.ops import native

pytestmark = pytest.mark.gpu

# rows and columns below, at and past 32-, 64-, 128- and 256-wide blocks; several tiles per CTA; few tiles with a long K, whose K
# blocks two or four CTAs share (uneven shares, a last block that is not whole)
SHAPES = [(1, 8, 64), (31, 72, 40), (129, 136, 200), (257, 264, 520), (300, 1000, 136), (5000, 712, 72), (100, 136, 1096),
          (97, 520, 4104), (777, 1032, 2888), (1000, 264, 4616), (9000, 1288, 136)]


def _error(y, ref):
    return ((y.double() - ref).norm() / ref.norm()).item()


def _gelu_grad(x):
    x = x.double().requires_grad_(True)
    torch.nn.functional.gelu(x, approximate="tanh").sum().backward()
    return x.grad


@pytest.mark.parametrize("m,n,k", SHAPES)
@pytest.mark.parametrize("aligned", [True, False])
def test_epilogue_operands(m, n, k, aligned):
    torch.manual_seed(m + n)
    a, b = (torch.randn(r, k, device="cuda").bfloat16() for r in (m, n))

    def matrix(fill=None):        # a view whose rows are not 16 bytes apart needs the element-wise accesses
        t = torch.randn(m, n if aligned else n + 3, device="cuda").bfloat16()
        return (t if fill is None else t.fill_(fill))[:, :n]

    ref, x, u = a.double() @ b.double().t(), matrix(), matrix(7.0)
    bias = torch.randn(n, device="cuda").bfloat16()
    tol = 2.0 ** -8               # one rounding to bf16 is at most 2^-9 of a value
    assert _error(G.gemm(a, b, residual=x, out=matrix(7.0)), ref + x.double()) < tol
    assert _error(G.gemm(a, b, act="relu_bwd", aux_in=x, out=matrix(7.0)), ref * (x > 0)) < tol
    assert _error(G.gemm(a, b, act="gelu_bwd", aux_in=x, residual=u, out=matrix(7.0)), ref * _gelu_grad(x) + u.double()) < tol
    pre = ref + bias.double()
    assert _error(G.gemm(a, b, bias=bias, act="gelu", aux_out=u, out=matrix(7.0)), torch.nn.functional.gelu(pre, approximate="tanh")) < tol
    assert _error(u, pre) < tol
    native.raise_on_device_error()


@pytest.mark.parametrize("m,n,k", SHAPES)
@pytest.mark.parametrize("aligned", [True, False])
def test_fp32_outputs(m, n, k, aligned):
    torch.manual_seed(m + n)
    a, b = torch.randn(m, k, device="cuda").bfloat16(), torch.randn(n, k, device="cuda").bfloat16()
    ref, tol = a.double() @ b.double().t(), k * 2.0 ** -23        # every product added with one truncation to 24 bits
    out = torch.full((m, n if aligned else n + 1), 7.0, device="cuda")[:, :n]
    assert _error(G.gemm(a, b, out=out), ref) < tol
    first = out.double()
    assert _error(G.gemm(a, b, out=out, accumulate=True), first + ref) < tol + 2.0 ** -24
    whole = torch.randn(3, m, n, device="cuda")
    batched = whole.clone()
    G.gemm(a.expand(3, m, k).contiguous(), b.expand(3, n, k).contiguous(), out=batched, accumulate=True)
    assert _error(batched, whole.double() + ref) < tol + 2.0 ** -24
    native.raise_on_device_error()


@pytest.mark.parametrize("aligned", [True, False])
def test_added_results_keep_subnormal_numbers(aligned):
    """fp32 outputs that are added to, by the copy engine and element by element: no sum is flushed to zero."""
    a = torch.ones(256, 64, device="cuda").bfloat16()
    out = torch.full((256, 256 if aligned else 257), 1e-40, device="cuda")[:, :256]
    G.gemm(a, a, alpha=1e-41 / 64, out=out, accumulate=True)
    want = torch.full((), 1e-40) + torch.full((), 64.0) * torch.tensor(1e-41 / 64)
    # numbers are multiples of 2^-149 here; the scale, its product and the sum are off by half of one each, the scale's 64-fold
    assert (out.cpu().double() - want.double()).abs().max() <= 34 * 2.0 ** -149
    assert out.min() > 1.05e-40
    native.raise_on_device_error()
