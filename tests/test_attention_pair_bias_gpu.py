"""Backward attention at head_dim 64 with a bias per (query, key), whose gradients leave through the tile of dS: more work items than SMs,
so that a CTA stages the gradients of one item while it starts the next, ragged tiles, and contexts without keys among them."""
import math

import pytest
import torch

from spiraltorch_b200.ops import attention as A
from spiraltorch_b200.ops import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("B,Sq,Sk,H,causal,lengths", [(1, 1, 1, 1, False, False), (90, 130, 130, 2, True, False), (60, 257, 257, 2, False, True),
                                                      (200, 31, 160, 1, False, False), (80, 128, 128, 4, True, True)])
def test_gradients(B, Sq, Sk, H, causal, lengths, f32):
    torch.manual_seed(B + Sq)
    q, g = (torch.randn(B, Sq, H, 64, device="cuda").bfloat16() for _ in range(2))
    k, v = (torch.randn(B, Sk, H, 64, device="cuda").bfloat16() for _ in range(2))
    bias = torch.randn(B, Sq, Sk, device="cuda")
    n = torch.randint(0, min(Sq, Sk) + 1, (B,), device="cuda", dtype=torch.int32) if lengths else None
    o, lse = A.attention_forward(q, k, v, causal, attn_bias=bias, lengths=n)
    out = [torch.full(t.shape, 7.0, dtype=torch.float32 if f32 else torch.bfloat16, device="cuda") for t in (q, k, v)]
    got = A.attention_backward(q, k, v, o, lse, g, causal, None, *out, attn_bias=bias, lengths=n)
    qd, kd, vd = (t.double().transpose(1, 2).requires_grad_(True) for t in (q, k, v))
    s = qd @ kd.transpose(-1, -2) / math.sqrt(64) + bias.double()[:, None]
    keys, rows = torch.arange(Sk, device="cuda"), torch.arange(Sq, device="cuda")
    if causal:
        s = s.masked_fill(keys > rows[:, None], -1e30)
    if lengths:
        s = s.masked_fill(keys >= n[:, None, None, None], -1e30)
    y = torch.softmax(s, -1) @ vd
    if lengths:
        y = y * (rows[:, None] < n[:, None, None, None])
    for x, ref in zip(got, torch.autograd.grad(y, (qd, kd, vd), g.double().transpose(1, 2))):
        # P, dS, the output in delta and the result are rounded to bf16, 2^-9 each; a single key has no gradient but through v
        ref = ref.transpose(1, 2)
        assert (x.double() - ref).norm() <= 4 * 2.0 ** -9 * ref.norm() + (2.0 ** -6 if Sk == 1 else 0.0) * g.double().norm()
    native.raise_on_device_error()
