"""Forward attention at head_dim 128 with a bias per key and valid lengths, where a lane stores its own row: ragged query tiles, contexts
without keys, strided inputs, and the fp32 copy of the output."""
import math

import pytest
import torch

from spiraltorch_b200.ops import attention as A
from spiraltorch_b200.ops import native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,Sq,Sk,H", [(3, 20, 20, 2), (2, 128, 257, 1), (150, 129, 129, 2), (2, 385, 300, 3)])
@pytest.mark.parametrize("extras", ["bias", "lengths", "both"])
def test_forward(B, Sq, Sk, H, extras):
    torch.manual_seed(Sq + Sk)
    qkv = torch.randn(3, B, max(Sq, Sk), H, 128, device="cuda").bfloat16()
    q, k, v = qkv[0][:, :Sq], qkv[1][:, :Sk], qkv[2][:, :Sk]
    bias = torch.randn(B, H, Sk, device="cuda") if extras != "lengths" else None
    lengths = torch.randint(0, Sk + 1, (B,), device="cuda", dtype=torch.int32) if extras != "bias" else None
    out32 = torch.full((B, Sq, H, 128), 7.0, device="cuda")
    o, lse = A.attention_forward(q, k, v, False, key_bias=bias, lengths=lengths, out32=out32)
    s = q.double().transpose(1, 2) @ k.double().transpose(1, 2).transpose(-1, -2) / math.sqrt(128)
    if bias is not None:
        s = s + bias.double()[:, :, None, :]
    live = torch.ones(B, Sq, dtype=torch.bool, device="cuda")
    if lengths is not None:
        s = s.masked_fill(torch.arange(Sk, device="cuda") >= lengths[:, None, None, None], -math.inf)
        live = torch.arange(Sq, device="cuda") < lengths[:, None]
    ref = torch.softmax(s, -1).nan_to_num() @ v.double().transpose(1, 2)
    ref = ref.transpose(1, 2) * live[..., None, None]
    assert not o[~live].any() and not out32[~live].any() and torch.isinf(lse.transpose(1, 2)[~live]).all()
    # P is rounded to bf16 (2^-9 of every product), and so is o
    assert (out32.double() - ref).norm() <= 2 * 2.0 ** -9 * ref.norm()
    assert (o.double() - ref).norm() <= 3 * 2.0 ** -9 * ref.norm()
    exact = torch.logsumexp(s, -1).transpose(1, 2)[live]
    assert (lse.transpose(1, 2)[live].double() - exact).abs().max() <= 1e-4       # ex2.approx and lg2.approx over up to 385 keys
    native.raise_on_device_error()
