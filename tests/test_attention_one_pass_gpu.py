"""Backward attention in one pass over the tile pairs (head_dim 64, up to eight key tiles) against 64 bits, at its edges: one, two
and three key tiles (one sum of dQ, one of two tiles, two sums), the last count it takes and the first it leaves to two passes,
other query than key lengths, contexts without keys; the same bits on every run."""
import ctypes
import math

import pytest
import torch

from spiraltorch_b200.ops import attention as A
from spiraltorch_b200.ops import native

pytestmark = pytest.mark.gpu


def _exact(q, k, v, g, causal, bias, lengths):
    q, k, v = (t.double().transpose(1, 2).requires_grad_(True) for t in (q, k, v))
    s = q @ k.transpose(-1, -2) / math.sqrt(q.shape[-1])
    keys, rows = torch.arange(k.shape[2], device=q.device), torch.arange(q.shape[2], device=q.device)
    if bias is not None:
        s = s + bias.double()[:, None, None, :]
    if causal:
        s = s.masked_fill(keys > rows[:, None], -1e30)
    if lengths is not None:
        s = s.masked_fill(keys >= lengths[:, None, None, None], -1e30)
    o = torch.softmax(s, -1) @ v
    if lengths is not None:
        o = o * (rows[:, None] < lengths[:, None, None, None])
    return [t.transpose(1, 2) for t in torch.autograd.grad(o, (q, k, v), g.double().transpose(1, 2))]


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("B,Sq,Sk,H,causal,extras", [(2, 128, 128, 3, True, False), (3, 200, 256, 2, False, True),
                                                     (2, 385, 385, 2, True, True), (150, 300, 257, 1, False, True),
                                                     (1, 1024, 1024, 2, True, False), (2, 100, 1025, 1, False, True)])
def test_gradients(B, Sq, Sk, H, causal, extras, f32):
    torch.manual_seed(Sq + Sk)
    q, g = (torch.randn(B, Sq, H, 64, device="cuda").bfloat16() for _ in range(2))
    k, v = (torch.randn(B, Sk, H, 64, device="cuda").bfloat16() for _ in range(2))
    bias = torch.randn(B, Sk, device="cuda") if extras else None
    lengths = torch.randint(0, min(Sq, Sk) + 1, (B,), device="cuda", dtype=torch.int32) if extras else None
    o, lse = A.attention_forward(q, k, v, causal, key_bias=bias, lengths=lengths)

    def run():
        dtype = torch.float32 if f32 else torch.bfloat16
        out = [torch.full(t.shape, 7.0, dtype=dtype, device="cuda") for t in (q, k, v)]
        return A.attention_backward(q, k, v, o, lse, g, causal, None, *out, key_bias=bias, lengths=lengths)

    got, again = run(), run()
    for x, y, ref in zip(got, again, _exact(q, k, v, g, causal, bias, lengths)):
        assert torch.equal(x, y)
        # P, dS, the output in delta and the result are rounded to bf16, 2^-9 each
        assert (x.double() - ref).norm() <= 4 * 2.0 ** -9 * ref.norm()
    native.raise_on_device_error()


def test_without_room_for_the_sums(monkeypatch):
    """Where their workspace cannot be had, the gradients come from two passes: the same but for the order of dQ's sum."""
    torch.manual_seed(0)
    q, k, v, g = (torch.randn(2, 300, 2, 64, device="cuda").bfloat16() for _ in range(4))
    o, lse = A.attention_forward(q, k, v, True)
    one = A.attention_backward(q, k, v, o, lse, g, True)
    empty = torch.empty

    def refuse(*size, **kw):
        if size[0] == q.numel() * 2 + 4:
            raise torch.cuda.OutOfMemoryError("no room")
        return empty(*size, **kw)

    monkeypatch.setattr(A.torch, "empty", refuse)
    for x, y in zip(one, A.attention_backward(q, k, v, o, lse, g, True)):
        assert (x.float() - y.float()).abs().max() <= 2 * 2.0 ** -8 * y.float().abs().max()     # one rounding to bf16 each
    native.raise_on_device_error()


def test_two_passes_without_the_room(monkeypatch):
    """The workspace is asked for once, by the size that the library names, and two passes follow its refusal."""
    torch.manual_seed(0)
    q, k, v, g = (torch.randn(2, 300, 2, 64, device="cuda").bfloat16() for _ in range(4))
    o, lse = A.attention_forward(q, k, v, True)
    one = A.attention_backward(q, k, v, o, lse, g, True)
    empty, refused = torch.empty, []
    workspace = native.lib().st_attn_bwd_workspace
    workspace.restype = ctypes.c_longlong
    room = workspace(*(ctypes.c_int(n) for n in (2, 2, 300, 300, 64)))
    assert room > 2 * q.numel()

    def refuse(*size, **kw):
        if size[0] == room:
            refused.append(room)
            raise torch.cuda.OutOfMemoryError("no room")
        return empty(*size, **kw)

    monkeypatch.setattr(A.torch, "empty", refuse)
    two = A.attention_backward(q, k, v, o, lse, g, True)
    assert refused == [room]
    for x, y in zip(one, two):
        assert (x.float() - y.float()).abs().max() <= 2 * 2.0 ** -8 * y.float().abs().max()     # one rounding to bf16 each
    native.raise_on_device_error()


def test_bits_do_not_depend_on_the_room_where_they_must_repeat(monkeypatch):
    monkeypatch.setenv("SPIRAL_DETERMINISTIC_REDUCTION", "1")
    torch.manual_seed(0)
    q, k, v, g = (torch.randn(2, 700, 2, 64, device="cuda").bfloat16() for _ in range(4))
    o, lse = A.attention_forward(q, k, v, True)
    want = A.attention_backward(q, k, v, o, lse, g, True)
    empty = torch.empty

    def refuse(*size, **kw):
        if kw.get("dtype") is torch.float32 and size[0] != tuple(lse.shape):
            raise torch.cuda.OutOfMemoryError("no room")
        return empty(*size, **kw)

    monkeypatch.setattr(A.torch, "empty", refuse)
    for x, y in zip(A.attention_backward(q, k, v, o, lse, g, True), want):
        assert torch.equal(x, y)
    native.raise_on_device_error()


@pytest.mark.parametrize("seq,room", [(256, 0), (257, 2)])
def test_room_for_fp32_gradients(seq, room):
    """Up to two key tiles fp32 gradients of the queries are the only sum, added to where they are; beyond, one per two tiles."""
    torch.manual_seed(0)
    q, k, v, g = (torch.randn(8, seq, 2, 64, device="cuda").bfloat16() for _ in range(4))
    o, lse = A.attention_forward(q, k, v, False)
    out = [torch.empty(t.shape, device="cuda") for t in (q, k, v)]
    got = [x.clone() for x in A.attention_backward(q, k, v, o, lse, g, False, None, *out)]
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    A.attention_backward(q, k, v, o, lse, g, False, None, *out)
    # beside the sums: one fp32 number per row, and blocks that are multiples of 512 bytes
    assert torch.cuda.max_memory_allocated() - before <= room * q.numel() * 4 + lse.numel() * 4 + 4096
    for x, ref in zip(got, _exact(q, k, v, g, False, None, None)):
        assert (x.double() - ref).norm() <= 4 * 2.0 ** -9 * ref.norm()
    native.raise_on_device_error()
