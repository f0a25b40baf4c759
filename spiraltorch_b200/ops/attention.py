"""Scaled-dot-product attention, forward and backward, on the tcgen05 kernels
(``csrc/attention/attn_fwd.cu``, ``csrc/attention/attn_bwd.cu``).

Tensors are ``[B, S, H, D]`` views (D contiguous, any B/S/H strides), so Q, K and V can be
slices of one fused QKV projection output and O feeds the output projection without a copy.
CPU tensors use an fp32 PyTorch statement of the same math (also the test oracle).

Reference parity: ``Tensor::scaled_dot_attention`` (crates/st-tensor/src/pure.rs:4061-4157,
online-softmax ``fused_attention_cpu`` :11845-11919); the backward has no counterpart in
the reference (its attention is forward-only).
"""
from __future__ import annotations

import ctypes
import functools
import math
import os
from typing import Optional

import torch

from . import native

launch_count = 0


class _FwdArgs(ctypes.Structure):
    _fields_ = [(n, ctypes.c_void_p) for n in ("Q", "K", "V", "O", "lse")] + \
               [(n, ctypes.c_longlong) for n in ("q_sb", "q_ss", "q_sh", "k_sb", "k_ss", "k_sh",
                                                "v_sb", "v_ss", "v_sh", "o_sb", "o_ss", "o_sh")] + \
               [(n, ctypes.c_int) for n in ("B", "H", "Sq", "Sk", "D")] + \
               [("scale", ctypes.c_float), ("causal", ctypes.c_int)] + \
               [("key_bias", ctypes.c_void_p), ("kb_sb", ctypes.c_longlong), ("kb_sh", ctypes.c_longlong),
                ("attn_bias", ctypes.c_void_p), ("ab_sb", ctypes.c_longlong), ("ab_sh", ctypes.c_longlong),
                ("ab_sq", ctypes.c_longlong), ("lengths", ctypes.c_void_p)]


class _BwdArgs(ctypes.Structure):
    _fields_ = [(n, ctypes.c_void_p) for n in ("Q", "K", "V", "O", "dO", "lse", "delta", "dQ_acc",
                                               "dQ", "dK", "dV")] + \
               [(n, ctypes.c_longlong) for n in ("q_sb", "q_ss", "q_sh", "k_sb", "k_ss", "k_sh",
                                                "v_sb", "v_ss", "v_sh", "o_sb", "o_ss", "o_sh",
                                                "do_sb", "do_ss", "do_sh",
                                                "dq_sb", "dq_ss", "dq_sh", "dk_sb", "dk_ss", "dk_sh",
                                                "dv_sb", "dv_ss", "dv_sh")] + \
               [(n, ctypes.c_int) for n in ("B", "H", "Sq", "Sk", "D")] + \
               [("scale", ctypes.c_float), ("causal", ctypes.c_int)] + \
               [("key_bias", ctypes.c_void_p), ("kb_sb", ctypes.c_longlong), ("kb_sh", ctypes.c_longlong),
                ("attn_bias", ctypes.c_void_p), ("ab_sb", ctypes.c_longlong), ("ab_sh", ctypes.c_longlong),
                ("ab_sq", ctypes.c_longlong), ("lengths", ctypes.c_void_p)]


def attention_reference(q, k, v, causal: bool, scale: float, bias: Optional[torch.Tensor] = None,
                        key_bias: Optional[torch.Tensor] = None, attn_bias: Optional[torch.Tensor] = None,
                        lengths: Optional[torch.Tensor] = None):
    """fp32 reference: q,k,v ``[B,S,H,D]`` → (o ``[B,S,H,D]`` fp32, lse ``[B,H,S]``).

    ``key_bias`` ``[B, Sk]`` or ``[B, H, Sk]`` and ``attn_bias`` ``[B, Sq, Sk]`` or ``[B, H, Sq, Sk]`` are added
    to ``scale * q·kᵀ``; with ``lengths`` ``[B]`` keys at or beyond the length are masked and queries at or
    beyond it give zero rows (crates/st-core/src/backend/cuda_attention.cu:117-202)."""
    qf, kf, vf = (t.float().permute(0, 2, 1, 3) for t in (q, k, v))
    s = torch.matmul(qf, kf.transpose(-1, -2)) * scale
    if bias is not None:
        s = s + bias
    if key_bias is not None:
        kb = key_bias.float()
        s = s + (kb[:, None, None, :] if kb.dim() == 2 else kb[:, :, None, :])
    if attn_bias is not None:
        ab = attn_bias.float()
        s = s + (ab[:, None] if ab.dim() == 3 else ab)
    sq, sk = s.shape[-2:]
    if causal:
        mask = torch.ones(sq, sk, dtype=torch.bool, device=s.device).tril(sk - sq)
        s = s.masked_fill(~mask, float("-inf"))
    if lengths is not None:
        ln = lengths.to(s.device).view(-1, 1, 1, 1)
        dead = (torch.arange(sk, device=s.device).view(1, 1, 1, sk) >= ln) | \
               (torch.arange(sq, device=s.device).view(1, 1, sq, 1) >= ln)
        s = s.masked_fill(dead, float("-inf"))
    lse = torch.logsumexp(s, dim=-1)
    p = torch.exp(s - lse.unsqueeze(-1))
    p = torch.where(torch.isfinite(lse).unsqueeze(-1), p, torch.zeros_like(p))     # fully masked rows → zeros
    o = torch.matmul(p, vf).permute(0, 2, 1, 3)
    return o, lse


def _bias_args(a, q, k, key_bias, attn_bias, lengths, keep: list) -> None:
    """Fill the bias / length fields of an argument block (fp32 biases, int32 lengths, keys contiguous)."""
    B, Sq, H, _ = q.shape
    Sk = k.shape[1]
    if key_bias is not None:
        kb = key_bias.to(torch.float32)
        if kb.shape not in ((B, Sk), (B, H, Sk)):
            raise ValueError(f"attention: key_bias must be [B, Sk] or [B, H, Sk], got {tuple(kb.shape)}")
        kb = kb.contiguous()
        keep.append(kb)
        a.key_bias = kb.data_ptr()
        a.kb_sb, a.kb_sh = kb.stride(0), (kb.stride(1) if kb.dim() == 3 else 0)
    if attn_bias is not None:
        ab = attn_bias.to(torch.float32)
        if ab.shape not in ((B, Sq, Sk), (B, H, Sq, Sk)):
            raise ValueError(f"attention: attn_bias must be [B, Sq, Sk] or [B, H, Sq, Sk], got {tuple(ab.shape)}")
        ab = ab.contiguous()
        keep.append(ab)
        a.attn_bias = ab.data_ptr()
        a.ab_sb, a.ab_sh, a.ab_sq = ab.stride(0), (ab.stride(1) if ab.dim() == 4 else 0), ab.stride(-2)
    if lengths is not None:
        ln = lengths.to(device=q.device, dtype=torch.int32).contiguous()
        if ln.shape != (B,):
            raise ValueError(f"attention: lengths must be [B], got {tuple(ln.shape)}")
        keep.append(ln)
        a.lengths = ln.data_ptr()


def set_pair_kernel(on: bool) -> None:
    """Forward attention without a bias per (query, key) runs the pair kernel by default, where its pairs fill the chip:
    two 128-row query tiles per CTA share every K / V tile, with the probabilities and the output accumulator in tensor
    memory.  ``False`` selects the single-tile kernel for every case."""
    native.lib().st_attn_fwd_set_pair_kernel(1 if on else 0)


def pair_kernel_enabled() -> bool:
    return bool(native.lib().st_attn_fwd_get_pair_kernel())


_env_applied = False


def _apply_env_once() -> None:
    """``ST_ATTN_FWD_PAIR=0`` in the environment selects the single-tile forward kernel for the whole process."""
    global _env_applied
    if not _env_applied:
        _env_applied = True
        v = os.environ.get("ST_ATTN_FWD_PAIR")
        if v is not None:
            set_pair_kernel(v.strip().lower() not in ("0", "false", "off", ""))


def _check_layout(t: torch.Tensor, name: str) -> None:
    if t.dim() != 4 or t.stride(-1) != 1 or t.dtype != torch.bfloat16:
        raise ValueError(f"{name} must be a bf16 [B,S,H,D] view with contiguous D")


def _check_shapes(q, k, v) -> None:
    """K and V must agree with each other and with Q's batch, heads and head dimension: the kernel sizes every
    access from Q's B/H/D and K's length, so a smaller K or V would be read past its allocation."""
    if k.shape != v.shape:
        raise ValueError(f"attention: k {tuple(k.shape)} and v {tuple(v.shape)} differ")
    if k.dim() != 4 or q.dim() != 4 or (k.shape[0], k.shape[2], k.shape[3]) != (q.shape[0], q.shape[2], q.shape[3]):
        raise ValueError(f"attention: k/v {tuple(k.shape)} do not match q {tuple(q.shape)} in batch, heads or head_dim")


def _bias_workspace(q, k, key_bias, attn_bias, lengths) -> Optional[torch.Tensor]:
    """Room for the padded key-bias rows of the kernels that take a key bias or lengths without a bias per (query, key)."""
    if attn_bias is not None or (key_bias is None and lengths is None):
        return None
    lib = native.lib()
    lib.st_attn_bias_workspace.restype = ctypes.c_longlong
    n = lib.st_attn_bias_workspace(ctypes.c_int(q.shape[0]), ctypes.c_int(q.shape[2]), ctypes.c_int(k.shape[1]))
    return torch.empty(n, dtype=torch.float32, device=q.device)


def attention_forward(q, k, v, causal: bool = True, scale: Optional[float] = None, *,
                      key_bias: Optional[torch.Tensor] = None, attn_bias: Optional[torch.Tensor] = None,
                      lengths: Optional[torch.Tensor] = None, out32: Optional[torch.Tensor] = None):
    """Returns ``(o, lse)``; ``o`` is contiguous ``[B,S,H,D]`` bf16, ``lse`` fp32 ``[B,H,S]``.
    Optional additive biases and valid lengths as in :func:`attention_reference`.  ``out32`` (CUDA, contiguous fp32 of
    ``o``'s shape, pair kernel) also receives the output before it is rounded."""
    global launch_count
    B, Sq, H, D = q.shape
    Sk = k.shape[1]
    scale = 1.0 / math.sqrt(D) if scale is None else scale
    if not native.use_native(q):
        o, lse = attention_reference(q, k, v, causal, scale, key_bias=key_bias, attn_bias=attn_bias, lengths=lengths)
        return o.to(q.dtype).contiguous(), lse
    native.require_cuda("attention_forward", q, k, v, key_bias, attn_bias, lengths)
    _apply_env_once()
    _check_shapes(q, k, v)
    for t, n in ((q, "q"), (k, "k"), (v, "v")):
        _check_layout(t, n)
    o = torch.empty((B, Sq, H, D), dtype=torch.bfloat16, device=q.device)
    lse = torch.empty((B, H, Sq), dtype=torch.float32, device=q.device)
    a = _FwdArgs()
    a.Q, a.K, a.V, a.O, a.lse = q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), lse.data_ptr()
    a.q_sb, a.q_ss, a.q_sh = q.stride(0), q.stride(1), q.stride(2)
    a.k_sb, a.k_ss, a.k_sh = k.stride(0), k.stride(1), k.stride(2)
    a.v_sb, a.v_ss, a.v_sh = v.stride(0), v.stride(1), v.stride(2)
    a.o_sb, a.o_ss, a.o_sh = o.stride(0), o.stride(1), o.stride(2)
    a.B, a.H, a.Sq, a.Sk, a.D = B, H, Sq, Sk, D
    a.scale, a.causal = float(scale), int(causal)
    keep: list = []
    _bias_args(a, q, k, key_bias, attn_bias, lengths, keep)
    work = _bias_workspace(q, k, key_bias, attn_bias, lengths)
    if out32 is not None:
        assert out32.shape == o.shape and out32.dtype == torch.float32 and out32.is_contiguous() and out32.device == q.device
    native.check(native.lib().st_attn_fwd_f32(ctypes.byref(a), native.ptr(out32), native.ptr(work), native.stream_ptr(q.device)),
                 "st_attn_fwd")
    launch_count += 1
    return o, lse


@functools.cache
def _one_pass_room(f32: bool):
    """The library's function for the floats of workspace that the one-pass form takes."""
    size = native.entry("st_attn_bwd_workspace_f32" if f32 else "st_attn_bwd_workspace", "iiiii")
    size.restype = ctypes.c_longlong
    return size


def attention_backward(q, k, v, o, lse, do, causal: bool = True, scale: Optional[float] = None,
                       dq=None, dk=None, dv=None, *, key_bias=None, attn_bias=None, lengths=None, do32=None):
    """Returns ``(dq, dk, dv)`` (bf16, ``[B,S,H,D]``); outputs may be preallocated strided views, all bf16 or all fp32.
    ``do32`` (CUDA, contiguous fp32): the output's gradient, of which ``do`` then receives the bf16 form."""
    global launch_count
    B, Sq, H, D = q.shape
    Sk = k.shape[1]
    scale = 1.0 / math.sqrt(D) if scale is None else scale
    if not native.use_native(q):
        with torch.enable_grad():
            qf, kf, vf = (t.detach().float().requires_grad_(True) for t in (q, k, v))
            of, _ = attention_reference(qf, kf, vf, causal, scale, key_bias=key_bias, attn_bias=attn_bias,
                                        lengths=lengths)
            g = torch.autograd.grad(of, (qf, kf, vf), do.float())
        outs = []
        for grad, given in zip(g, (dq, dk, dv)):
            if given is None:
                outs.append(grad.to(q.dtype))
            else:
                given.copy_(grad.to(given.dtype))
                outs.append(given)
        return tuple(outs)
    native.require_cuda("attention_backward", q, k, v, o, lse, do, dq, dk, dv, key_bias, attn_bias, lengths)
    _check_shapes(q, k, v)
    if o.shape != q.shape or do.shape != q.shape:
        raise ValueError(f"attention_backward: o {tuple(o.shape)} and do {tuple(do.shape)} must match q {tuple(q.shape)}")
    for t, n in ((q, "q"), (k, "k"), (v, "v"), (o, "o"), (do, "do")):
        _check_layout(t, n)
    dev = q.device
    dq = torch.empty((B, Sq, H, D), dtype=torch.bfloat16, device=dev) if dq is None else dq
    dk = torch.empty((B, Sk, H, D), dtype=torch.bfloat16, device=dev) if dk is None else dk
    dv = torch.empty((B, Sk, H, D), dtype=torch.bfloat16, device=dev) if dv is None else dv
    delta = torch.empty((B, H, Sq), dtype=torch.float32, device=dev)
    # all fields before the biases at once: one by one they take 8 us, as long as a launch
    strides = [n for t in (q, k, v, o, do, dq, dk, dv) for n in t.stride()[:3]]
    a = _BwdArgs(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), do.data_ptr(), lse.data_ptr(), delta.data_ptr(),
                 None, dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), *strides, B, H, Sq, Sk, D, float(scale), int(causal))
    keep: list = []
    _bias_args(a, q, k, key_bias, attn_bias, lengths, keep)
    work = _bias_workspace(q, k, key_bias, attn_bias, lengths)
    f32 = dq.dtype == torch.float32
    for t, n in ((dq, "dq"), (dk, "dk"), (dv, "dv")):
        if t.dtype != (torch.float32 if f32 else torch.bfloat16) or t.stride(-1) != 1:
            raise ValueError(f"attention_backward: {n} must be a view with contiguous D, and all gradients bf16 or all fp32")
    sums = None
    # One pass over the tile pairs instead of two, where the kernel takes it.  The passes add the parts of dQ in different orders,
    # so where bits must repeat the form does not depend on the memory left.
    if D == 64 and attn_bias is None and not native.deterministic_reduction():
        room = _one_pass_room(f32)(B, H, Sq, Sk, D)
        if room:
            try:
                sums = torch.empty(room, dtype=torch.float32, device=dev)
            except torch.cuda.OutOfMemoryError:      # two passes need no such room
                pass
    if do32 is not None:
        assert do32.shape == do.shape and do32.dtype == torch.float32 and do32.is_contiguous() and do32.device == dev
        assert do32.data_ptr() % 16 == 0
    native.check(native.lib().st_attn_bwd_one_pass(ctypes.byref(a), native.ptr(do32), ctypes.c_int(int(f32)), native.ptr(work),
                                                   native.ptr(sums), native.stream_ptr(dev)), "st_attn_bwd")
    launch_count += 3
    return dq, dk, dv


class _AttentionFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, k, v, causal, scale, key_bias, attn_bias, lengths):
        o, lse = attention_forward(q, k, v, causal, scale, key_bias=key_bias, attn_bias=attn_bias, lengths=lengths)
        ctx.save_for_backward(q, k, v, o, lse)
        ctx.causal, ctx.scale = causal, scale
        ctx.extras = (key_bias, attn_bias, lengths)     # biases are constants here: no gradient flows to them
        return o

    @staticmethod
    def backward(ctx, do):
        q, k, v, o, lse = ctx.saved_tensors
        if do.stride(-1) != 1 or do.dtype != q.dtype:
            do = do.to(q.dtype).contiguous()
        kb, ab, ln = ctx.extras
        dq, dk, dv = attention_backward(q, k, v, o, lse, do, ctx.causal, ctx.scale, key_bias=kb, attn_bias=ab,
                                        lengths=ln)
        return dq, dk, dv, None, None, None, None, None


class _AttentionF32Fn(torch.autograd.Function):
    """The same for fp32 ``[B,S,D]`` tensors of one head: one conversion launch brings q, k and v to bf16, the kernels write
    the output and the gradients in fp32 themselves, and the output's gradient is rounded in the pass that forms the row
    products with it."""

    @staticmethod
    def forward(ctx, q, k, v, causal, scale, key_bias, lengths):
        from . import multi
        qb, kb, vb = (t.unsqueeze(2) for t in multi.to_bf16((q.detach(), k.detach(), v.detach())))
        out = torch.empty_like(q, memory_format=torch.contiguous_format)
        o, lse = attention_forward(qb, kb, vb, causal, scale, key_bias=key_bias, lengths=lengths, out32=out.unsqueeze(2))
        ctx.save_for_backward(qb, kb, vb, o, lse)
        ctx.causal, ctx.scale, ctx.extras = causal, scale, (key_bias, lengths)
        return out

    @staticmethod
    def backward(ctx, do):
        q, k, v, o, lse = ctx.saved_tensors
        d32 = do.to(torch.float32).contiguous()
        if d32.data_ptr() % 16:
            d32 = d32.clone()
        dq, dk, dv = (torch.empty(t.shape, dtype=torch.float32, device=t.device) for t in (q, k, v))
        attention_backward(q, k, v, o, lse, torch.empty_like(o), ctx.causal, ctx.scale, dq, dk, dv, key_bias=ctx.extras[0],
                           lengths=ctx.extras[1], do32=d32.unsqueeze(2))
        return dq.squeeze(2), dk.squeeze(2), dv.squeeze(2), None, None, None, None


def takes_f32(q, k, v) -> bool:
    """Whether :class:`_AttentionF32Fn` takes these ``[B,S,D]`` tensors."""
    return pair_kernel_on() and all(t.is_cuda and t.dtype == torch.float32 and t.dim() == 3 and t.is_contiguous()
                                    and t.data_ptr() % 16 == 0 and t.numel() > 0 for t in (q, k, v))


def pair_kernel_on() -> bool:
    _apply_env_once()
    return pair_kernel_enabled()


def attention(q, k, v, causal: bool = True, scale: Optional[float] = None, *,
              key_bias: Optional[torch.Tensor] = None, attn_bias: Optional[torch.Tensor] = None,
              lengths: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Differentiable attention on ``[B,S,H,D]`` tensors (gradients for q, k, v; the biases are constants)."""
    return _AttentionFn.apply(q, k, v, causal, scale, key_bias, attn_bias, lengths)
