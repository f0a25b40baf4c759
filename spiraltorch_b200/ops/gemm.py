"""bf16 GEMM with fused epilogues on the tcgen05 kernel (``csrc/gemm/gemm_sm100.cu``).

``gemm`` computes ``C[M,N] = epilogue(alpha * A @ B^T)`` where each operand may be stored
K-major (``A`` is ``[M,K]``, ``B`` is ``[N,K]``) or MN-major (``A`` is ``[K,M]``, ``B`` is
``[K,N]``), so a linear layer's forward, data-gradient and weight-gradient all run without a
transposition pass.  CPU tensors take an fp32 PyTorch path with the same semantics (that is
the numerical oracle in the tests).

Reference parity: ``Tensor::matmul``, ``matmul_bias_relu/gelu``, ``matmul_bias_add_relu/gelu``
(crates/st-tensor/src/pure.rs:2013,4406,4637,4824,5084).
"""
from __future__ import annotations

import ctypes
import struct
from typing import Optional

import torch

from . import native

ACT_NONE, ACT_RELU, ACT_GELU, ACT_GELU_BWD, ACT_RELU_BWD = 0, 1, 2, 3, 4
_ACT_NAMES = {None: 0, "none": 0, "relu": 1, "gelu": 2, "gelu_bwd": 3, "relu_bwd": 4}

#: number of native kernel launches issued through this module (for bench accounting)
launch_count = 0


# StGemmArgs of csrc/gemm/gemm_sm100.cu: A, B, C, bias, residual, aux_out, aux_in; lda, ldb, ldc, ldr, ld_aux_out,
# ld_aux_in and the batch strides of A, B, C; M, N, K, batch, a_mn_major, b_mn_major, out_fp32, accumulate, act; alpha;
# max_ctas.  Packed in one call: filling the 27 fields of a ctypes structure costs as much as the launch itself.
_pack_args = struct.Struct("@7P9q9ifi").pack


#: split the K loop of weight-gradient GEMMs whose tile count fills the SMs badly (the partial
#: sums meet in fp32 atomics, so the summation order is not fixed); native.deterministic_reduction()
#: (SPIRAL_DETERMINISTIC_REDUCTION / SPIRAL_DETERMINISTIC) turns it off per call
SPLIT_K = True
_NUM_SMS = 148


def _split_k(M: int, N: int, K: int) -> int:
    tiles = ((M + 127) // 128) * ((N + 255) // 256 if N > 128 else 1)
    best, best_eff = 1, tiles / (-(-tiles // _NUM_SMS) * _NUM_SMS)
    for s in (2, 3, 4):
        if K % (s * 64) or K // s < 2048:
            continue
        work = tiles * s
        eff = work / (-(-work // _NUM_SMS) * _NUM_SMS)
        if eff > best_eff + 0.04:
            best, best_eff = s, eff
    return best


def _partial_splits(M: int, N: int, K: int) -> int:
    """Parts of the K loop of a weight gradient whose few tiles would leave most SMs idle (the first convolution of a
    256-image batch: one tile over a million pixels, 4.9 ms on one SM and 0.06 ms in 128 parts).  Each part writes its own
    fp32 result and a second kernel adds them in a fixed order.  Only for results of at most 256 x 256: the 768 x 768
    ones of the 85 M language model are faster with the two to four atomic parts of ``_split_k`` (16.2 against 16.6 ms a
    step).  A part keeps at least 512 rows, below which the parts cost more than the loop."""
    if M * N > 1 << 16:
        return 1
    tiles = ((M + 127) // 128) * ((N + 255) // 256)
    most = min(_NUM_SMS // tiles, K // 512)
    return next((s for s in range(most, 1, -1) if K % s == 0), 1)


def gelu_tanh(x: torch.Tensor) -> torch.Tensor:
    return torch.nn.functional.gelu(x, approximate="tanh")


def gelu_tanh_grad(x: torch.Tensor) -> torch.Tensor:
    k0, k1 = 0.7978845608028654, 0.044715
    u = k0 * (x + k1 * x ** 3)
    t = torch.tanh(u)
    return 0.5 * (1 + t) + 0.5 * x * (1 - t * t) * k0 * (1 + 3 * k1 * x * x)


def _reference(a, b, a_mn, b_mn, out, out_dtype, bias, act, residual, aux_out, aux_in, alpha, accumulate):
    """fp32 PyTorch statement of the kernel's semantics (CPU path and test oracle)."""
    af = a.float().transpose(-1, -2) if a_mn else a.float()
    bf = b.float() if b_mn else b.float().transpose(-1, -2)
    v = alpha * (af @ bf)
    if bias is not None:
        v = v + bias.float()
    if aux_out is not None:
        aux_out.copy_(v.to(aux_out.dtype))
    if act == ACT_RELU:
        v = torch.relu(v)
    elif act == ACT_GELU:
        v = gelu_tanh(v)
    elif act == ACT_GELU_BWD:
        v = v * gelu_tanh_grad(aux_in.float())
    elif act == ACT_RELU_BWD:
        v = torch.where(aux_in.float() > 0, v, torch.zeros_like(v))
    if residual is not None:
        v = v + residual.float()
    if out is None:
        return v.to(out_dtype)
    if accumulate:
        v = v + out.float()
    out.copy_(v.to(out.dtype))
    return out


# bf16 copies of fp32 parameters: a weight is rounded once per optimizer step instead of once per forward.
# Entries are keyed by storage address and invalidated by the tensor's version counter; each entry also HOLDS its
# source tensor, so the address cannot be freed and handed to another tensor while the entry lives (a recycled
# address with an equal version would otherwise return another tensor's values).  Least-recently-used entries are
# dropped once the cache holds more than _BF16_CACHE_BYTES of sources and copies.
from collections import OrderedDict as _OrderedDict

_bf16_cache: "_OrderedDict" = _OrderedDict()
_bf16_cache_bytes = 0
_BF16_CACHE_BYTES = 1 << 30


def cached_bf16(t: torch.Tensor) -> torch.Tensor:
    """bf16 copy of ``t`` (itself when it already is bf16), reused until ``t`` is modified in place."""
    global _bf16_cache_bytes
    if t.dtype == torch.bfloat16:
        return t
    key = (t.data_ptr(), tuple(t.shape), tuple(t.stride()), t.dtype, t.device)
    hit = _bf16_cache.get(key)
    if hit is not None and hit[0] == t._version:
        _bf16_cache.move_to_end(key)
        return hit[1]
    out = t.detach().to(torch.bfloat16).contiguous()
    cost = t.numel() * (t.element_size() + 2)
    if cost > _BF16_CACHE_BYTES // 4:
        return out                                   # too large to be worth pinning
    if hit is not None:
        _bf16_cache_bytes -= hit[3]
    _bf16_cache[key] = (t._version, out, t.detach(), cost)      # the detached alias keeps the storage alive
    _bf16_cache.move_to_end(key)
    _bf16_cache_bytes += cost
    while _bf16_cache_bytes > _BF16_CACHE_BYTES and len(_bf16_cache) > 1:
        _, old = _bf16_cache.popitem(last=False)
        _bf16_cache_bytes -= old[3]
    return out


def has_cached_bf16(t: torch.Tensor) -> bool:
    """Whether ``t``'s current values have a cached copy."""
    hit = _bf16_cache.get((t.data_ptr(), tuple(t.shape), tuple(t.stride()), t.dtype, t.device))
    return hit is not None and hit[0] == t._version


def renew_cached_bf16(t: torch.Tensor, copy: torch.Tensor) -> None:
    """``copy`` holds the bf16 form of ``t``'s values as they are now: it takes the place of the cached one."""
    key = (t.data_ptr(), tuple(t.shape), tuple(t.stride()), t.dtype, t.device)
    hit = _bf16_cache.get(key)
    if hit is not None:
        _bf16_cache[key] = (t._version, copy, hit[2], hit[3])


def clear_bf16_cache() -> None:
    """Drops every cached bf16 copy (CUDA-graph capture calls this so that the casts it needs are captured too)."""
    global _bf16_cache_bytes
    _bf16_cache.clear()
    _bf16_cache_bytes = 0


def _pad_to(t: torch.Tensor, rows: int, cols: int) -> torch.Tensor:
    if t.shape[-2] == rows and t.shape[-1] == cols and t.stride(-1) == 1 and t.stride(-2) % 8 == 0 \
            and t.data_ptr() % 16 == 0:
        return t
    out = t.new_zeros(*t.shape[:-2], rows, cols)
    out[..., : t.shape[-2], : t.shape[-1]] = t
    return out


def _tma_ready(t: torch.Tensor) -> torch.Tensor:
    """``t``, or a padded copy: TMA needs 16-byte aligned rows, so the contiguous dimension is padded to a multiple of 8."""
    stride = t.stride()
    c = t.shape[-1]
    if stride[-1] == 1 and stride[-2] % 8 == 0 and c % 8 == 0 and (len(stride) < 3 or stride[0] % 8 == 0) \
            and t.data_ptr() % 16 == 0:
        return t
    return _pad_to(t.contiguous() if stride[-1] != 1 else t, t.shape[-2], (c + 7) // 8 * 8)


def gemm(a: torch.Tensor, b: torch.Tensor, *, a_mn: bool = False, b_mn: bool = False,
         out: Optional[torch.Tensor] = None, out_dtype: Optional[torch.dtype] = None,
         bias: Optional[torch.Tensor] = None, act=None, residual: Optional[torch.Tensor] = None,
         aux_out: Optional[torch.Tensor] = None, aux_in: Optional[torch.Tensor] = None,
         alpha: float = 1.0, accumulate: bool = False, max_ctas: int = 0) -> torch.Tensor:
    """``C = epilogue(alpha * op(A) @ op(B)^T)``; 2-D or batched 3-D operands.

    ``a``: ``[M,K]`` (or ``[K,M]`` when ``a_mn``); ``b``: ``[N,K]`` (or ``[K,N]`` when ``b_mn``).
    Epilogue order: ``+bias`` → store ``aux_out`` → activation (``relu``/``gelu``, or multiply
    by the derivative evaluated at ``aux_in`` for ``gelu_bwd``/``relu_bwd``) → ``+residual`` →
    ``+out`` when ``accumulate`` → cast to ``out``'s dtype (bf16 or fp32).
    """
    global launch_count
    act_id = _ACT_NAMES[act] if not isinstance(act, int) else act
    on_cuda = native.use_native(a)
    if out is not None:
        out_dtype = out.dtype
    elif out_dtype is None:
        out_dtype = torch.bfloat16 if on_cuda else a.dtype
    if not on_cuda:
        return _reference(a, b, a_mn, b_mn, out, out_dtype, bias, act_id, residual, aux_out, aux_in,
                          alpha, accumulate)

    device = native.require_cuda("gemm", a, b, out, bias, residual, aux_out, aux_in)
    shape_a, shape_b = a.shape, b.shape
    batched = len(shape_a) == 3
    if batched:
        assert len(shape_b) == 3 and shape_a[0] == shape_b[0]
    K, M = (shape_a[-2], shape_a[-1]) if a_mn else (shape_a[-1], shape_a[-2])
    Kb, N = (shape_b[-2], shape_b[-1]) if b_mn else (shape_b[-1], shape_b[-2])
    if K != Kb:
        raise ValueError(f"gemm: inner dimensions differ ({K} vs {Kb})")
    if a.dtype != torch.bfloat16:
        a = a.to(torch.bfloat16)
    if b.dtype != torch.bfloat16:
        b = b.to(torch.bfloat16)
    a, b = _tma_ready(a), _tma_ready(b)
    batch = shape_a[0] if batched else 1
    if out is None:
        shape = (batch, M, N) if batched else (M, N)
        out = a.new_empty(shape) if out_dtype == torch.bfloat16 else a.new_empty(shape, dtype=out_dtype)
    else:
        assert out.stride(-1) == 1 and out.shape[-2] == M and out.shape[-1] == N
        assert out_dtype in (torch.bfloat16, torch.float32)
    operands = [0, 0, 0, 0, 0, 0, 0]           # addresses of the epilogue's operands, then the leading dimensions of the matrices
    for i, t in enumerate((bias, residual, aux_out, aux_in)):
        if t is not None:
            ld = t.stride()
            assert t.dtype == torch.bfloat16 and ld[-1] == 1, "epilogue operands must be bf16"
            operands[i] = t.data_ptr()
            if i:
                operands[3 + i] = ld[-2]
    lib, stream = native.lib(), native.raw_stream(device)
    stride_a, stride_b, stride_c = a.stride(), b.stride(), out.stride()
    fp32 = out_dtype == torch.float32
    target, ldc, k_part, parts, acc, max_ctas = out, stride_c[-2], K, batch, int(accumulate), int(max_ctas)
    strides = (stride_a[0], stride_b[0], stride_c[0]) if batched else (0, 0, 0)
    in_parts = False
    if SPLIT_K and a_mn and b_mn and fp32 and not batched and bias is None and residual is None and act_id == 0:
        n = _partial_splits(M, N, K) if aux_out is None and max_ctas == 0 and out.is_contiguous() else 1
        if n > 1:
            in_parts = True
            target, ldc, acc = torch.empty((n, M, N), dtype=torch.float32, device=a.device), N, 0
        elif accumulate and N % 32 == 0 and stride_c[0] % 4 == 0 and not native.deterministic_reduction():
            # weight-gradient shape with a poor tile count: split the long reduction over CTAs of the same tile
            # (expressed as a batch over K) and add the partials with fp32 atomics
            n = _split_k(M, N, K)
            acc = 2 if n > 1 else acc
        if n > 1:
            k_part, parts = K // n, n
            strides = (k_part * stride_a[0], k_part * stride_b[0], M * N if in_parts else 0)
    args = _pack_args(a.data_ptr(), b.data_ptr(), target.data_ptr(), *operands[:4], stride_a[-2], stride_b[-2], ldc, *operands[4:],
                      *strides, M, N, k_part, parts, int(a_mn), int(b_mn), fp32, acc, act_id, float(alpha), max_ctas)
    status = lib.st_gemm_bf16(args, ctypes.c_void_p(stream))
    if status:
        native.check(status, "st_gemm_bf16")
    launch_count += 1
    if in_parts:
        native.check(native.entry("st_reduce_partials", "ppiiip")(target.data_ptr(), out.data_ptr(), n, M * N, int(accumulate), stream),
                     "st_reduce_partials")
        launch_count += 1
    return out


class _LinearFn(torch.autograd.Function):
    """``y = x @ W^T (+ bias)`` with W stored ``[out, in]``; dgrad and wgrad on the same kernel."""

    @staticmethod
    def forward(ctx, x, weight, bias):
        x2 = x.reshape(-1, x.shape[-1])
        y = gemm(x2, weight, bias=bias)
        ctx.save_for_backward(x2, weight)
        ctx.has_bias = bias is not None
        ctx.x_shape = x.shape
        return y.reshape(*x.shape[:-1], weight.shape[0])

    @staticmethod
    def backward(ctx, dy):
        x2, weight = ctx.saved_tensors
        dy2 = dy.reshape(-1, dy.shape[-1])
        if dy2.dtype != x2.dtype or not dy2.is_contiguous():
            dy2 = dy2.to(x2.dtype).contiguous()
        dx = dw = db = None
        if ctx.needs_input_grad[0]:
            dx = gemm(dy2, weight, b_mn=True).reshape(ctx.x_shape)
        if ctx.needs_input_grad[1]:
            main_grad = getattr(weight, "main_grad", None)
            if main_grad is not None:
                # fp32 gradient accumulation straight from the epilogue
                gemm(dy2, x2, a_mn=True, b_mn=True, out=main_grad, accumulate=True)
                dw = None
            else:
                dw = gemm(dy2, x2, a_mn=True, b_mn=True, out_dtype=weight.dtype)
        if ctx.has_bias and ctx.needs_input_grad[2]:
            db = dy2.float().sum(0).to(dy2.dtype)
        return dx, dw, db


def linear(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Differentiable ``x @ weight^T + bias`` (weight ``[out, in]``)."""
    return _LinearFn.apply(x, weight, bias)
