"""LayerNorm / RMSNorm forward and backward (``csrc/norm/norm.cu``).

bf16 activations, fp32 statistics; parameter gradients are produced in fp32 and either
returned (cast to the parameter dtype) or accumulated into ``param.main_grad`` when that
attribute exists (fp32 gradient accumulation across micro-batches).

Reference parity: ``Tensor::layer_norm_affine`` / ``layer_norm_affine_add``
(crates/st-tensor/src/pure.rs:3702-4058), ``nn.LayerNorm`` (crates/st-nn/src/layers/normalization.rs:352).
RMSNorm has no counterpart in the reference.
"""
from __future__ import annotations

import ctypes
import functools
from typing import Optional

import torch

from . import native

launch_count = 0


def _scratch(lib, x2: torch.Tensor) -> torch.Tensor:
    """Partial parameter gradients of one backward call.  A tensor per call: a buffer kept for a device would be shared by its
    streams and threads, and a captured step would go on writing to it after a larger call had replaced it."""
    lib.st_norm_bwd_scratch_elems.restype = ctypes.c_longlong
    return x2.new_empty(native.entry("st_norm_bwd_scratch_elems", "ii")(*x2.shape), dtype=torch.float32)


@functools.cache
def _limit(entry: str) -> int:
    return getattr(native.lib(), entry)()


def gelu_max_features() -> int:
    """Widest rows of :func:`norm_gelu_forward` and its backward."""
    return _limit("st_norm_gelu_max_features")


def takes_f32(d: int, *tensors: Optional[torch.Tensor]) -> bool:
    """Whether the fp32 form of the kernels takes these tensors (``None`` entries are skipped)."""
    return d % 8 == 0 and d > 0 and all(
        t is None or (t.is_cuda and t.dtype == torch.float32 and t.is_contiguous() and t.data_ptr() % 16 == 0) for t in tensors) \
        and d <= _limit("st_norm_f32_max_features")


def _form(entry: str, types: str, x2: torch.Tensor, rounded: bool):
    return native.entry(entry if x2.dtype != torch.float32 else entry + ("_f32_rounded" if rounded else "_f32"), types)


def norm_reference(x, gamma, beta, eps, rms, residual=None):
    xf = x.float()
    if residual is not None:
        xf = (xf + residual.float()).to(x.dtype).float()
    if rms:
        rstd = torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + eps)
        y = xf * rstd * gamma.float()
        mean = torch.zeros_like(rstd)
    else:
        mean = xf.mean(-1, keepdim=True)
        var = (xf - mean).pow(2).mean(-1, keepdim=True)
        rstd = torch.rsqrt(var + eps)
        y = (xf - mean) * rstd * gamma.float()
        if beta is not None:
            y = y + beta.float()
    return y, xf, mean.squeeze(-1), rstd.squeeze(-1)


def norm_forward(x2: torch.Tensor, gamma, beta, eps: float, rms: bool, residual=None, out=None, copy_input: bool = False,
                 rounded: bool = False):
    """x2: [rows, d] bf16, or fp32 throughout where :func:`takes_f32`.  Returns (y, summed_input_or_None, mean, rstd); ``out``
    (contiguous, same shape and dtype) receives y when given.  fp32 form on CUDA: with ``copy_input`` and no residual the second
    result is a copy of x2; with ``rounded`` operands and results are rounded to bf16, as the bf16 form has them."""
    global launch_count
    rows, d = x2.shape
    if out is not None:
        assert out.shape == x2.shape and out.dtype == x2.dtype and out.is_contiguous() and out.device == x2.device
    if not native.use_native(x2):
        y, xs, mean, rstd = norm_reference(x2, gamma, beta, eps, rms, residual)
        y = y.to(x2.dtype)
        if out is not None:
            y = out.copy_(y)
        return y, (xs.to(x2.dtype) if residual is not None else None), mean, rstd
    device = native.require_cuda("norm_forward", x2, residual, gamma, beta)
    y = torch.empty_like(x2) if out is None else out
    s = torch.empty_like(x2) if residual is not None or (copy_input and x2.dtype == torch.float32) else None
    mean = x2.new_empty(rows, dtype=torch.float32)
    rstd = torch.empty_like(mean)
    status = _form("st_norm_fwd", "ippppppppiifp", x2, rounded)(
        int(rms), x2.data_ptr(), native.address(residual), native.address(gamma), native.address(beta), y.data_ptr(), native.address(s),
        mean.data_ptr(), rstd.data_ptr(), rows, d, eps, native.raw_stream(device))
    if status:
        native.check(status, "st_norm_fwd")
    launch_count += 1
    return y, s, mean, rstd


def norm_backward(dy2, x2, gamma, mean, rstd, rms: bool, dgamma: torch.Tensor,
                  dbeta: Optional[torch.Tensor], accumulate: bool, dres=None, out=None, rounded: bool = False):
    """Writes dx (returned; into ``out`` when given) and fp32 dgamma/dbeta (in place, ``+=`` when ``accumulate``).
    ``rounded`` as in :func:`norm_forward`."""
    global launch_count
    rows, d = x2.shape
    if out is not None:
        assert out.shape == x2.shape and out.dtype == x2.dtype and out.is_contiguous() and out.device == x2.device
    if not native.use_native(x2):
        xf, dyf, g = x2.float(), dy2.float(), gamma.float()
        xh = (xf - (0 if rms else mean.unsqueeze(-1))) * rstd.unsqueeze(-1)
        gy = dyf * g
        m1 = (gy * xh).mean(-1, keepdim=True)
        m2 = 0 if rms else gy.mean(-1, keepdim=True)
        dx = rstd.unsqueeze(-1) * (gy - m2 - xh * m1)
        if dres is not None:
            dx = dx + dres.float()
        dg = (dyf * xh).sum(0)
        dgamma.copy_(dgamma + dg if accumulate else dg)
        if dbeta is not None:
            db = dyf.sum(0)
            dbeta.copy_(dbeta + db if accumulate else db)
        dx = dx.to(x2.dtype)
        return dx if out is None else out.copy_(dx)
    device = native.require_cuda("norm_backward", dy2, x2, gamma, mean, rstd, dres, dgamma, dbeta)
    dx = torch.empty_like(x2) if out is None else out
    scratch = _scratch(native.lib(), x2)
    status = _form("st_norm_bwd", "ipppppppppipiip", x2, rounded)(
        int(rms), dy2.data_ptr(), x2.data_ptr(), gamma.data_ptr(), native.address(mean), rstd.data_ptr(), native.address(dres),
        dx.data_ptr(), dgamma.data_ptr(), native.address(dbeta), int(accumulate), scratch.data_ptr(), rows, d, native.raw_stream(device))
    if status:
        native.check(status, "st_norm_bwd")
    launch_count += 2
    return dx


def norm_gelu_forward(x2: torch.Tensor, gamma, beta, eps: float):
    """``gelu(layer_norm(x2))`` of contiguous bf16 rows of at most :func:`gelu_max_features` on CUDA: ``(y, mean, rstd)``."""
    global launch_count
    device = native.require_cuda("norm_gelu_forward", x2, gamma, beta)
    rows, d = x2.shape
    y = torch.empty_like(x2)
    mean = x2.new_empty(rows, dtype=torch.float32)
    rstd = torch.empty_like(mean)
    native.check(native.entry("st_norm_gelu_fwd", "ppppppiifp")(
        x2.data_ptr(), gamma.data_ptr(), beta.data_ptr(), y.data_ptr(), mean.data_ptr(), rstd.data_ptr(), rows, d, eps,
        native.raw_stream(device)), "st_norm_gelu_fwd")
    launch_count += 1
    return y, mean, rstd


def norm_gelu_backward(dy2, x2, gamma, beta, mean, rstd, dgamma: torch.Tensor, dbeta: torch.Tensor) -> torch.Tensor:
    """Backward of :func:`norm_gelu_forward`: returns dx, writes the fp32 ``dgamma`` and ``dbeta``."""
    global launch_count
    device = native.require_cuda("norm_gelu_backward", dy2, x2, gamma, beta, mean, rstd, dgamma, dbeta)
    rows, d = x2.shape
    scratch = _scratch(native.lib(), x2)
    dx = torch.empty_like(x2)
    native.check(native.entry("st_norm_gelu_bwd", "pppppppppipiip")(
        dy2.data_ptr(), x2.data_ptr(), gamma.data_ptr(), beta.data_ptr(), mean.data_ptr(), rstd.data_ptr(), dx.data_ptr(),
        dgamma.data_ptr(), dbeta.data_ptr(), 0, scratch.data_ptr(), rows, d, native.raw_stream(device)), "st_norm_gelu_bwd")
    launch_count += 2
    return dx


class _NormFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, gamma, beta, eps, rms):
        x2 = x.reshape(-1, x.shape[-1])
        if not x2.is_contiguous():
            x2 = x2.contiguous()
        y, _, mean, rstd = norm_forward(x2, gamma, beta, eps, rms)
        ctx.save_for_backward(x2, gamma, mean, rstd)
        ctx.rms = rms
        ctx.has_beta = beta is not None
        ctx.gamma_ref, ctx.beta_ref = gamma, beta
        return y.reshape(x.shape)

    @staticmethod
    def backward(ctx, dy):
        x2, gamma, mean, rstd = ctx.saved_tensors
        dy2 = dy.reshape(x2.shape)
        if not dy2.is_contiguous() or dy2.dtype != x2.dtype:
            dy2 = dy2.to(x2.dtype).contiguous()
        gamma_p, beta_p = ctx.gamma_ref, ctx.beta_ref
        mg = getattr(gamma_p, "main_grad", None)
        mb = getattr(beta_p, "main_grad", None) if ctx.has_beta else None
        if mg is not None and (not ctx.has_beta or mb is not None):
            dx = norm_backward(dy2, x2, gamma, mean, rstd, ctx.rms, mg, mb, True)
            return dx.reshape(dy.shape), None, None, None, None
        dg = torch.empty(x2.shape[1], dtype=torch.float32, device=x2.device)
        db = torch.empty_like(dg) if ctx.has_beta else None
        dx = norm_backward(dy2, x2, gamma, mean, rstd, ctx.rms, dg, db, False)
        return (dx.reshape(dy.shape), dg.to(gamma.dtype),
                db.to(gamma.dtype) if db is not None else None, None, None)


def layer_norm(x, gamma, beta=None, eps: float = 1e-5) -> torch.Tensor:
    return _NormFn.apply(x, gamma, beta, eps, False)


def rms_norm(x, gamma, eps: float = 1e-6) -> torch.Tensor:
    return _NormFn.apply(x, gamma, None, eps, True)
