"""Finite checks, scaled copies and plain updates over lists of small fp32 tensors, and the mean-squared-error loss
(``csrc/elementwise/multi.cu``): one launch per list, and no device-to-host copy for what the host has to know - the
kernels write it into pinned memory, so a check is a launch and a stream synchronisation.

The callers (:mod:`spiraltorch_b200.nn`) keep their PyTorch statement for tensors that :func:`takes` refuses.
"""
from __future__ import annotations

import bisect
import ctypes
import functools
from typing import Optional, Sequence

import torch

from . import native

launch_count = 0
_CHECK, _DIV = 0, 1


def takes(tensors: Sequence[torch.Tensor]) -> bool:
    """Whether the kernels take these tensors: dense non-empty fp32 on the current CUDA device, outside a graph capture
    (a captured stream cannot be waited for) and outside function transforms and forward-mode differentiation (whose
    tensors are more than their memory)."""
    if not tensors or not tensors[0].is_cuda or torch.cuda.is_current_stream_capturing() \
            or torch._C._functorch.peek_interpreter_stack() is not None or torch.autograd.forward_ad._current_level >= 0:
        return False
    dev = tensors[0].device
    return dev.index == torch.cuda.current_device() and all(
        type(t) in (torch.Tensor, torch.nn.Parameter) and t.device == dev and t.dtype == torch.float32 and t.is_contiguous()
        and t.numel() > 0 for t in tensors)


@functools.cache
def _most() -> int:
    """Tensors that one launch takes."""
    return native.lib().st_multi_max()


def _run(op: int, src, dst, value: float) -> Optional[int]:
    """Index of the first tensor of ``src`` with a value that is not finite, or None."""
    global launch_count
    stream = torch.cuda.current_stream()
    launch, blocks_of = native.entry("st_multi", "iipppfpp"), native.entry("st_multi_blocks", "q")
    first = None
    for at in range(0, len(src), _most()):
        s = src[at:at + _most()]
        n = len(s)
        counts = [t.numel() for t in s]
        blocks = blocks_of(max(counts))
        bad = torch.empty(n * blocks, dtype=torch.int32, pin_memory=True)
        ptrs = (ctypes.c_void_p * n)(*[t.data_ptr() for t in s])
        outs = None if dst is None else (ctypes.c_void_p * n)(*[t.data_ptr() for t in dst[at:at + _most()]])
        native.check(launch(op, n, ptrs, outs, (ctypes.c_longlong * n)(*counts), value, bad.data_ptr(), stream.cuda_stream), "st_multi")
        launch_count += 1
        stream.synchronize()
        if first is None and bad.any():
            first = at + int(bad.nonzero()[0]) // blocks
    return first


def first_nonfinite(tensors: Sequence[torch.Tensor]) -> Optional[int]:
    """Index of the first tensor that holds an infinity or a NaN, or None."""
    return _run(_CHECK, tensors, None, 0.0)


def divided(tensors: Sequence[torch.Tensor], value: float):
    """``([t / value for t in tensors], index of the first tensor that is not finite or None)``."""
    out = [torch.empty_like(t) for t in tensors]
    return out, _run(_DIV, tensors, out, value)


def descend_(values: Sequence[torch.Tensor], grads: Sequence[torch.Tensor], lr: float) -> bool:
    """``v -= lr * g`` for every pair, in place.  The blocks of a launch run in any order: False, with nothing done, where memory
    of a value also belongs to another of the tensors, or where a gradient has not its value's shape."""
    global launch_count
    from . import gemm
    if any(v.shape != g.shape for v, g in zip(values, grads)):
        return False
    at_v, at_g, sizes = [t.data_ptr() for t in values], [t.data_ptr() for t in grads], [t.numel() for t in values]
    spans = sorted(zip(at_v, sizes))
    begins = [begin for begin, _ in spans]
    if any(begin + 4 * n > after for (begin, n), after in zip(spans, begins[1:])):
        return False
    for g, n in zip(at_g, sizes):
        below = bisect.bisect_left(begins, g + 4 * n) - 1        # the last value that begins before the gradient ends
        if below >= 0 and spans[below][0] + 4 * spans[below][1] > g:
            return False
    lib, stream = native.lib(), native.stream_ptr(values[0].device)
    # values whose bf16 copy is in use get the next one in the same launch (a new tensor: a graph may still hold the old one)
    halves = [torch.empty(v.shape, dtype=torch.bfloat16, device=v.device) if gemm.has_cached_bf16(v) else None for v in values]
    for at in range(0, len(values), _most()):
        part = slice(at, at + _most())
        n = len(values[part])
        array = ctypes.c_void_p * n
        native.check(lib.st_multi_step_bf16(
            ctypes.c_int(n), array(*at_g[part]), array(*at_v[part]), array(*[None if t is None else t.data_ptr() for t in halves[part]]),
            (ctypes.c_longlong * n)(*sizes[part]), ctypes.c_float(lr), stream), "st_multi_step_bf16")
        launch_count += 1
    for v, h in zip(values, halves):
        torch.autograd.graph.increment_version(v)      # copies of the values are cached by version
        if h is not None:
            gemm.renew_cached_bf16(v, h)
    return True


def to_bf16(tensors: Sequence[torch.Tensor]):
    """bf16 copies of dense 16-byte aligned fp32 CUDA tensors."""
    global launch_count
    device = native.require_cuda("to_bf16", *tensors)
    out = [torch.empty_like(t, dtype=torch.bfloat16, memory_format=torch.contiguous_format) for t in tensors]
    n = len(out)
    native.check(native.entry("st_multi_cast_bf16", "ipppp")(
        n, (ctypes.c_void_p * n)(*[t.data_ptr() for t in tensors]), (ctypes.c_void_p * n)(*[t.data_ptr() for t in out]),
        (ctypes.c_longlong * n)(*[t.numel() for t in out]), native.raw_stream(device)), "st_multi_cast_bf16")
    launch_count += 1
    return out


def mse_forward(p: torch.Tensor, t: torch.Tensor):
    """``(mean((p - t)^2) of shape (1, 1), all inputs are finite)``."""
    global launch_count
    native.require_cuda("mse_forward", p, t)
    lib, stream, n = native.lib(), torch.cuda.current_stream(), p.numel()
    value = p.new_empty((1, 1), dtype=torch.float32)
    work = p.new_empty(lib.st_mse_workspace(), dtype=torch.float32)
    bad = torch.empty(native.entry("st_mse_blocks", "q")(n), dtype=torch.int32, pin_memory=True)
    native.check(native.entry("st_mse_forward", "ppqpppp")(p.data_ptr(), t.data_ptr(), n, value.data_ptr(), work.data_ptr(),
                                                           bad.data_ptr(), stream.cuda_stream), "st_mse_forward")
    launch_count += 1
    stream.synchronize()
    return value, not bool(bad.any())


def mse_backward(p: torch.Tensor, t: torch.Tensor):
    """``(2 (p - t) / n, all inputs are finite)``."""
    global launch_count
    native.require_cuda("mse_backward", p, t)
    stream, n = torch.cuda.current_stream(), p.numel()
    g = torch.empty_like(p)
    bad = torch.empty(native.entry("st_mse_blocks", "q")(n), dtype=torch.int32, pin_memory=True)
    native.check(native.entry("st_mse_backward", "ppqppp")(p.data_ptr(), t.data_ptr(), n, g.data_ptr(), bad.data_ptr(),
                                                           stream.cuda_stream), "st_mse_backward")
    launch_count += 1
    stream.synchronize()
    return g, not bool(bad.any())
