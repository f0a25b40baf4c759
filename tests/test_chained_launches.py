"""Kernels whose start-up overlaps the end of the kernel before them: none touches global memory before it has waited for that
kernel (read from the sources), and what one kernel writes the next one reads, whatever stands between them in the stream."""
import re
from pathlib import Path

import pytest
import torch

from spiraltorch_b200.ops import attention as A
from spiraltorch_b200.ops import conv as C
from spiraltorch_b200.ops import gemm as G
from spiraltorch_b200.ops import multi, native
from spiraltorch_b200.ops import rank as R

CSRC = Path(__file__).resolve().parents[1] / "csrc"


def _block(text, start):
    """The text between the brace at or after ``start`` and its partner."""
    at, depth = text.index("{", start), 0
    for i in range(at, len(text)):
        depth += (text[i] == "{") - (text[i] == "}")
        if depth == 0:
            return text[at + 1:i]
    raise AssertionError("unbalanced braces")


def _chained_kernels():
    """(file and name, parameters, body) of every kernel that waits for the one before it."""
    found = []
    for path in sorted(CSRC.rglob("*.cu*")):
        text = re.sub(r"//[^\n]*|/\*.*?\*/", "", path.read_text(), flags=re.S)
        for m in re.finditer(r"__global__", text):
            body = _block(text, m.start())
            if "chain_begin(" in body:
                head = text[m.start():text.index("{", m.start())]
                name = [n for n in re.findall(r"(\w+)\s*\(", head) if n not in ("__launch_bounds__", "num_threads")][0]
                found.append((f"{path.name}:{name}", head, body))
    return found


def _without_lambdas(code):
    """What runs where it stands: the bodies of lambdas are left out."""
    while (m := re.search(r"=\s*\[&\]", code)) is not None:
        code = code[:m.start()] + code[m.start():].replace(_block(code, m.start()), "", 1).replace("[&]", "[]", 1)
    return code


def test_nothing_reads_global_memory_before_the_wait():
    kernels = _chained_kernels()
    assert len(kernels) > 40
    early = []
    for name, head, body in kernels:
        before = _without_lambdas(body[:body.index("chain_begin(")])
        pointers = re.findall(r"\*\s*(?:__restrict__\s+)?(\w+)\s*[,)]", head)
        access = r"\b(?:p|cm)\.\w+\s*\[|__ldg|[=(,?:]\s*\*\s*(?:p|cm)\.\w+|tma_load|bulk_load|atomic\w+\(" + "".join(rf"|\b{x}\s*\[" for x in pointers)
        if (hit := re.search(access, before)) is not None:
            early.append((name, hit.group(0)))
    assert not early


def test_addresses_of_constant_memory_depend_on_the_wait():
    """Loads through ``const __restrict__`` pointers may be moved across the wait unless their addresses depend on it; for
    pointers among the parameters and for local ones."""
    free = []
    for name, head, body in _chained_kernels():
        at = body.index("chain_begin(")
        behind = body[at + len("chain_begin("):body.index(")", at)].split(",")
        constant = re.findall(r"\bconst\s+[\w:]+\s*\*\s*__restrict__\s+(\w+)", head + body)
        free += [(name, x) for x in constant if x not in [b.strip() for b in behind]]
    assert not free


@pytest.mark.gpu
def test_convolution_reads_the_bias_that_was_just_written():
    """64 channels at 64 x 64 run the shared-row kernel; its bias is the last row of a product launched right before it."""
    torch.manual_seed(0)
    x = torch.randn(16, 64, 64, 64, device="cuda").bfloat16()
    w = (torch.randn(64, 9 * 64, device="cuda") / 24).bfloat16()
    b = torch.randn(64, 4096, device="cuda").bfloat16()
    products = [torch.randn(4096, 4096, device="cuda").bfloat16() for _ in range(6)]
    out = torch.zeros(4096, 64, device="cuda", dtype=torch.bfloat16)
    got = []
    for a in products:
        G.gemm(a, b, out=out)
        got.append(C.conv3x3(x, w, out[-1]))
    torch.cuda.synchronize()
    for a, y in zip(products, got):
        G.gemm(a, b, out=out)
        torch.cuda.synchronize()
        assert torch.equal(y, C.conv3x3(x, w, out[-1]))
    native.raise_on_device_error()


@pytest.mark.gpu
def test_products_with_a_block_limit_wait_for_their_turn():
    """A limited product leaves the other SMs to another stream; the next one's blocks must not sit beside it while it runs."""
    a, b = (torch.randn(4096, 4096, device="cuda").bfloat16() for _ in range(2))
    outs = [torch.zeros(4096, 4096, device="cuda") for _ in range(2)]

    def products():
        for out in outs:
            G.gemm(a, b, a_mn=True, b_mn=True, out=out, accumulate=True, max_ctas=40)
        torch.cuda.synchronize()

    products()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as trace:
        products()
    times = sorted((e.time_range.start, e.time_range.end) for e in trace.events() if "gemm_bf16_kernel" in e.name)
    if len(times) != 2:
        pytest.skip("kernels are not traced here")
    assert times[1][0] >= times[0][1]


def _select(x):
    return R.topk(x, 40)


def _bias_per_pair(q, bias):
    return A.attention_forward(q, q, q, False, attn_bias=bias)


def _bias_per_pair_backward(q, bias):
    o, lse = _bias_per_pair(q, bias)
    return A.attention_backward(q, q, q, o, lse, q, False, attn_bias=bias)


def _bias_per_key(q, bias):
    return A.attention_forward(q, q, q, False, key_bias=bias[:, 0].contiguous())


@pytest.mark.gpu
@pytest.mark.parametrize("op,kernel,dim", [(_select, "rank_topk_kernel", 0), (_bias_per_pair, "attn_fwd_kernel", 64),
                                           (_bias_per_pair_backward, "attn_bwd_kernel", 64), (_bias_per_key, "attn_fwd_pair_kernel", 128)])
def test_kernels_that_start_in_order(op, kernel, dim):
    """Selection, whose blocks would pile up on a few SMs, and attention that reads a bias through an L1 of its own size."""
    a = torch.randn(8192, 4096, device="cuda").bfloat16()
    args = (torch.randn(500, 3000, device="cuda"),) if not dim else (torch.randn(24, 256, 8, dim, device="cuda").bfloat16(),
                                                                     torch.randn(24, 256, 256, device="cuda"))

    def both():
        G.gemm(a, a)
        op(*args)
        torch.cuda.synchronize()

    both()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as trace:
        both()
    times = sorted((e.time_range.start, e.time_range.end, e.name) for e in trace.events() if "kernel" in e.name)
    if not any("gemm_bf16_kernel" in t[2] for t in times):
        pytest.skip("kernels are not traced here")
    found = [i for i, t in enumerate(times) if f"{kernel}<" in t[2] or t[2].endswith(kernel)]
    assert found and found[0] > 0
    for i in found:
        assert times[i][0] >= max(t[1] for t in times[:i])


def _chain(a, b, steps=6):
    """Products that each read what the one before wrote, followed by the loss over the last two: two fp32 matrices and a number."""
    outs, x = [], a
    for _ in range(steps):
        x = G.gemm(x, b, alpha=1.0 / 32)
        outs.append(x)
    p, t = outs[-1].float(), outs[-2].float()
    return [*outs, multi.mse_forward(p, t)[0]]


def _synchronised(a, b, steps=6):
    """The same with a synchronisation behind every kernel."""
    outs, x = [], a
    for _ in range(steps):
        x = G.gemm(x, b, alpha=1.0 / 32)
        torch.cuda.synchronize()
        outs.append(x)
    p, t = outs[-1].float(), outs[-2].float()
    torch.cuda.synchronize()
    return [*outs, multi.mse_forward(p, t)[0]]


def _operands(seed):
    torch.manual_seed(seed)
    return torch.randn(2048, 1024, device="cuda").bfloat16(), torch.randn(1024, 1024, device="cuda").bfloat16()


@pytest.mark.gpu
@pytest.mark.parametrize("stream", ["legacy", "own"])
def test_one_stream(stream):
    """Chained kernels one after the other, and behind the fill of a counter that the loss kernel's blocks count on (mse_forward)."""
    s = torch.cuda.default_stream() if stream == "legacy" else torch.cuda.Stream()
    for seed in range(4):
        a, b = _operands(seed)
        want = _synchronised(a, b)
        torch.cuda.synchronize()
        with torch.cuda.stream(s):
            got = _chain(a, b)
        s.synchronize()
        assert all(torch.equal(x, y) for x, y in zip(got, want))
    native.raise_on_device_error()


@pytest.mark.gpu
@pytest.mark.parametrize("how", ["wait_event", "wait_stream"])
def test_two_streams_hand_a_buffer_back_and_forth(how):
    """Each product reads, on its stream, what the one before wrote on the other, into buffers that are used again."""
    a, b = _operands(0)
    streams, buffers = [torch.cuda.Stream() for _ in range(2)], [torch.empty_like(a) for _ in range(2)]
    x, want = a, []
    for _ in range(12):
        x = G.gemm(x, b, alpha=1.0 / 32)
        torch.cuda.synchronize()
        want.append(x.clone())
    torch.cuda.synchronize()
    x, got = a, []
    for i in range(12):
        here, other = streams[i & 1], streams[1 - (i & 1)]
        if how == "wait_event":
            here.wait_event(other.record_event())
        else:
            here.wait_stream(other)
        with torch.cuda.stream(here):
            G.gemm(x, b, alpha=1.0 / 32, out=buffers[i & 1])
            x = buffers[i & 1]
            got.append(x.clone())
            G.gemm(x, b, alpha=2.0)                 # one more chained kernel behind the copy
    torch.cuda.synchronize()
    assert all(torch.equal(x, y) for x, y in zip(got, want))
    native.raise_on_device_error()


@pytest.mark.gpu
def test_fill_between_chained_kernels():
    """A fill of the accumulated output stands between two products that add to it."""
    a, b = _operands(1)
    out = torch.empty(2048, 1024, device="cuda")
    want = G.gemm(a, b, out_dtype=torch.float32)
    torch.cuda.synchronize()
    for _ in range(20):
        G.gemm(a, b, out=out, accumulate=True)
        out.zero_()
        G.gemm(a, b, out=out, accumulate=True)
        got = out.clone()
        assert torch.equal(got, want)
    native.raise_on_device_error()
