"""The public ``st.nn`` / ``st.Tensor`` API on CUDA must run on the repository's kernels and agree with
the CPU path (fp32 PyTorch) to bf16 tolerance: per-op forward/backward checks of ``nn.functional``,
attention with additive biases and ragged lengths, and two small models trained through
``SpiralSession("cuda").trainer()`` whose per-op launch counters prove the kernel path was taken."""
import math

import pytest
import torch

import spiraltorch as st
from spiraltorch_b200.nn import functional as Fn
from spiraltorch_b200.ops import attention as A
from spiraltorch_b200.ops import conv as C
from spiraltorch_b200.ops import gemm as G
from spiraltorch_b200.ops import native, norm as N

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _rel(a, b):
    return ((a.float().cpu() - b.float().cpu()).abs().max() / b.float().abs().max().clamp(min=1e-6)).item()


def _bf(*ts):
    """Round test inputs to bf16-representable values: the kernels round operands to bf16 at their boundary, and
    comparing like with like keeps ReLU / max-pool decisions identical on both paths."""
    out = tuple(t.bfloat16().float() for t in ts)
    return out if len(out) > 1 else out[0]


def _grads(fn, inputs, dy):
    leaves = [t.detach().clone().requires_grad_(True) if t is not None and t.is_floating_point() else t for t in inputs]
    y = fn(*leaves)
    gs = torch.autograd.grad(y, [t for t in leaves if t is not None and t.requires_grad], dy.to(y.device))
    return y.detach(), gs


@pytest.mark.parametrize("act", [None, "relu", "gelu"])
def test_linear_forward_and_gradients(act):
    torch.manual_seed(0)
    x, w, b, dy = _bf(torch.randn(96, 40), torch.randn(40, 72) * 0.2, torch.randn(1, 72), torch.randn(96, 72))
    before = G.launch_count
    y_g, g_g = _grads(lambda a, ww, bb: Fn.linear(a, ww, bb, act), [x.to(DEV), w.to(DEV), b.to(DEV)], dy)
    assert G.launch_count - before == 3          # forward, data gradient, weight gradient on the tcgen05 GEMM
    y_c, g_c = _grads(lambda a, ww, bb: Fn.linear(a, ww, bb, act), [x, w, b], dy)
    assert _rel(y_g, y_c) < 2e-2
    for a, c in zip(g_g, g_c):
        assert _rel(a, c) < 3e-2


def test_layer_norm_with_residual_forward_and_gradients():
    torch.manual_seed(1)
    x, r, g, b, dy = _bf(torch.randn(200, 64), torch.randn(200, 64), 1 + 0.1 * torch.randn(1, 64),
                         0.1 * torch.randn(1, 64), torch.randn(200, 64))
    before = N.launch_count
    y_g, g_g = _grads(lambda a, gg, bb, rr: Fn.layer_norm(a, gg, bb, 1e-5, rr), [t.to(DEV) for t in (x, g, b, r)], dy)
    assert N.launch_count > before
    y_c, g_c = _grads(lambda a, gg, bb, rr: Fn.layer_norm(a, gg, bb, 1e-5, rr), [x, g, b, r], dy)
    assert _rel(y_g, y_c) < 3e-2
    for a, c in zip(g_g, g_c):
        assert _rel(a, c) < 4e-2


def test_embedding_forward_and_gradient():
    torch.manual_seed(2)
    w, dy = _bf(torch.randn(50, 32), torch.randn(63, 32))
    ids = torch.randint(0, 50, (7, 9))
    y_g, g_g = _grads(lambda ww: Fn.embedding(ids.to(DEV), ww), [w.to(DEV)], dy)
    y_c, g_c = _grads(lambda ww: Fn.embedding(ids, ww), [w], dy)
    assert _rel(y_g, y_c) < 1e-2 and _rel(g_g[0], g_c[0]) < 2e-2


@pytest.mark.parametrize("shape", [
    # (N, C, H, W, OC, kernel, stride, padding)
    (4, 64, 16, 16, 64, (3, 3), (1, 1), (1, 1)),      # implicit GEMM through 4-D TMA boxes
    (2, 8, 12, 12, 16, (3, 3), (1, 1), (1, 1)),       # 3x3 with few channels: im2col kernel + GEMM
    (3, 3, 11, 9, 5, (5, 3), (2, 1), (2, 0)),         # general geometry: unfold + GEMM
])
def test_conv2d_forward_and_gradients(shape):
    n, c, h, w_, oc, k, s, p = shape
    torch.manual_seed(3)
    x, w, b = _bf(torch.randn(n, c, h, w_), torch.randn(oc, c * k[0] * k[1]) / math.sqrt(c * k[0] * k[1]),
                  torch.randn(1, oc))
    f = lambda xx, ww, bb: Fn.conv2d(xx, ww, bb, k, s, p)          # noqa: E731
    y_c = f(x, w, b)
    dy = _bf(torch.randn_like(y_c))
    before = G.launch_count + C.launch_count
    y_g, g_g = _grads(f, [x.to(DEV), w.to(DEV), b.to(DEV)], dy)
    assert G.launch_count + C.launch_count - before >= 3
    _, g_c = _grads(f, [x, w, b], dy)
    assert _rel(y_g, y_c) < 2e-2
    for a, cc in zip(g_g, g_c):
        assert _rel(a, cc) < 3e-2


def test_max_pool_forward_and_gradient():
    torch.manual_seed(4)
    x, dy = _bf(torch.randn(3, 6, 10, 8), torch.randn(3, 6, 5, 4))
    y_g, g_g = _grads(Fn.max_pool2x2, [x.to(DEV)], dy)
    y_c, g_c = _grads(Fn.max_pool2x2, [x], dy)
    assert _rel(y_g, y_c) < 1e-2 and _rel(g_g[0], g_c[0]) < 1e-2


# ---- attention with biases, lengths, non-causal masks -------------------------------------------
@pytest.mark.parametrize("cfg", [
    # (B, S, H, D, causal, key_bias heads?, attn_bias heads?, lengths)
    (2, 256, 2, 64, False, False, False, None),
    (2, 200, 2, 64, False, True, None, [200, 77]),           # S not a multiple of 128, ragged lengths
    (3, 300, 1, 128, True, False, True, [300, 129, 1]),
    (2, 128, 2, 128, False, None, False, [0, 128]),          # an empty context gives zero rows
    (1, 384, 2, 64, True, True, True, None),
])
def test_attention_bias_and_lengths_forward_backward(cfg):
    B, S, H, D, causal, kb_heads, ab_heads, lengths = cfg
    torch.manual_seed(5)
    q, k, v = (torch.randn(B, S, H, D, device=DEV).bfloat16() for _ in range(3))
    kb = None if kb_heads is None else (torch.randn(B, H, S, device=DEV) if kb_heads else torch.randn(B, S, device=DEV))
    ab = None if ab_heads is None else (torch.randn(B, H, S, S, device=DEV) if ab_heads
                                        else torch.randn(B, S, S, device=DEV))
    ln = None if lengths is None else torch.tensor(lengths, device=DEV, dtype=torch.int32)
    scale = 1.0 / math.sqrt(D)
    o, lse = A.attention_forward(q, k, v, causal, scale, key_bias=kb, attn_bias=ab, lengths=ln)
    qf, kf, vf = (t.float().requires_grad_(True) for t in (q, k, v))
    o_ref, lse_ref = A.attention_reference(qf, kf, vf, causal, scale, key_bias=kb, attn_bias=ab, lengths=ln)
    assert _rel(o, o_ref) < 2e-2
    live = torch.isfinite(lse_ref)
    assert torch.equal(torch.isfinite(lse), live)
    assert (lse[live] - lse_ref[live]).abs().max().item() < 2e-2
    do = torch.randn(B, S, H, D, device=DEV).bfloat16()
    dq, dk, dv = A.attention_backward(q, k, v, o, lse, do, causal, scale, key_bias=kb, attn_bias=ab, lengths=ln)
    g = torch.autograd.grad(o_ref, (qf, kf, vf), do.float())
    for got, want in zip((dq, dk, dv), g):
        assert torch.isfinite(got.float()).all()
        assert _rel(got, want) < 4e-2
    torch.cuda.synchronize()
    assert native.read_error_word()[0] == 0


def test_tensor_scaled_dot_attention_with_biases_takes_the_kernel():
    torch.manual_seed(6)
    ctxs, seq, d = 3, 160, 64
    q, k, v = (torch.randn(ctxs * seq, d) for _ in range(3))
    zb, ab = torch.randn(ctxs, seq), torch.randn(ctxs * seq, seq)
    cpu = st.Tensor(q).scaled_dot_attention(st.Tensor(k), st.Tensor(v), contexts=ctxs, sequence=seq,
                                            z_bias=st.Tensor(zb), attn_bias=st.Tensor(ab))
    before = A.launch_count
    gpu = st.Tensor(q).cuda().scaled_dot_attention(st.Tensor(k).cuda(), st.Tensor(v).cuda(), contexts=ctxs,
                                                   sequence=seq, z_bias=st.Tensor(zb).cuda(),
                                                   attn_bias=st.Tensor(ab).cuda())
    assert A.launch_count == before + 1
    assert _rel(gpu.torch(), cpu.torch()) < 2e-2
    ln_cpu = st.Tensor(q).layer_norm_affine_add(st.Tensor(k), st.Tensor(torch.ones(1, d)), st.Tensor(torch.zeros(1, d)))
    ln_gpu = st.Tensor(q).cuda().layer_norm_affine_add(st.Tensor(k).cuda(), st.Tensor(torch.ones(1, d)).cuda(),
                                                       st.Tensor(torch.zeros(1, d)).cuda())
    assert _rel(ln_gpu.torch(), ln_cpu.torch()) < 3e-2


def test_functional_attention_is_differentiable_on_the_kernels():
    torch.manual_seed(7)
    q, k, v = (torch.randn(2, 192, 64, device=DEV, requires_grad=True) for _ in range(3))
    zb = torch.randn(2, 192, device=DEV)
    out = Fn.scaled_dot_attention(q, k, v, z_bias=zb, lengths=torch.tensor([192, 100], device=DEV))
    out.square().sum().backward()
    qc, kc, vc = (t.detach().cpu().requires_grad_(True) for t in (q, k, v))
    ref = Fn.scaled_dot_attention(qc, kc, vc, z_bias=zb.cpu(), lengths=torch.tensor([192, 100]))
    ref.square().sum().backward()
    assert _rel(out.detach(), ref.detach()) < 3e-2
    for a, c in zip((q, k, v), (qc, kc, vc)):
        assert _rel(a.grad, torch.nan_to_num(c.grad)) < 6e-2


# ---- models through the public trainer ------------------------------------------------------------
def _train(device: str, build, epochs: int, lr: float = 5e-2):
    model, loss, batches = build()
    sess = st.SpiralSession(device, seed=11)
    if device == "cuda":
        model.to("cuda")
        batches = [(x.cuda(), y.cuda()) for x, y in batches]
    trainer = sess.trainer(fallback_learning_rate=lr)
    losses = [trainer.train_epoch(model, loss, batches).average_loss for _ in range(epochs)]
    return losses, {n: t.torch().cpu() for n, t in model.state_dict()}


def _readme_model():
    g = torch.Generator().manual_seed(0)
    x = torch.randn(256, 8, generator=g)
    wv = torch.randn(8, 1, generator=g) / math.sqrt(8)
    y = torch.sin(x @ wv) + 0.01 * torch.randn(256, 1, generator=g)
    model = st.nn.Sequential()
    fc1 = st.nn.Linear(8, 32, name="fc1").init_normal(0.3, seed=1)
    head = st.nn.Linear(32, 1, name="head").init_normal(0.3, seed=2)
    model.add(fc1); model.add(st.nn.Relu()); model.add(head)
    batches = [(st.Tensor(x[i:i + 32]), st.Tensor(y[i:i + 32])) for i in range(0, 256, 32)]
    return model, st.nn.MeanSquaredError(), batches


def test_readme_model_trains_on_the_kernels_and_matches_cpu():
    counts0 = dict(Fn.launch_counts)
    gemm0 = G.launch_count
    gpu_losses, gpu_state = _train("cuda", _readme_model, 6)
    assert Fn.launch_counts["linear"] - counts0["linear"] >= 6 * 8 * 2        # two Linear layers per batch
    assert G.launch_count - gemm0 >= 6 * 8 * 2 * 3                            # fwd + dgrad + wgrad each
    cpu_losses, cpu_state = _train("cpu", _readme_model, 6)
    assert gpu_losses[-1] < gpu_losses[0]
    for a, b in zip(gpu_losses, cpu_losses):
        assert abs(a - b) < 3e-2 * max(1.0, abs(b)), (gpu_losses, cpu_losses)
    for name in cpu_state:
        assert _rel(gpu_state[name], cpu_state[name]) < 5e-2, name


def test_zconv_recipe_trains_on_the_kernels_and_matches_cpu():
    from spiraltorch_b200.models import recipes

    def build():
        model, loss, batches, _ = recipes.zconv_classification(seed=0)
        return model, loss, batches
    counts0 = dict(Fn.launch_counts)
    gpu_losses, gpu_state = _train("cuda", build, 4, lr=0.5)
    for op in ("conv2d", "max_pool2x2", "linear"):
        assert Fn.launch_counts[op] - counts0[op] >= 4 * 4, op
    cpu_losses, cpu_state = _train("cpu", build, 4, lr=0.5)
    assert gpu_losses[-1] < gpu_losses[0]
    for a, b in zip(gpu_losses, cpu_losses):
        assert abs(a - b) < 5e-2 * max(1.0, abs(b)), (gpu_losses, cpu_losses)
    torch.cuda.synchronize()
    assert native.read_error_word()[0] == 0


# ---- whole-sequence recurrent scans ---------------------------------------------------------------------
@pytest.mark.parametrize("cell,hidden,dilation", [("tanh", 32, 1), ("wave", 64, 2), ("wave", 32, 1), ("wave", 16, 3),
                                                  ("lstm", 64, 1), ("lstm", 40, 1)])
def test_rnn_sequence_kernel_matches_step_loop(cell, hidden, dilation):
    from spiraltorch_b200.ops import recurrent as R
    torch.manual_seed(8)
    B, T, I = 9, 7, 24
    G_ = {"tanh": 1, "wave": 2, "lstm": 4}[cell]
    x, w_ih, w_hh, b, dh = _bf(torch.randn(B, T, I), torch.randn(I, G_ * hidden) * 0.3,
                               torch.randn(hidden, G_ * hidden) * 0.3, torch.randn(1, G_ * hidden) * 0.1,
                               torch.randn(B, hidden))
    f = lambda *a: R.rnn_sequence(*a, cell, dilation)       # noqa: E731
    before = R.launch_count
    y_g, g_g = _grads(f, [t.to(DEV) for t in (x, w_ih, w_hh, b)], dh)
    assert R.launch_count - before == 2                     # one forward scan, one backward scan
    y_c, g_c = _grads(f, [x, w_ih, w_hh, b], dh)
    assert _rel(y_g, y_c) < 2e-2
    for a, c in zip(g_g, g_c):
        assert _rel(a, c) < 4e-2
    torch.cuda.synchronize()
    assert native.read_error_word()[0] == 0


def test_wave_rnn_module_training_step_runs_on_the_scan_kernel():
    from spiraltorch_b200.ops import recurrent as R
    torch.manual_seed(9)
    layer = st.nn.WaveRnn("wave", 32, 64, 16, dilation=2)
    cpu_x, cpu_g = torch.randn(32, 16 * 32), torch.randn(32, 64)
    ref_dx = layer.backward(st.Tensor(cpu_x), st.Tensor(cpu_g)).torch()
    ref_acc = {p.name: p.gradient.clone() for p in layer.parameters()}
    layer.zero_accumulators()
    layer.to("cuda")
    before = R.launch_count
    y = layer.forward(st.Tensor(cpu_x).cuda())
    dx = layer.backward(st.Tensor(cpu_x).cuda(), st.Tensor(cpu_g).cuda()).torch()
    assert R.launch_count - before == 3                     # forward scan; forward + backward scan of backward()
    assert y.shape() == (32, 64)
    assert _rel(dx, ref_dx) < 5e-2
    for p in layer.parameters():
        assert _rel(p.gradient, ref_acc[p.name]) < 5e-2, p.name


def _wave_model(seed):
    torch.manual_seed(seed)
    m = st.nn.Sequential()
    m.add(st.nn.WaveRnn("wave", 32, 64, 16))
    m.add(st.nn.Linear(64, 8, name="head"))
    m.to("cuda")
    return m


def test_graphed_train_step_matches_eager_steps_and_reports_non_finite_inputs():
    loss = st.nn.MeanSquaredError()
    torch.manual_seed(11)
    batches = [(torch.randn(32, 16 * 32, device="cuda"), torch.randn(32, 8, device="cuda")) for _ in range(4)]
    eager, graphed = _wave_model(5), _wave_model(5)
    step = st.nn.GraphedTrainStep(graphed, loss, st.Tensor._wrap(batches[0][0]), st.Tensor._wrap(batches[0][1]), learning_rate=1e-2)
    for p, q in zip(eager.parameters(), graphed.parameters()):
        assert torch.equal(p.value, q.value)                      # warm-up and capture left the parameters untouched
    for x, y in batches:
        xe, ye = st.Tensor._wrap(x), st.Tensor._wrap(y)
        pred = eager.forward(xe)
        want = float(loss.forward(pred, ye).torch())
        eager.backward(xe, loss.backward(pred, ye))
        eager.apply_step(1e-2)
        got = float(step(xe, ye))
        assert got == pytest.approx(want, rel=2e-3)
    step.check()
    assert step.replays == 4
    for p, q in zip(eager.parameters(), graphed.parameters()):
        assert _rel(q.value, p.value) < 2e-3, p.name
    # an eager forward after graphed training must see the trained weights, not a stale low-precision copy
    xe = st.Tensor._wrap(batches[0][0])
    assert _rel(graphed.forward(xe).torch(), eager.forward(xe).torch()) < 2e-2
    bad = batches[0][1].clone()
    bad[0, 0] = float("nan")
    step(xe, st.Tensor._wrap(bad))
    with pytest.raises(st.TensorError):
        step.check()


@pytest.mark.gpu
@pytest.mark.parametrize("sizes", [[1], [5, 0, 1024], [4097, 33, 70000, 2], [7] * 100, [3_000_001, 1]])
def test_tensor_lists_in_one_launch(sizes):
    """Checks, divisions and updates of lists: single elements, block edges, more tensors than one launch holds."""
    from spiraltorch_b200.ops import multi
    g = torch.Generator(device="cuda").manual_seed(1)
    ts = [torch.randn(n, generator=g, device="cuda") for n in sizes if n]
    assert multi.takes(ts) and not multi.takes(ts + [torch.empty(0, device="cuda")]) and not multi.takes([ts[0].cpu()])
    assert not multi.takes([torch.randn(4, 6, device="cuda").t()]) and not multi.takes([ts[0].double()])
    assert multi.first_nonfinite(ts) is None
    out, bad = multi.divided(ts, 3.0)
    # correctly rounded, as on the CPU
    assert bad is None and all(torch.equal(o.cpu(), t.cpu() / 3.0) for o, t in zip(out, ts))
    values = [torch.randn(t.shape, generator=g, device="cuda") for t in ts]
    want, versions = [v - 0.01 * t for v, t in zip(values, ts)], [v._version for v in values]
    multi.descend_(values, ts, 0.01)
    assert all(torch.equal(v, w) and v._version > n for v, w, n in zip(values, want, versions))
    for k, odd in ((len(ts) - 1, float("nan")), (len(ts) // 2, float("-inf"))):
        ts[k][-1] = odd
        assert multi.first_nonfinite(ts) == k and multi.divided(ts, 2.0)[1] == k


@pytest.mark.gpu
@pytest.mark.parametrize("rows,cols", [(1, 1), (3, 341), (32, 32), (33, 32), (4096, 100)])
def test_mean_squared_error_in_one_launch(rows, cols):
    import spiraltorch as st
    p, t = torch.randn(rows, cols, device="cuda"), torch.randn(rows, cols, device="cuda")
    loss = st.nn.MeanSquaredError()
    ref = (p.double() - t.double()).pow(2).mean().item()
    assert abs(loss.forward(st.Tensor(p), st.Tensor(t)).torch().item() - ref) <= 1e-6 * ref
    want = torch.autograd.functional.jacobian(lambda x: (x - t).pow(2).mean(), p) if p.numel() < 2000 else 2 * (p - t) / p.numel()
    assert torch.allclose(loss.backward(st.Tensor(p), st.Tensor(t)).torch(), want, rtol=3e-7, atol=0)     # two roundings
    t[-1, -1] = float("inf")
    for call in (loss.forward, loss.backward):
        with pytest.raises(Exception, match="non-finite"):
            call(st.Tensor(p), st.Tensor(t))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("rows,d", [(1, 8), (7, 256), (9, 264), (2400, 768), (5000, 1024), (3, 1032), (2500, 2048)])
def test_norm_with_a_warp_per_row(rows, d, rms, dtype):
    """Vector counts 1 to 4 per lane, partial ones, more rows than a grid holds, the first width past the warp form (bf16
    only), residual and gradient sums; bounds: one rounding of the output type, fp32 sums over the rows."""
    if dtype == torch.float32 and d > 1024:
        assert not N.takes_f32(d)
        return
    torch.manual_seed(rows + d)
    x, r, dy, dres = (torch.randn(rows, d, device=DEV).to(dtype) for _ in range(4))
    g, b = torch.randn(d, device=DEV).to(dtype), (None if rms else torch.randn(d, device=DEV).to(dtype))
    tol = 2 ** -8 if dtype == torch.bfloat16 else 2e-6
    y, s, mean, rstd = N.norm_forward(x, g, b, 1e-5, rms, r)
    assert torch.equal(s, x + r)
    sd = s.double()
    mu = 0 if rms else sd.mean(-1, keepdim=True)
    rs = torch.rsqrt((sd - mu).pow(2).mean(-1, keepdim=True) + 1e-5)
    want = (sd - mu) * rs * g.double() + (0 if rms else b.double())
    assert ((y.double() - want).abs() <= tol * want.abs() + 1e-5).all()
    dg, db = torch.full((d,), 0.5, device=DEV), (None if rms else torch.full((d,), 0.25, device=DEV))
    dx = N.norm_backward(dy, s, g, mean, rstd, rms, dg, db, True, dres)
    xh, gy = (sd - mu) * rs, dy.double() * g.double()
    m2 = 0 if rms else gy.mean(-1, keepdim=True)
    want = rs * (gy - m2 - xh * (gy * xh).mean(-1, keepdim=True)) + dres.double()
    assert ((dx.double() - want).abs() <= tol * want.abs() + 2e-5).all()
    assert torch.allclose(dg.double(), 0.5 + (dy.double() * xh).sum(0), rtol=1e-5, atol=1e-3)
    if not rms:
        assert torch.allclose(db.double(), 0.25 + dy.double().sum(0), rtol=1e-5, atol=1e-3)


def test_layer_norm_backward_reads_the_values_of_the_forward():
    x, g, b = (torch.randn(s, device=DEV, requires_grad=True) for s in ((6, 64), (1, 64), (1, 64)))
    want = torch.autograd.grad(Fn.layer_norm(x, g, b).sum(), (x, g, b))
    h = x * 1.0
    y = Fn.layer_norm(h, g, b).sum()
    with torch.no_grad():
        h.mul_(3.0)
        g.add_(1.0)
    assert all(torch.equal(p, q) for p, q in zip(torch.autograd.grad(y, (x, g, b)), want))


@pytest.mark.parametrize("B,Sq,Sk,H,D,causal,heads,lengths", [
    (3, 130, 130, 2, 64, False, False, [130, 0, 1]), (4, 257, 257, 1, 128, True, True, [128, 129, 127, 257]),
    (2, 300, 77, 1, 64, False, True, None), (2, 100, 385, 2, 128, False, False, [385, 90]), (1, 1, 1, 1, 64, True, False, None),
    (2, 200, 200, 3, 64, False, None, [199, 64])])
def test_attention_with_key_bias_and_lengths_on_the_pair_kernel(B, Sq, Sk, H, D, causal, heads, lengths):
    """Empty, one-key and tile-edge lengths, query tiles beyond them, unequal sequence lengths, bias per head, masked keys;
    forward and both backward passes against the general kernels' arithmetic in fp32.  P and dS are bf16: 2^-8 of the
    largest value."""
    torch.manual_seed(Sq + Sk + D)
    q, do = (torch.randn(B, Sq, H, D, device=DEV).bfloat16() for _ in range(2))
    k, v = (torch.randn(B, Sk, H, D, device=DEV).bfloat16() for _ in range(2))
    kb = None
    if heads is not None:
        kb = torch.randn(*((B, H, Sk) if heads else (B, Sk)), device=DEV) * 2
        kb[..., Sk // 3] = float("-inf")
    ln = None if lengths is None else torch.tensor(lengths, device=DEV, dtype=torch.int32)
    o32 = torch.empty(B, Sq, H, D, device=DEV)
    o, lse = A.attention_forward(q, k, v, causal, None, key_bias=kb, lengths=ln, out32=o32)
    qf, kf, vf = (t.float().requires_grad_(True) for t in (q, k, v))
    ro, rlse = A.attention_reference(qf, kf, vf, causal, 1 / math.sqrt(D), key_bias=kb, lengths=ln)
    close = lambda x, y: (x.float() - y).abs().max() <= 2e-2 * y.abs().max().clamp(min=1e-3)  # noqa: E731
    assert close(o, ro) and close(o32, ro) and torch.equal(o, o32.bfloat16())
    live = torch.isfinite(rlse)
    assert torch.equal(live, torch.isfinite(lse)) and (lse[live] - rlse[live]).abs().max() < 1e-2 if live.any() else True
    grads = torch.autograd.grad(torch.nan_to_num(ro), (qf, kf, vf), do.float(), allow_unused=True)
    grads = [torch.nan_to_num(g) for g in grads]
    f32 = [torch.full(t.shape, float("nan"), device=DEV) for t in (q, k, v)]
    given = torch.empty_like(do)
    A.attention_backward(q, k, v, o, lse, given, causal, None, *f32, key_bias=kb, lengths=ln, do32=do.float())
    assert torch.equal(given, do)
    b16 = A.attention_backward(q, k, v, o, lse, do, causal, None, key_bias=kb, lengths=ln)
    for g, f, h in zip(grads, f32, b16):
        assert close(f, g) and torch.equal(f.bfloat16(), h)


def test_attention_backward_does_not_read_the_returned_output():
    q, k, v = (torch.randn(3, 150, 64, device=DEV, requires_grad=True) for _ in range(3))
    g = torch.randn(3, 150, 64, device=DEV)
    want = torch.autograd.grad(Fn.scaled_dot_attention(q, k, v), (q, k, v), g)
    y = Fn.scaled_dot_attention(q, k, v)
    with torch.no_grad():
        y.detach().zero_()
    assert all(torch.equal(a, b) for a, b in zip(torch.autograd.grad(y, (q, k, v), g), want))


@pytest.mark.parametrize("B,width,hidden,out", [(1, 8, 8, 8), (37, 72, 264, 64), (130, 128, 1032, 256), (1000, 512, 2048, 512)])
def test_contrastive_step_written_out_over_the_kernels(B, width, hidden, out):
    """Against the autograd form (which a hook selects), both measured from 64 bits: gradients are sums of bf16 products, so
    neither may be further off than the rounding of its operands, and the written-out form not further than the other."""
    from spiraltorch_b200.models import contrastive as M
    enc = M.ContrastiveEncoder(width, hidden, out, device=DEV, seed=B)
    for p in list(enc.gammas) + list(enc.betas) + list(enc.biases):
        p.data.add_(0.1 * torch.randn(p.shape, device=DEV).to(p.dtype))
    base = torch.randn(B, width, device=DEV)
    assert M._schedulable(enc, base, 0.1) and not M._schedulable(enc, base.double(), 0.1)

    def step():
        enc.zero_grad(set_to_none=True)
        loss = M.contrastive_step(enc, base, 0.1, seed=5)
        assert not loss.requires_grad
        return loss.item(), [p.grad.clone() for p in enc.parameters()]
    loss, grads = step()
    handle = enc.register_forward_hook(lambda *a: None)
    assert not M._schedulable(enc, base, 0.1)
    loss_a, grads_a = step()
    handle.remove()
    p64 = [p.detach().double().requires_grad_(True) for p in enc.parameters()]
    g = torch.Generator(device=DEV).manual_seed(5)
    z = []
    for n in [torch.randn(base.shape, generator=g, device=DEV) for _ in range(2)]:
        h = base.double() + 0.1 * n.double()
        for i in range(3):
            h = h @ p64[i].t() + p64[3 + i]
            if i < 2:
                h = torch.nn.functional.gelu(torch.nn.functional.layer_norm(h, h.shape[-1:], p64[6 + i], p64[8 + i], 1e-5), approximate="tanh")
        z.append(torch.nn.functional.normalize(h, dim=-1))
    want = torch.nn.functional.cross_entropy(z[0] @ z[1].t() / 0.1, torch.arange(B, device=DEV))
    want.backward()
    assert abs(loss - want.item()) <= 2e-2 * max(want.item(), 1.0)
    for a, b, p in zip(grads, grads_a, p64):
        scale = p.grad.norm()
        assert a.dtype == torch.bfloat16 and a.shape == p.shape
        if B > 1:       # one pair has no negatives: its gradients are rounding noise around zero
            assert (a - p.grad).norm() <= max(1.3 * (b - p.grad).norm().item(), 0.01 * scale.item())
    first = [p.grad.clone() for p in enc.parameters()]
    M.contrastive_step(enc, base, 0.1, seed=5)                        # gradients accumulate
    assert all((p.grad - 2 * f).norm() <= 0.02 * (2 * f).norm() + 1e-6 for p, f in zip(enc.parameters(), first)) or B == 1


@pytest.mark.parametrize("cell,B,T,H,dilation", [
    ("tanh", 1, 1, 1, 1), ("tanh", 5, 9, 33, 1), ("tanh", 900, 3, 128, 1), ("tanh", 3, 5, 129, 1), ("wave", 7, 12, 5, 1),
    ("wave", 6, 40, 64, 2), ("wave", 9, 11, 96, 3), ("wave", 900, 7, 72, 5), ("wave", 3, 130, 100, 60), ("wave", 2, 4, 128, 9),
    ("lstm", 4, 7, 32, 1), ("lstm", 5, 6, 65, 1), ("lstm", 700, 4, 96, 1), ("lstm", 2, 3, 97, 1)])
def test_recurrent_scans_with_weights_in_registers(cell, B, T, H, dilation):
    """Sizes at and past the register forms' edges, units that do not fill a warp, one and four rows per CTA, skip histories
    in shared and in global memory, dilations of 1 and beyond the sequence.  The scan is fp32 between bf16 projections:
    2^-8 of the largest value, per step of error growth at most."""
    from spiraltorch_b200.ops import recurrent as R
    torch.manual_seed(H + B)
    gates, width = {"tanh": 1, "wave": 2, "lstm": 4}[cell], 16
    x = torch.randn(B, T, width, device=DEV).bfloat16().float()
    w_ih, w_hh, b = (((torch.rand(s, device=DEV) * 2 - 1) / H ** 0.5).bfloat16().float() for s in
                     ((width, gates * H), (H, gates * H), (1, gates * H)))
    leaves = [t.requires_grad_(True) for t in (x, w_ih, w_hh, b)]
    assert R.scan_supported(H, cell)
    h = R.rnn_sequence(*leaves, cell, dilation)
    g = torch.randn(B, H, device=DEV)
    grads = torch.autograd.grad(h, leaves, g)
    wide = [t.detach().double().requires_grad_(True) for t in leaves]
    want = R.rnn_sequence_reference(*wide, cell, dilation)
    assert (h - want).abs().max() <= 1e-4
    for a, r in zip(grads, torch.autograd.grad(want, wide, g.double())):
        assert (a - r).norm() <= 5e-3 * r.norm() + 1e-6


@pytest.mark.parametrize("rows,cols", [(1, 8), (33, 72), (1000, 264), (1024, 64)])
def test_column_sums_of_short_matrices(rows, cols):
    from spiraltorch_b200.ops import elementwise as E
    x = torch.randn(rows, cols, device=DEV).bfloat16()
    s = E.colsum(x)
    assert torch.allclose(s.double(), x.double().sum(0), rtol=1e-5, atol=1e-4) and torch.equal(s, E.colsum(x))


def test_updates_renew_the_cached_bf16_values():
    """The copy that the next forward reads is that of the updated values, and a graph built before keeps the old one."""
    from spiraltorch_b200.ops import multi
    w, other, g = (torch.randn(40, 24, device=DEV) for _ in range(3))
    old = G.cached_bf16(w)
    kept = old.clone()
    multi.descend_([w, other], [g, g], 0.5)
    new = G.cached_bf16(w)
    assert torch.equal(old, kept) and new.data_ptr() != old.data_ptr() and torch.equal(new, w.bfloat16())
    assert not G.has_cached_bf16(other)
    w.mul_(2.0)                                      # a change the cache has not seen
    assert not G.has_cached_bf16(w) and torch.equal(G.cached_bf16(w), w.bfloat16())


def test_trainer_still_refuses_gradients_that_overflow_in_accumulation():
    class Doubled(st.nn.Linear):
        def backward(self, x, grad):
            out = super().backward(x, grad)
            self.weight.gradient.mul_(float("inf"))
            return out
    lin = Doubled("fc", 8, 8)
    lin.init_normal(0.1, seed=1)
    trainer = st.SpiralSession("cuda", seed=1).trainer(fallback_learning_rate=0.1)
    trainer.prepare(lin)
    batch = (st.Tensor(torch.randn(16, 8, device=DEV)), st.Tensor(torch.randn(16, 8, device=DEV)))
    with pytest.raises(Exception, match="non-finite gradient"):
        trainer.train_epoch(lin, st.nn.MeanSquaredError(), [batch])
    assert all(p.gradient is None for p in lin.parameters())


@pytest.mark.parametrize("rows,d,residual", [(1, 8, False), (33, 128, True), (2500, 264, False), (1300, 1024, True)])
def test_layer_norm_of_fp32_tensors_has_the_values_of_the_bf16_form(rows, d, residual):
    """Bit for bit, where both take the same kernel: operands, output and input gradient are bf16 values wherever the tensors are fp32.  A wider result moved
    elements across the ReLU behind it, and with them whole gradients of small batches."""
    torch.manual_seed(rows + d)
    x, dy = torch.randn(rows, d, device=DEV), torch.randn(rows, d, device=DEV)
    g, b, r = (torch.randn(s, device=DEV) for s in ((1, d), (1, d), (rows, d)))
    r = r if residual else None
    leaves = [t.requires_grad_(True) for t in (x, g, b)]
    y = Fn.layer_norm(*leaves, residual=r)
    got = torch.autograd.grad(y, leaves, dy)
    xb, gb, bb, rb = (None if t is None else t.detach().bfloat16() for t in (x, g.reshape(-1), b.reshape(-1), r))
    want, summed, mean, rstd = N.norm_forward(xb, gb, bb, 1e-5, False, rb)
    dg, db = torch.empty(d, device=DEV), torch.empty(d, device=DEV)
    dx = N.norm_backward(dy.bfloat16(), xb if summed is None else summed, gb, mean, rstd, False, dg, db, False)
    assert torch.equal(y, want.float()) and torch.equal(got[0], dx.float())
    assert torch.equal(got[1].reshape(-1), dg) and torch.equal(got[2].reshape(-1), db)


def test_contrastive_step_under_autocast_takes_the_autograd_form():
    """Its similarity products come out in 16 bits there, which the kernels of the written-out form must never see."""
    from spiraltorch_b200.models import contrastive as M
    enc = M.ContrastiveEncoder(64, 128, 64, device=DEV, seed=1)
    base = torch.randn(48, 64, device=DEV)

    def step(hooked):
        enc.zero_grad(set_to_none=True)
        handle = enc.register_forward_hook(lambda *a: None) if hooked else None
        loss = M.contrastive_step(enc, base, 0.1, seed=5)
        if handle is not None:
            handle.remove()
        return [loss] + [p.grad.clone() for p in enc.parameters()]
    with torch.autocast("cuda", dtype=torch.bfloat16):
        assert not M._schedulable(enc, base, 0.1)
        got, want = step(False), step(True)
    assert M._schedulable(enc, base, 0.1)
    assert all(torch.isfinite(a).all() and (a.float() - b.float()).norm() <= 1e-2 * b.float().norm() for a, b in zip(got, want))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float64])
def test_contrastive_step_does_not_depend_on_the_default_dtype(dtype):
    from spiraltorch_b200.models import contrastive as M
    enc = M.ContrastiveEncoder(64, 128, 64, device=DEV, seed=1)
    base = torch.randn(48, 64, device=DEV)

    def step():
        enc.zero_grad(set_to_none=True)
        assert M._schedulable(enc, base, 0.1)
        return [M.contrastive_step(enc, base, 0.1, seed=5)] + [p.grad.clone() for p in enc.parameters()]
    want = step()
    torch.set_default_dtype(dtype)
    try:
        got = step()
    finally:
        torch.set_default_dtype(torch.float32)
    assert all(a.dtype == b.dtype and torch.allclose(a.float(), b.float(), rtol=1e-2, atol=1e-5) for a, b in zip(got, want))


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("Sq,Sk,D,causal,lengths", [(200, 200, 64, False, [130, 64, 1, 200]), (300, 300, 128, True, [129, 256, 127, 0]),
                                                    (100, 385, 64, False, [90, 385, 260, 5])])
def test_padding_that_is_not_finite_stays_out_of_attention_with_lengths(Sq, Sk, D, causal, lengths, bad):
    """Queries at and beyond the length give zeros and queries below it do not see the keys beyond it, whatever stands there;
    the padded queries leave nothing in dV and in the live rows of dQ."""
    torch.manual_seed(Sq + D)
    B, ln = len(lengths), torch.tensor(lengths, device=DEV, dtype=torch.int32)
    q, do = torch.randn(B, Sq, D, device=DEV), torch.randn(B, Sq, D, device=DEV)
    k, v = torch.randn(B, Sk, D, device=DEV), torch.randn(B, Sk, D, device=DEV)
    zb = torch.randn(B, Sk, device=DEV)
    dead_q = torch.arange(Sq, device=DEV) >= ln[:, None]
    dead_k = torch.arange(Sk, device=DEV) >= ln[:, None]

    def run(q, k):
        leaves = [t.detach().clone().requires_grad_(True) for t in (q, k, v)]
        o = Fn.scaled_dot_attention(*leaves, z_bias=zb, causal=causal, lengths=ln)
        return [o.detach()] + list(torch.autograd.grad(o, leaves, do))
    fill = lambda t, dead: torch.where(dead[..., None], torch.full_like(t, bad), t)  # noqa: E731
    clean, spoilt_q, spoilt = run(q, k), run(fill(q, dead_q), k), run(fill(q, dead_q), fill(k, dead_k))
    assert not clean[0][dead_q].any()
    for got in (spoilt_q, spoilt):
        assert torch.equal(got[0], clean[0])
    assert torch.equal(spoilt_q[1][~dead_q], clean[1][~dead_q]) and torch.equal(spoilt_q[3], clean[3])
    ref = Fn.scaled_dot_attention(fill(q, dead_q).cpu(), fill(k, dead_k).cpu(), v.cpu(), z_bias=zb.cpu(), causal=causal, lengths=ln.cpu())
    assert torch.isfinite(ref).all() and (clean[0].cpu() - ref).abs().max() <= 2e-2 * ref.abs().max()


def test_updates_refuse_or_broadcast_gradients_of_another_shape():
    """As ``value.sub_(lr * gradient)`` does; the launch over all parameters reads as many elements as the value has."""
    from spiraltorch_b200.ops import multi
    lin = st.nn.Linear("fc", 8, 16)
    lin.init_normal(0.1, seed=1)
    lin.to(DEV)
    before = [p.value.clone() for p in lin.parameters()]
    for p in lin.parameters():
        p.gradient = torch.ones_like(p.value)
    lin.weight.gradient = torch.arange(16.0, device=DEV).reshape(1, 16)
    lin.apply_step(0.5)
    assert torch.equal(lin.weight.value, before[0] - 0.5 * torch.arange(16.0, device=DEV)) and torch.equal(lin.bias.value, before[1] - 0.5)
    lin.weight.gradient = torch.ones(3, 5, device=DEV)
    with pytest.raises(RuntimeError):
        lin.apply_step(0.5)
    assert not multi.descend_([lin.weight.value], [torch.ones(16, device=DEV)], 0.5)


def test_parameters_over_one_storage_get_both_updates():
    from spiraltorch_b200.nn.modules import Parameter
    from spiraltorch_b200.ops import multi

    class Tied(st.nn.Linear):
        twin = None

        def parameters(self):
            return super().parameters() + ([self.twin] if self.twin else [])
    lin = Tied("fc", 300, 400)
    lin.init_normal(0.1, seed=1)
    lin.to(DEV)
    for twin in (lin.weight.value, lin.weight.value.view(-1)[1000:].view(-1, 1)):      # the whole storage, and a part of it
        lin.twin = Parameter("twin", twin)
        assert lin.twin.value.data_ptr() == twin.data_ptr()
        want = lin.weight.value.clone()
        for p in lin.parameters():
            p.gradient = torch.randn_like(p.value)
        want -= 0.5 * lin.weight.gradient
        want.view(-1)[want.numel() - twin.numel():] -= 0.5 * lin.twin.gradient.reshape(-1)
        lin.apply_step(0.5)
        assert torch.equal(lin.weight.value, want)
    a, g = torch.zeros(100, device=DEV), torch.zeros(200, device=DEV)
    for values, grads, ok in (([a[:50], a[50:]], [g[:50], g[50:100]], True), ([a[50:], a[:51]], [g[:50], g[50:101]], False),
                              ([a[:50]], [a[50:]], True), ([a[:50]], [a[49:99]], False), ([a[60:]], [a[21:61]], False),
                              ([a[10:20], g[:10]], [a[:10], a[20:30]], True), ([a[10:20], g[:10]], [g[10:20], a[10:20]], False)):
        assert multi.descend_(values, grads, 0.5) is ok
    lin.twin = Parameter("twin", torch.zeros(300, 400, device=DEV))
    lin.twin.gradient, lin.weight.gradient = lin.weight.value, torch.ones(300, 400, device=DEV)      # read as another step writes it
    want = lin.weight.value - 0.5
    lin.apply_step(0.5)
    assert torch.equal(lin.weight.value, want) and torch.equal(lin.twin.value, -0.5 * want)


def test_replaced_methods_of_one_module_or_parameter_are_still_heard():
    def trained(lin):
        trainer = st.SpiralSession("cuda", seed=1).trainer(fallback_learning_rate=0.1)
        trainer.prepare(lin)
        trainer.train_epoch(lin, st.nn.MeanSquaredError(), [(st.Tensor(torch.randn(16, 8, device=DEV)), st.Tensor(torch.randn(16, 8, device=DEV)))])

    lin = st.nn.Linear("fc", 8, 8)
    lin.init_normal(0.1, seed=1)
    plain_backward = lin.backward

    def backward(x, grad):
        out = plain_backward(x, grad)
        lin.weight.gradient.mul_(float("inf"))
        return out
    lin.backward = backward
    with pytest.raises(Exception, match="non-finite gradient"):
        trained(lin)
    assert all(p.gradient is None for p in lin.parameters())
    del lin.backward
    before, calls = [p.value.clone() for p in lin.parameters()], []
    lin.weight.apply_step = lambda lr: calls.append(lr)                       # a parameter that its owner froze
    lin.bias.accumulate = lambda grad: calls.append(grad)
    trained(lin)
    assert len(calls) == 2 and all(torch.equal(p.value, b) for p, b in zip(lin.parameters(), before))


def test_contrastive_step_runs_the_hooks_of_accumulation_nodes():
    from spiraltorch_b200.models import contrastive as M
    enc = M.ContrastiveEncoder(64, 128, 64, device=DEV, seed=1)
    base = torch.randn(48, 64, device=DEV)
    params = list(enc.parameters())
    M.contrastive_step(enc, base, 0.1, seed=5)
    want = [p.grad.clone() for p in params]
    views = [p.expand_as(p) for p in params]                  # graphs that keep the nodes, and with them their hooks, alive
    seen = []
    for v in views:
        v.grad_fn.next_functions[0][0].register_hook(lambda *a: seen.append(1))
    assert not M._schedulable(enc, base, 0.1)
    enc.zero_grad(set_to_none=True)
    M.contrastive_step(enc, base, 0.1, seed=5)
    assert len(seen) == len(params) == 10
    assert all((p.grad.float() - w.float()).norm() <= 2e-2 * w.float().norm() for p, w in zip(params, want))
    views.pop(0)
    assert not M._schedulable(enc, base, 0.1)
    del v, views
    assert M._schedulable(enc, base, 0.1)


@pytest.mark.parametrize("form", ["bf16", "fp32", "gelu"])
def test_captured_norm_backward_keeps_its_own_scratch(form):
    """A larger eager backward between capture and replay, with its memory handed on to other tensors."""
    dtype = torch.float32 if form == "fp32" else torch.bfloat16
    g, b = torch.randn(768, device=DEV).to(dtype), torch.randn(768, device=DEV).to(dtype)

    def inputs(rows):
        return torch.randn(rows, 768, device=DEV).to(dtype), torch.randn(rows, 768, device=DEV).to(dtype)

    def backward(x, dy, dg, db):
        if form == "gelu":
            _, mean, rstd = N.norm_gelu_forward(x, g, b, 1e-5)
            return N.norm_gelu_backward(dy, x, g, b, mean, rstd, dg, db)
        _, _, mean, rstd = N.norm_forward(x, g, b, 1e-5, False)
        return N.norm_backward(dy, x, g, mean, rstd, False, dg, db, False)
    x, dy = inputs(64)
    dg, db, want_g, want_b = (torch.zeros(768, device=DEV) for _ in range(4))
    want = backward(x, dy, want_g, want_b).clone()
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        dx = backward(x, dy, dg, db)
    backward(*inputs(20000), torch.zeros_like(dg), torch.zeros_like(db))
    other = [torch.full((1 << 18,), 3.0, device=DEV) for _ in range(16)]
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(dx, want) and torch.equal(dg, want_g) and torch.equal(db, want_b)
    assert all(bool((t == 3.0).all()) for t in other)


def test_tensor_lists_of_very_different_sizes():
    """Blocks by size: one tensor that fills the chip between small ones, and the last element of each found."""
    from spiraltorch_b200.ops import multi
    sizes = [3, 40_000_003, 1, 1025, 1_300_000]
    ts = [torch.randn(n, device=DEV) for n in sizes]
    out, bad = multi.divided(ts, 3.0)
    assert bad is None and all(torch.equal(o[-2000:].cpu(), t[-2000:].cpu() / 3.0) for o, t in zip(out, ts))
    values = [torch.randn(n, device=DEV) for n in sizes]
    want = [v - 0.25 * t for v, t in zip(values, ts)]
    assert multi.descend_(values, ts, 0.25) and all(torch.equal(v, w) for v, w in zip(values, want))
    for k in (4, 3, 2, 1, 0):
        ts[k][-1] = float("nan")
        assert multi.first_nonfinite(ts) == k and multi.divided(ts, 2.0)[1] == k


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("B,S,H,D", [(1, 128, 16, 128), (1, 777, 16, 64), (2, 777, 16, 64), (1, 300, 98, 64), (1, 896, 40, 64), (1, 129, 74, 128), (1, 129, 75, 128)])
def test_attention_in_pairs_and_single_tiles(B, S, H, D, causal):
    """On both sides of the rule between the two kernels: one tile per head, one round of either, two rounds, one round more in
    single tiles.  P is bf16: 2^-8 of the largest value."""
    torch.manual_seed(S + H)
    q, k, v = (torch.randn(B, S, H, D, device=DEV).bfloat16() for _ in range(3))
    o, lse = A.attention_forward(q, k, v, causal)
    ro, rlse = A.attention_reference(q, k, v, causal, 1 / math.sqrt(D))
    assert (o.float() - ro).abs().max() <= 2e-2 * ro.abs().max() and (lse - rlse).abs().max() < 1e-2


@pytest.mark.parametrize("rows,cols", [(1, 64), (128, 72), (129, 8), (129, 9472), (513, 9480), (700, 136), (1030, 64), (1030, 72), (2000, 128), (300, 136), (1000, 37888)])
def test_column_sums_on_both_sides_of_their_rules(rows, cols):
    """Lanes and widths of both forms, columns and rows that fill none of them; fp32 sums of terms of order one."""
    from spiraltorch_b200.ops import elementwise as E
    x = torch.randn(rows, cols, device=DEV).bfloat16()
    want = x.double().sum(0)
    acc = torch.full((cols,), 2.0, device=DEV)
    assert torch.allclose(E.colsum(x).double(), want, rtol=1e-5, atol=1e-4)
    assert torch.allclose(E.colsum(x, acc, accumulate=True).double(), want + 2.0, rtol=1e-5, atol=1e-4)


@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("rows,d", [(592, 264), (593, 512), (1184, 520), (1185, 1024), (1, 1024), (296, 64), (297, 768), (888, 72), (889, 72), (1, 8)])
def test_norm_on_both_sides_of_its_rules(rows, d, rms):
    """Forward by a block or a warp per row, backward by a block per row, in steps of two rows, and with two steps per CTA."""
    torch.manual_seed(rows + d)
    x, dy = (torch.randn(rows, d, device=DEV).bfloat16() for _ in range(2))
    g, b = torch.randn(d, device=DEV).bfloat16(), (None if rms else torch.randn(d, device=DEV).bfloat16())
    y, _, mean, rstd = N.norm_forward(x, g, b, 1e-5, rms)
    xd = x.double()
    mu = 0 if rms else xd.mean(-1, keepdim=True)
    rs = torch.rsqrt((xd - mu).pow(2).mean(-1, keepdim=True) + 1e-5)
    xh = (xd - mu) * rs
    want = xh * g.double() + (0 if rms else b.double())
    assert ((y.double() - want).abs() <= 2 ** -8 * want.abs() + 1e-5).all()
    dg, db = torch.full((d,), 0.5, device=DEV), (None if rms else torch.full((d,), 0.25, device=DEV))
    dx = N.norm_backward(dy, x, g, mean, rstd, rms, dg, db, True)
    gy = dy.double() * g.double()
    want = rs * (gy - (0 if rms else gy.mean(-1, keepdim=True)) - xh * (gy * xh).mean(-1, keepdim=True))
    assert ((dx.double() - want).abs() <= 2 ** -8 * want.abs() + 2e-5).all()
    assert torch.allclose(dg.double(), 0.5 + (dy.double() * xh).sum(0), rtol=1e-5, atol=1e-3)
    assert rms or torch.allclose(db.double(), 0.25 + dy.double().sum(0), rtol=1e-5, atol=1e-3)


def test_contrastive_step_leaves_tangents_transforms_and_modes_to_the_autograd_form():
    import torch.autograd.forward_ad as fwAD
    from torch.utils._python_dispatch import TorchDispatchMode
    from spiraltorch_b200.models import contrastive as M
    enc = M.ContrastiveEncoder(64, 128, 64, device=DEV, seed=1)
    base = torch.randn(48, 64, device=DEV)

    class Count(TorchDispatchMode):
        ops = 0

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            Count.ops += 1
            return func(*args, **(kwargs or {}))
    with Count():
        assert not M._schedulable(enc, base, 0.1)
    with fwAD.dual_level():
        assert not M._schedulable(enc, base, 0.1)
        with pytest.raises(RuntimeError):
            M.contrastive_step(enc, fwAD.make_dual(base, torch.ones_like(base)), 0.1, seed=5)
    assert M._schedulable(enc, base, 0.1)


def test_losses_and_updates_keep_what_belongs_to_their_tensors():
    """Forward-mode tangents and gradients with a graph go through PyTorch's operators."""
    import torch.autograd.forward_ad as fwAD
    p, t = torch.randn(16, 8, device=DEV), torch.randn(16, 8, device=DEV)
    loss, target = st.nn.MeanSquaredError(), st.Tensor._wrap(t)
    with fwAD.dual_level():
        value = loss.forward(st.Tensor._wrap(fwAD.make_dual(p, torch.ones_like(p))), target).torch()
        tangent = fwAD.unpack_dual(value).tangent
        assert torch.allclose(tangent, (2 * (p - t)).mean())
    lin = st.nn.Linear("fc", 8, 8)
    lin.init_normal(0.1, seed=1)
    lin.to(DEV)
    rate = torch.ones((), device=DEV, requires_grad=True)
    lin.weight.gradient = rate * torch.ones_like(lin.weight.value)
    lin.apply_step(0.5)
    assert torch.autograd.grad(lin.weight.value.sum(), rate)[0].item() == -32.0
