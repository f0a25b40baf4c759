"""Implicit-GEMM 3x3 convolution, pooling and the conv classifier."""
import pytest
import torch
import torch.nn.functional as F

from spiraltorch_b200.models.conv_classifier import ConvClassifier
from spiraltorch_b200.ops import conv as C


def _rel(a, b):
    return ((a.float() - b.float()).abs().max() / b.float().abs().max().clamp(min=1e-6)).item()


def test_weight_layout_conversions():
    w = torch.arange(2 * 3 * 9, dtype=torch.float32).reshape(2, 27)
    tap = C.to_tap_major(w, 3)
    assert torch.equal(C.from_tap_major(tap, 3), w)
    assert tap[0, 0 * 3 + 1] == w[0, 1 * 9 + 0]            # [tap][ic] <- [ic][tap]
    x = torch.randn(2, 5, 5, 3)
    y = C.conv3x3(x, tap, None)
    ref = F.conv2d(x.permute(0, 3, 1, 2), w.reshape(2, 3, 3, 3), padding=1).permute(0, 2, 3, 1)
    assert torch.allclose(y, ref, atol=1e-5)
    dy = torch.randn(2, 5, 5, 2)
    xg = x.clone().requires_grad_(True)
    F.conv2d(xg.permute(0, 3, 1, 2), w.reshape(2, 3, 3, 3), padding=1).permute(0, 2, 3, 1).backward(dy)
    dx = C.conv3x3(dy, C.dgrad_weights(tap, 3), None)
    assert torch.allclose(dx, xg.grad, atol=1e-5)


def test_classifier_backward_matches_autograd_cpu():
    torch.manual_seed(0)
    model = ConvClassifier(num_classes=10, image=16, device="cpu", dtype=torch.float32)
    imgs, labels = torch.randn(4, 3, 16, 16), torch.randint(0, 10, (4,))
    loss = model.forward_backward(imgs, labels)
    P = {k: v.detach().clone().requires_grad_(True) for k, v in model.p.items()}
    x = imgs
    for s in range(4):
        for i in range(2):
            w = P[f"conv{s}_{i}.weight"]
            ic = w.shape[1] // 9
            w4 = w.reshape(w.shape[0], 3, 3, ic).permute(0, 3, 1, 2)
            x = torch.relu(F.conv2d(x, w4, P[f"conv{s}_{i}.bias"], padding=1))
        x = F.max_pool2d(x, 2)
    logits = x.mean((2, 3)) @ P["head.weight"].t() + P["head.bias"]
    ref = F.cross_entropy(logits[:, :10], labels)
    ref.backward()
    assert abs(loss.item() - ref.item()) < 1e-4
    for name, p in model.p.items():
        g, r = p.main_grad, P[name].grad
        assert torch.allclose(g, r, atol=1e-4, rtol=1e-3), (name, (g - r).abs().max().item())
    assert model(imgs).shape == (4, 10)
    names = [n for n, _ in model.reference_state_dict()]
    assert "conv0_0::weight" in names and dict(model.reference_state_dict())["head::weight"].shape() == (512, 10)


@pytest.mark.gpu
@pytest.mark.parametrize("N,H,Cin,OC", [(4, 64, 64, 64), (8, 32, 64, 128), (8, 16, 128, 256), (16, 8, 256, 512), (2, 32, 3, 64)])
def test_conv_kernels_match_reference(N, H, Cin, OC):
    torch.manual_seed(1)
    x = torch.randn(N, H, H, Cin, device="cuda").bfloat16()
    w = (torch.randn(OC, 9 * Cin, device="cuda") * (2.0 / (9 * Cin)) ** 0.5).bfloat16()
    b = torch.randn(OC, device="cuda").bfloat16()
    y = C.conv3x3(x, w, b, relu=True)
    ref = C._conv_ref(x.cpu().float(), w.cpu().float(), b.cpu().float(), 1, None)
    assert _rel(y.cpu(), ref) < 2e-2
    dy = torch.randn(N, H, H, OC, device="cuda").bfloat16()
    dw = torch.full((OC, 9 * Cin), 0.25, device="cuda")
    C.conv3x3_wgrad(dy, x, dw)
    rdw = torch.full((OC, 9 * Cin), 0.25)
    C.conv3x3_wgrad(dy.cpu().float(), x.cpu().float(), rdw)
    assert _rel(dw.cpu(), rdw) < 2e-2
    if Cin % 64 == 0:
        dx = C.conv3x3(dy, C.dgrad_weights(w, Cin), relu_mask_of=x)
        rdx = C._conv_ref(dy.cpu().float(), C.dgrad_weights(w.cpu().float(), Cin), None, 4, x.cpu().float())
        assert _rel(dx.cpu(), rdx) < 2e-2
    p, idx = C.maxpool2(y)
    rp, ridx = C.maxpool2(y.cpu().float())
    assert torch.equal(p.cpu().float(), rp)
    g = torch.randn_like(p)
    assert torch.equal(C.maxpool2_backward(g, idx, H, H).cpu().float(), C.maxpool2_backward(g.cpu().float(), idx.cpu(), H, H))
    assert _rel(C.global_avgpool(p).cpu(), C.global_avgpool(p.cpu().float())) < 1e-2
    from spiraltorch_b200.ops import native
    torch.cuda.synchronize()
    assert native.read_error_word()[0] == 0


@pytest.mark.gpu
def test_classifier_cuda_tracks_cpu():
    torch.manual_seed(2)
    gpu = ConvClassifier(num_classes=100, image=64, device="cuda")
    cpu = ConvClassifier(num_classes=100, image=64, device="cpu", dtype=torch.float32)
    cpu.flat_w.copy_(gpu.flat_w.float().cpu())
    imgs, labels = torch.randn(8, 3, 64, 64), torch.randint(0, 100, (8,))
    lg = gpu.forward_backward(imgs.cuda(), labels.cuda())
    lc = cpu.forward_backward(imgs, labels)
    assert abs(lg.item() - lc.item()) < 5e-2
    cos = torch.nn.functional.cosine_similarity(gpu.flat_grad.cpu(), cpu.flat_grad, dim=0).item()
    assert cos > 0.98, cos


@pytest.mark.gpu
@pytest.mark.parametrize("N,H,W,Cin,OC", [(2, 6, 10, 3, 64), (1, 4, 4, 5, 72), (3, 12, 6, 8, 40), (2, 24, 24, 64, 64), (2, 64, 64, 64, 8), (64, 16, 16, 64, 256), (130, 32, 32, 64, 264)])
def test_conv_steps_off_the_main_sizes(N, H, W, Cin, OC):
    """Column matrices with odd and vectorised channel counts, output tiles 64 columns wide, the data gradient's weights,
    and the fused pool / ReLU / bias backward."""
    torch.manual_seed(N * H + OC)
    x = torch.randn(N, H, W, Cin, device="cuda").bfloat16()
    w = (torch.randn(OC, 9 * Cin, device="cuda") * (2.0 / (9 * Cin)) ** 0.5).bfloat16()
    wt = C.dgrad_weights(w, Cin)
    assert torch.equal(wt.cpu(), C.dgrad_weights(w.cpu(), Cin))
    y = C.conv3x3(x, w, None, relu=True)
    assert _rel(y.cpu(), C._conv_ref(x.cpu().float(), w.cpu().float(), None, 1, None)) < 2e-2      # bf16 output: 2^-8
    dy = torch.randn(N, H, W, OC, device="cuda").bfloat16()
    dw, rdw = torch.zeros(OC, 9 * Cin, device="cuda"), torch.zeros(OC, 9 * Cin)
    C.conv3x3_wgrad(dy, x, dw)
    C.conv3x3_wgrad(dy.cpu().float(), x.cpu().float(), rdw)
    assert _rel(dw.cpu(), rdw) < 1e-4                                                               # fp32 sums
    pooled, idx = C.maxpool2(y)
    g = torch.randn_like(pooled)
    db, rdb = torch.full((OC,), 0.5, device="cuda"), torch.full((OC,), 0.5)
    dx = C.maxpool2_relu_backward(g, idx, pooled, H, W, db)
    ref = C.maxpool2_relu_backward(g.cpu().float(), idx.cpu(), pooled.cpu().float(), H, W, rdb)
    assert torch.equal(dx.cpu().float(), ref) and torch.allclose(db.cpu(), rdb, rtol=1e-4, atol=1e-4)
    masked = torch.where(y > 0, C.maxpool2_backward(g, idx, H, W), torch.zeros_like(y))
    assert torch.equal(dx, masked)


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K,accumulate", [(64, 32, 65536, False), (72, 40, 1536, True), (128, 64, 1024, False), (8, 200, 3 * 521, True),
                                              (200, 72, 4096, True)])
def test_weight_gradient_in_parts(M, N, K, accumulate):
    """Few output tiles over a long sum: the parts' fixed-order sum, odd divisors of K, and boxes outside the matrix."""
    from spiraltorch_b200.ops import gemm as G
    torch.manual_seed(M + N)
    a, b = torch.randn(K, M, device="cuda").bfloat16(), torch.randn(K, N, device="cuda").bfloat16()
    out = torch.full((M, N), 0.5, device="cuda")
    ref = a.double().t() @ b.double() + (0.5 if accumulate else 0.0)
    G.gemm(a, b, a_mn=True, b_mn=True, out=out, accumulate=accumulate)
    assert ((out - ref).norm() / ref.norm()).item() < 1e-5
    again = torch.full((M, N), 0.5, device="cuda")
    G.gemm(a, b, a_mn=True, b_mn=True, out=again, accumulate=accumulate)
    assert torch.equal(out, again)


@pytest.mark.gpu
@pytest.mark.parametrize("rows,cols", [(1, 8), (1000, 64), (257, 104), (3000, 256), (100, 264)])
def test_column_sums_of_narrow_matrices(rows, cols):
    from spiraltorch_b200.ops import elementwise as E
    x = torch.randn(rows, cols, device="cuda").bfloat16()
    assert torch.allclose(E.colsum(x).double(), x.double().sum(0), rtol=1e-5, atol=1e-3)


@pytest.mark.gpu
@pytest.mark.parametrize("N,H,W,Cin,OC", [(1, 8, 8, 64, 64), (3, 16, 16, 64, 72), (5, 32, 32, 128, 200), (7, 16, 16, 128, 320), (2, 8, 64, 320, 136)])
def test_weight_gradient_over_taps_and_channels(monkeypatch, N, H, W, Cin, OC):
    """Columns run over (tap, channel), so tiles of 192 and 256 cross taps and end past the last one, and the pixel splits
    need not be equal; the caller's fixed order takes the narrow tiles."""
    torch.manual_seed(OC + N)
    x, dy = torch.randn(N, H, W, Cin).bfloat16(), torch.randn(N, H, W, OC).bfloat16()
    want = torch.zeros(OC, 9 * Cin, dtype=torch.float64)
    xp = torch.nn.functional.pad(x.double(), (0, 0, 1, 1, 1, 1))
    for tap in range(9):
        shifted = xp[:, tap // 3:tap // 3 + H, tap % 3:tap % 3 + W]
        want[:, tap * Cin:(tap + 1) * Cin] = dy.double().reshape(-1, OC).t() @ shifted.reshape(-1, Cin)
    bound = N * H * W * 2.0 ** -24 * 4 * (N * H * W) ** 0.5          # fp32 sums of about sqrt(pixels), one rounding per term
    for fixed in ("0", "1"):
        monkeypatch.setenv("SPIRAL_DETERMINISTIC_REDUCTION", fixed)
        got = torch.zeros(OC, 9 * Cin, device="cuda")
        C.conv3x3_wgrad(dy.cuda(), x.cuda(), got)
        assert (got.cpu().double() - want).abs().max().item() <= bound


@pytest.mark.gpu
@pytest.mark.parametrize("N,H,W,Cin", [(1, 1, 1, 3), (2, 5, 51, 1), (3, 7, 13, 2), (1, 16, 16, 3), (2, 9, 29, 3), (3, 10, 9, 4)])
def test_column_matrix_of_images(N, H, W, Cin):
    """Pixels that do not fill the last block, borders on every side, channel counts with and without padding: exact copies."""
    x = torch.randn(N, H, W, Cin, device="cuda").bfloat16()
    col = C.im2col(x, 64).float().cpu()
    want = torch.nn.functional.unfold(x.float().cpu().permute(0, 3, 1, 2), 3, padding=1)
    want = want.reshape(N, Cin, 9, H * W).permute(0, 3, 2, 1).reshape(N * H * W, 9 * Cin)
    assert torch.equal(col[:, :9 * Cin], want) and not col[:, 9 * Cin:].any()


@pytest.mark.gpu
@pytest.mark.parametrize("N,H,W,Cin,OC", [(80, 4, 64, 64, 64), (5, 64, 64, 64, 8), (80, 8, 32, 128, 64), (80, 16, 16, 192, 72),
                                          (80, 32, 8, 64, 128), (30, 6, 128, 64, 64), (40, 4, 128, 64, 128), (40, 32, 32, 64, 128)])
def test_conv_with_shared_row_blocks(N, H, W, Cin, OC):
    """Up to 128 output channels over whole tiles of 256 pixels: resident and streamed weights, every width, channels that do
    not fill the tile, one and several tiles per SM, and both epilogues; the seventh does not fit in shared memory."""
    torch.manual_seed(H * W + OC)
    x = torch.randn(N, H, W, Cin).bfloat16()
    w = (torch.randn(OC, 9 * Cin) * (9 * Cin) ** -0.5).bfloat16()
    bias, mask = torch.randn(OC).bfloat16(), torch.randn(N, H, W, OC).bfloat16()
    want = C._conv_ref(x.float(), w.float(), None, 0, None)
    for act, got in (("relu", C.conv3x3(x.cuda(), w.cuda(), bias.cuda(), relu=True)), ("mask", C.conv3x3(x.cuda(), w.cuda(), relu_mask_of=mask.cuda()))):
        ref = torch.relu(want + bias.float()) if act == "relu" else torch.where(mask.float() > 0, want, torch.zeros(()))
        err = (got.float().cpu() - ref).abs()
        assert (err <= 2.0 ** -8 * ref.abs() + 1e-4).all()            # one bf16 rounding, fp32 sums of terms of order one


@pytest.mark.gpu
def test_data_gradient_weights_stay_differentiable():
    w = torch.randn(8, 9 * 16, device="cuda").bfloat16().requires_grad_()
    out = C.dgrad_weights(w, 16)
    g = torch.randn_like(out)
    out.backward(g)
    with torch.no_grad():
        assert torch.equal(C.dgrad_weights(w, 16), out) and torch.equal(C.dgrad_weights(w.grad, 16), g)
