"""First convolution of an image network: its column matrix straight from NCHW images and the padded weights of the same launch."""
import pytest
import torch

from spiraltorch_b200.ops import conv as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,H,W", [(1, 1, 1), (3, 5, 7), (2, 64, 64), (7, 33, 18)])
@pytest.mark.parametrize("channels", [1, 2, 3, 4])
def test_stem_columns(N, H, W, channels):
    torch.manual_seed(N + H)
    images = torch.randn(N, channels, H, W, device="cuda").bfloat16()
    weights = torch.randn(40, 9 * channels, device="cuda").bfloat16()
    col, padded = C.stem_columns(images, weights)
    assert torch.equal(col, C.im2col(images.permute(0, 2, 3, 1).contiguous(), 64))
    assert torch.equal(padded[:, : 9 * channels], weights) and not padded[:, 9 * channels:].any()
    assert C.stem_columns(images.permute(0, 1, 3, 2), weights) is None or W == 1 or H == 1


@pytest.mark.parametrize("shape", [(2, 4, 6, 24), (1, 2, 2, 6)])
def test_pool_without_argmax(shape):
    x = torch.randn(shape, device="cuda").bfloat16()
    y, none = C.maxpool2(x, argmax=False)
    assert none is None and torch.equal(y, C.maxpool2(x)[0])
