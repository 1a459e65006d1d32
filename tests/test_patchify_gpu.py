"""Image patches, all dtype pairs, vector and element paths: copies, so exact."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from dart_pytorch_b200.ops import kernels as K


@pytest.mark.parametrize("B,C,H,W,P", [(2, 3, 32, 48, 16), (3, 1, 8, 8, 8), (1, 3, 24, 12, 4), (2, 2, 16, 32, 8), (1, 4, 9, 6, 3),
                                       (130, 3, 40, 8, 8)])
@pytest.mark.parametrize("src", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("dst", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("offset", [0, 1])
def test_patchify(B, C, H, W, P, src, dst, offset):
    img = torch.randn(B * C * H * W + offset, device="cuda").to(src)[offset:].view(B, C, H, W)
    want = img.view(B, C, H // P, P, W // P, P).permute(0, 2, 4, 3, 5, 1).reshape(B * (H // P) * (W // P), P * P * C).to(dst)
    assert torch.equal(K.patchify(img, P, out_dtype=dst), want)
