"""The fused GroupNorm + GELU keeps the tensor operations' bits in the gradient of the volume too."""
import pytest
import torch

from xadvcool_b200 import surrogate as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,groups", [((2, 1, 3, 5, 16), 4), ((4, 4, 16, 19, 128), 8), ((2, 8, 32, 38, 64), 8),
                                          ((1, 32, 128, 152, 16), 4)])
def test_volume_gradient_bits(shape, groups, cuda):
    gen = torch.Generator().manual_seed(3)
    y = (5.0 + 2.0 * torch.randn(shape, generator=gen)).cuda().to(S.BF16).requires_grad_()
    g = (1.0 + 0.3 * torch.randn(shape[-1], generator=gen)).cuda()
    s = (0.3 * torch.randn(shape[-1], generator=gen)).cuda()
    d = torch.randn(shape, generator=gen).cuda().to(S.BF16)
    fused, = torch.autograd.grad(S._NormAct.apply(y, g, s, groups), y, d)
    tensor, = torch.autograd.grad(S.norm_gelu(y, g, s, groups), y, d)
    assert torch.equal(fused, tensor)
