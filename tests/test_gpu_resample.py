"""The surrogate's resampling kernels against the tensor operations they replace, bit for bit where sums are exact."""
import pytest
import torch

from xadvcool_b200 import surrogate as S

pytestmark = pytest.mark.gpu

SHAPES = [  # coarse N, D, H, W, channels of the coarse and of the skip volume
    (1, 1, 1, 1, 8, 8),
    (2, 3, 5, 7, 16, 24),
    (3, 2, 33, 19, 128, 64),
    (1, 16, 64, 76, 32, 16),
]


def _exact(shape, gen):
    """BF16 values on a grid of 1/16: sums of eight are exact in FP32 in any order"""
    return (torch.randint(-64, 65, shape, generator=gen).float() / 16).cuda().to(S.BF16)


@pytest.mark.parametrize("shape", SHAPES)
def test_resample(cuda, shape):
    N, D, H, W, Ca, Cb = shape
    gen = torch.Generator().manual_seed(6)
    fine = (N, 2 * D, 2 * H, 2 * W)
    low, skip = _exact((N, D, H, W, Ca), gen).requires_grad_(), _exact(fine + (Cb,), gen).requires_grad_()
    d, dp = _exact(fine + (Ca + Cb,), gen), _exact((N, D, H, W, Cb), gen)
    res = []
    for conv in (S.conv3d, None):
        cat, pool = S.Surrogate._up_cat(low, skip, conv), S.Surrogate._pool(skip, conv)
        res.append((cat, pool, *torch.autograd.grad((cat, pool), (low, skip), (d, dp))))
    for a, b in zip(*res):
        assert torch.equal(a, b)


def test_resample_layouts(cuda):
    """Strided and offset operands, and gradients through a graph of the gradient."""
    gen = torch.Generator().manual_seed(7)
    low, skip = _exact((2, 3, 2, 4, 16), gen), _exact((2, 6, 4, 8, 8), gen)
    ref = S.Surrogate._up_cat(low, skip)
    flat = torch.empty(low.numel() + 1, dtype=S.BF16, device="cuda")
    flat[1:] = low.reshape(-1)
    assert torch.equal(S._UpCat2.apply(flat[1:].view(low.shape), skip.transpose(2, 3).contiguous().transpose(2, 3)), ref)
    with pytest.raises(RuntimeError):  # odd extents are refused, as before
        S.Surrogate._pool(skip[:, :5].contiguous(), S.conv3d)
    x = low.requires_grad_()
    for f, g in ((lambda t: S._UpCat2.apply(t, skip), lambda t: S.Surrogate._up_cat(t, skip)),):
        r = []
        for fn in (f, g):
            dx, = torch.autograd.grad(fn(x).float().pow(2).sum(), x, create_graph=True)
            r.append(torch.autograd.grad(dx.float().sum(), x)[0])
        assert torch.equal(*r)
