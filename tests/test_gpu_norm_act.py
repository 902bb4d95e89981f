"""The fused GroupNorm + GELU kernels against the tensor operations in 64 bits, at the edges of their rules."""
import pytest
import torch
import torch.nn.functional as F

from xadvcool_b200 import surrogate as S

pytestmark = pytest.mark.gpu

SHAPES = [  # N, D, H, W, C, groups
    (1, 1, 1, 1, 8, 2),         # one voxel, one octet, groups of half an octet
    (2, 1, 3, 5, 16, 4),        # fewer voxels than a block takes in one pass
    (3, 4, 17, 19, 32, 8),
    (1, 5, 31, 33, 64, 1),      # all channels one group
    (9, 2, 9, 7, 128, 8),       # more samples than the warps of the gradient's last sum
    (2, 3, 5, 11, 256, 8),      # the widest
    (1, 20, 128, 152, 16, 4),   # several voxels a thread
]


def _ref(y, g, s, G):
    N, C = y.shape[0], y.shape[-1]
    h = y.reshape(N, -1, G, C // G)
    h = (h - h.mean(dim=(1, 3), keepdim=True)) * torch.rsqrt(h.var(dim=(1, 3), unbiased=False, keepdim=True) + S.EPS)
    return F.gelu(h.reshape(y.shape) * g + s)


@pytest.mark.parametrize("shape", SHAPES)
def test_norm_act(cuda, shape):
    *dims, G = shape
    C = dims[-1]
    gen = torch.Generator().manual_seed(3)
    y = (5.0 + 2.0 * torch.randn(dims, generator=gen)).cuda().to(S.BF16).requires_grad_()
    g = (1.0 + 0.3 * torch.randn(C, generator=gen)).cuda().requires_grad_()
    s = (0.3 * torch.randn(C, generator=gen)).cuda().requires_grad_()
    d = torch.randn(dims, generator=gen).cuda().to(S.BF16)
    assert S._norm_act_takes(y, g, s, G)
    out = S._NormAct.apply(y, g, s, G)
    dy, dg, ds = torch.autograd.grad(out, (y, g, s), d)
    assert torch.equal(out, S.norm_gelu(y, g, s, G))  # the tensor operations' bits
    y64, g64, s64 = (t.detach().double().requires_grad_() for t in (y, g, s))
    ref = _ref(y64, g64, s64, G)
    ry, rg, rs = torch.autograd.grad(ref, (y64, g64, s64), d.double())
    # BF16 results: half a unit in the last place (2^-9 relative), and FP32's rounding of values of order one (h carries
    # mean / std = 2.5 times 2^-24, a few operations each) as the absolute part
    for a, r in ((out, ref), (dy, ry)):
        assert ((a.double() - r).abs() <= r.abs() * 2.0 ** -8 + 1e-5 * max(1.0, r.abs().max().item())).all()
    # FP32 sums over n terms of magnitude about 1 carried in FP64 after 8: the terms' own FP32 error
    n = out.numel() // C
    assert (dg.double() - rg).abs().max().item() <= 1e-5 * n ** 0.5 * 8
    assert (ds.double() - rs).abs().max().item() <= 1e-5 * n ** 0.5 * 8


def test_norm_act_groups_are_apart_and_layouts(cuda):
    """A group's infinity stays in that group; transposed and offset operands give the plain call's bits; a graph of the
    gradient is still to be had."""
    gen = torch.Generator().manual_seed(4)
    y = torch.randn((2, 3, 4, 5, 16), generator=gen).cuda().to(S.BF16)
    g, s = torch.ones(16).cuda(), torch.zeros(16).cuda()
    out = S._NormAct.apply(y, g, s, 4)
    bad = y.clone()
    bad[0, 0, 0, 0, 0] = float("inf")
    o = S._NormAct.apply(bad, g, s, 4)
    assert torch.equal(o[..., 4:], out[..., 4:]) and torch.equal(o[1], out[1]) and o[0, ..., :4].isnan().all()
    assert torch.equal(S._NormAct.apply(y.transpose(1, 2).contiguous().transpose(1, 2), g, s, 4), out)
    flat = torch.empty(y.numel() + 1, dtype=S.BF16, device="cuda")
    flat[1:] = y.reshape(-1)
    assert torch.equal(S._NormAct.apply(flat[1:].view(y.shape), g, s, 4), out)
    y64 = y.requires_grad_()
    dy, = torch.autograd.grad(S._NormAct.apply(y64, g, s, 4).float().pow(2).sum(), y64, create_graph=True)
    r, = torch.autograd.grad(S.norm_gelu(y64, g, s, 4).float().pow(2).sum(), y64, create_graph=True)
    a, b = (torch.autograd.grad(t.float().pow(2).sum(), y64)[0] for t in (dy, r))
    assert torch.allclose(a.float(), b.float(), rtol=0.05, atol=0.05 * b.abs().max().item())
