"""The convolution kernels at the edges of their tiling rules, against torch on the same BF16 operands."""
import pytest
import torch
import torch.nn.functional as F

from xadvcool_b200 import surrogate as S

pytestmark = pytest.mark.gpu

SHAPES = [  # N, D, H, W, Ci, Co, ksize
    (1, 1, 1, 1, 16, 16, 3),        # one voxel: every other tap is padding
    (1, 2, 3, 300, 256, 32, 3),     # rows wider than a tile, planes that only fit in narrow tiles
    (1, 5, 130, 9, 16, 16, 3),      # column taller than a tile, z walks shorter than the ring
    (3, 7, 13, 43, 48, 16, 3),      # three 16-channel blocks a tap, resident weights
    (1, 6, 20, 21, 96, 32, 3),      # three 32-channel blocks a tap, streamed weights
    (2, 3, 9, 26, 112, 48, 3),      # seven blocks: one a stage
    (1, 9, 17, 38, 64, 192, 3),     # output channels in slices
    (2, 4, 16, 19, 128, 256, 3),
    (1, 2, 33, 257, 16, 32, 1),     # 1x1x1: no halo
    (1, 3, 5, 7, 80, 240, 1),
]


@pytest.mark.parametrize("shape", SHAPES)
def test_forward_tiles(cuda, shape):
    N, D, H, W, Ci, Co, k = shape
    g = torch.Generator().manual_seed(5)
    x = torch.randn((N, D, H, W, Ci), generator=g).cuda().to(S.BF16)
    w = (0.1 * torch.randn((k ** 3, Co, Ci), generator=g)).cuda().to(S.BF16)
    b = torch.randn((Co,), generator=g).cuda()
    y = S.conv_forward(x, w, b, k, out_fp32=True)
    assert S.kernel_status() == 0
    wt = w.float().view(k, k, k, Co, Ci).permute(3, 4, 0, 1, 2).contiguous()
    ref = F.conv3d(x.float().permute(0, 4, 1, 2, 3), wt, b, padding=k // 2).permute(0, 2, 3, 4, 1)
    # exact BF16 products summed in FP32 in another order: 27 * 256 terms at most, each sum within 2^-24 of the
    # sum of magnitudes per addition, which random signs keep far below 1e-5 of the largest possible sum
    scale = (x.float().abs().amax() * w.float().abs().sum(dim=(0, 2)).amax()).item()
    assert (y - ref).abs().max().item() <= 1e-5 * scale
    # the order of the additions does not depend on the tile: a sub-volume gives the same bits away from its cut
    if H > 4:
        part = S.conv_forward(x[:, :, :H - 2].contiguous(), w, b, k, out_fp32=True)
        assert torch.equal(part[:, :, :H - 3], y[:, :, :H - 3])


GRAD_SHAPES = [
    (1, 1, 1, 1, 16, 16, 3),        # one voxel
    (2, 3, 9, 300, 32, 48, 3),      # rows wider than a tile: d_out copied row by row, its halo columns zero
    (1, 2, 5, 300, 32, 48, 1),
    (1, 4, 70, 9, 16, 32, 3),       # three dx taps in M = 128, columns taller than a tile
    (1, 9, 11, 20, 48, 16, 3),      # three dx taps in M = 64, input channels in blocks
    (1, 5, 8, 13, 64, 64, 3),       # two dx taps in M = 128 and one in M = 64
    (1, 3, 6, 10, 128, 144, 3),     # output channels in a block of 128 and one of 16
    (1, 2, 3, 5, 256, 256, 3),
    (2, 12, 21, 19, 80, 96, 1),
]


@pytest.mark.parametrize("shape", GRAD_SHAPES)
def test_weight_grad_tiles(cuda, shape):
    N, D, H, W, Ci, Co, k = shape
    g = torch.Generator().manual_seed(6)
    x = torch.randn((N, D, H, W, Ci), generator=g).cuda().to(S.BF16)
    dy = torch.randn((N, D, H, W, Co), generator=g).cuda().to(S.BF16)
    dw, db = S.conv_weight_grad(x, dy, k, True)
    assert S.kernel_status() == 0
    xp, d2 = F.pad(x.double(), (0, 0, 1, 1, 1, 1, 1, 1)), dy.double().reshape(-1, Co)
    # an accumulator takes at most 256 truncating additions (2^-23 of the running sum each), 3e-5 of the sum of
    # magnitudes at worst; that sum is near 0.64 per voxel against maxima near 4.5 * 4.5
    tol = 1e-6 * x.float().abs().amax().item() * dy.float().abs().amax().item() * N * D * H * W
    for t in range(k ** 3):
        z, r, c = (t // 9, t // 3 % 3, t % 3) if k == 3 else (1, 1, 1)
        ref = d2.T @ xp[:, z:z + D, r:r + H, c:c + W].reshape(-1, Ci)
        assert (dw[t] - ref).abs().max().item() <= tol, t
    assert (db - d2.sum(0)).abs().max().item() <= 1e-6 * dy.float().abs().amax().item() * N * D * H * W
