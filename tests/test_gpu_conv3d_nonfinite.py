"""Weight gradients of operands with infinities and NaN: a tap that does not use the voxel stays finite."""
import pytest
import torch
import torch.nn.functional as F

from xadvcool_b200 import surrogate as S

pytestmark = pytest.mark.gpu

INF, NAN = float("inf"), float("nan")
CASES = [  # shape (N, D, H, W, Ci, Co, ksize), operand, (voxel, channel, value) ...
    ((2, 4, 6, 10, 16, 16, 3), "dy", [((0, 0, 0, 0), 3, INF)]),                # a corner: most taps look outside
    ((1, 3, 9, 300, 32, 48, 3), "dy", [((0, 2, 8, 299), 0, -INF), ((0, 1, 4, 150), 40, NAN)]),  # rows split in tiles
    ((1, 5, 70, 9, 16, 32, 3), "dy", [((0, 2, 35, 8), 1, INF), ((0, 2, 36, 8), 1, -INF)]),
    ((1, 3, 6, 10, 128, 144, 3), "dy", [((0, 1, 0, 5), 130, INF)]),            # the second block of output channels
    ((2, 3, 9, 300, 32, 48, 1), "dy", [((1, 0, 3, 17), 5, INF)]),
    ((2, 4, 6, 10, 16, 16, 3), "x", [((1, 2, 3, 4), 7, INF)]),                 # an inner voxel
    ((1, 3, 9, 300, 32, 48, 3), "x", [((0, 1, 4, 253), 9, -INF), ((0, 1, 4, 254), 9, -INF)]),  # beside a tile's edge
    ((1, 9, 11, 20, 48, 16, 3), "x", [((0, 4, 5, 6), 33, NAN)]),
]


@pytest.mark.parametrize("shape,operand,spots", CASES)
def test_weight_grad_keeps_taps_that_do_not_use_the_voxel(cuda, shape, operand, spots):
    N, D, H, W, Ci, Co, k = shape
    g = torch.Generator().manual_seed(8)
    x = torch.randn((N, D, H, W, Ci), generator=g).to(S.BF16)
    dy = torch.randn((N, D, H, W, Co), generator=g).to(S.BF16)
    big = x.float().abs().amax().item() * dy.float().abs().amax().item()
    for voxel, c, value in spots:
        (dy if operand == "dy" else x)[voxel + (c,)] = value
    dw, db = S.conv_weight_grad(x.cuda(), dy.cuda(), k, True)
    assert S.kernel_status() == 0
    dw, xd, dp = dw.cpu().double(), x.double().reshape(-1, Ci), F.pad(dy.double(), (0, 0, 1, 1, 1, 1, 1, 1))
    tol = 1e-6 * big * N * D * H * W  # as for finite operands: 256 truncating additions an accumulator
    for t in range(k ** 3):
        z, r, c = (2 - t // 9, 2 - t // 3 % 3, 2 - t % 3) if k == 3 else (1, 1, 1)
        ref = dp[:, z:z + D, r:r + H, c:c + W].reshape(-1, Co).T @ xd  # zeros of d_out outside, every input voxel once
        ok = ref.isfinite()
        assert torch.equal(dw[t].isfinite(), ok) and torch.equal(dw[t].isnan(), ref.isnan()), t
        assert torch.equal(dw[t][ref.isinf()], ref[ref.isinf()]), t
        assert (dw[t] - ref)[ok].abs().max().item() <= tol if ok.any() else True, t
    assert torch.equal(db.isfinite().cpu(), dy.float().sum((0, 1, 2, 3)).isfinite())
