"""The convolutions where a block walks many tiles: planes kept from one z to the next, the rings of planes and weights going
round, accumulator buffers used again, and weight-gradient accumulators added to a partial more than once. The tiles are
those of 148 SMs; each shape states what it is there for and the test checks that it still is."""
import ctypes as C

import pytest
import torch
import torch.nn.functional as F

from xadvcool_b200 import _capi
from xadvcool_b200 import surrogate as S

pytestmark = pytest.mark.gpu


def _plan(shape):
    fwd, wg = (C.c_longlong * 8)(), (C.c_longlong * 7)()
    _capi.call("xac_test_conv_plan", *shape, 148, fwd, wg)
    return (dict(zip("units ctas march planes resident stages buffers blocks".split(), fwd)),
            dict(zip("units ctas march planes per_flush buffers rows".split(), wg)))


FORWARD = [  # N, D, H, W, Ci, Co, ksize; planes kept, weights resident
    ((1, 32, 128, 152, 16, 16, 3), 1, 1),
    ((1, 33, 127, 151, 16, 16, 3), 1, 1),   # odd extents: ragged tiles, z walks that end inside a strip
    ((2, 17, 61, 149, 48, 16, 3), 1, 1),
    ((4, 16, 64, 76, 96, 32, 3), 0, 0),     # weights streamed, eight stages
    ((3, 15, 63, 75, 96, 32, 3), 0, 0),     # three stages
    ((1, 40, 90, 90, 256, 64, 3), 0, 0),
    ((2, 32, 128, 152, 16, 16, 1), 0, 1),
]


@pytest.mark.parametrize("shape,march,resident", FORWARD)
def test_forward_over_many_tiles(cuda, shape, march, resident):
    plan = _plan(shape)[0]
    assert plan["units"] >= 3 * plan["ctas"] and plan["march"] == march and plan["resident"] == resident, plan
    N, D, H, W, Ci, Co, k = shape
    g = torch.Generator("cuda").manual_seed(11)
    x = torch.randn((N, D, H, W, Ci), generator=g, device="cuda").to(S.BF16)
    w = (0.1 * torch.randn((k ** 3, Co, Ci), generator=g, device="cuda")).to(S.BF16)
    b = torch.randn((Co,), generator=g, device="cuda")
    y = S.conv_forward(x, w, b, k, out_fp32=True)
    assert S.kernel_status() == 0
    wt = w.float().view(k, k, k, Co, Ci).permute(3, 4, 0, 1, 2).contiguous()
    ref = F.conv3d(x.float().permute(0, 4, 1, 2, 3), wt, b, padding=k // 2).permute(0, 2, 3, 4, 1)
    # exact BF16 products summed in FP32 in another order, as in the small shapes; a plane, stage or tile out of turn is an
    # error of the size of the outputs
    scale = (x.float().abs().amax() * w.float().abs().sum(dim=(0, 2)).amax()).item()
    assert (y - ref).abs().max().item() <= 1e-5 * scale


WEIGHT = [  # N, D, H, W, Ci, Co, ksize; planes kept, accumulator buffers, d_out by rows
    ((4, 32, 128, 152, 48, 16, 3), 1, 2, 0),  # 14 additions to a partial
    ((2, 24, 100, 150, 32, 48, 3), 1, 1, 0),
    ((2, 24, 100, 300, 32, 48, 3), 0, 1, 1),
    ((2, 20, 60, 60, 128, 256, 3), 1, 1, 1),  # output channels in two blocks
    ((2, 32, 128, 152, 16, 16, 1), 0, 2, 1),
]


@pytest.mark.parametrize("shape,march,buffers,rows", WEIGHT)
def test_weight_grad_over_many_tiles(cuda, shape, march, buffers, rows):
    plan = _plan(shape)[1]
    per_cta = -(-plan["units"] // plan["ctas"])
    assert per_cta > plan["per_flush"] and plan["march"] == march and plan["buffers"] == buffers, plan
    assert plan["rows"] == rows, plan
    N, D, H, W, Ci, Co, k = shape
    g = torch.Generator("cuda").manual_seed(12)
    # one sign: the sum of magnitudes is the sum, so a lost tile (1 / units of it, 2e-4 and more) stands out
    x = torch.rand((N, D, H, W, Ci), generator=g, device="cuda").to(S.BF16)
    dy = torch.rand((N, D, H, W, Co), generator=g, device="cuda").to(S.BF16)
    dw, db = S.conv_weight_grad(x, dy, k, True)
    assert S.kernel_status() == 0
    # 256 additions of an accumulator, each truncated by 2^-23 of its sum at most, then fewer than 50 roundings of 2^-24:
    # 3.4e-5 of the sum; the largest number of tiles here is 4096
    tol = 3.5e-5
    assert 1.0 / plan["units"] > 4 * tol
    xp, d2 = F.pad(x, (0, 0, 1, 1, 1, 1, 1, 1)), dy.double().reshape(-1, Co).T.contiguous()
    for t in range(k ** 3):
        z, r, c = (t // 9, t // 3 % 3, t % 3) if k == 3 else (1, 1, 1)
        ref = d2 @ xp[:, z:z + D, r:r + H, c:c + W].reshape(-1, Ci).double()
        assert ((dw[t] - ref).abs() <= tol * ref).all(), t
    assert ((db - d2.sum(1)).abs() <= 1e-5 * d2.sum(1)).all()
