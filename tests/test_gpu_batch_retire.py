"""A batch whose tiles are strided over the blocks at first and, as designs retire, few enough that a block takes a contiguous
run of them: each design keeps the steps and bits of its own solve through the change."""
import numpy as np
import pytest

from xadvcool_b200 import designs
from xadvcool_b200.batch import Batch
from xadvcool_b200.lattice import Lattice

pytestmark = pytest.mark.gpu

STRIDED_ABOVE = 4 * 148 * 4 * 256  # row positions: four tiles for each resident block


@pytest.mark.parametrize("precision", ["fp32", "fp16"])
def test_retirement_across_the_change_of_tile_order(precision, cuda):
    ds = []
    for k, (nx, ny, nz) in enumerate([(96, 64, 18), (120, 60, 20), (64, 70, 17), (128, 64, 16), (90, 66, 19), (100, 50, 21)]):
        m, h, u, _ = designs.gyroid_design(k, nx=nx, ny=ny, nz=nz, buf=6)
        ds.append(dict(mask=m, heat_source=h, tau_fluid=0.6 + 0.01 * k, u_inlet_val=min(u, 0.03), Pr=2.0, k_ratio=20.0,
                       heat_power=0.02))
    positions = [(d["mask"].shape[0] + 31) // 32 * 32 * d["mask"].shape[1] * d["mask"].shape[2] for d in ds]
    assert sum(positions) > STRIDED_ABOVE > max(positions)
    run = dict(max_steps=3000, stats_every=100, tol_ke=3e-4, tol_T=3e-4, min_steps=200)
    b = Batch(ds, precision=precision)
    res = b.run(**run)
    got = [[t.cpu().numpy() for t in b.lattice(i).fields()] for i in range(len(ds))]
    b.close()
    active = lambda step: sum(p for p, r in zip(positions, res) if r["steps"] > step)
    assert active(100) > STRIDED_ABOVE > active(max(r["steps"] for r in res) - 1) > 0
    for d, r, f in zip(ds, res, got):
        with Lattice(d["mask"], precision=precision, **{k: v for k, v in d.items() if k != "mask"}) as lat:
            ref = lat.run(**run)
            want = [t.cpu().numpy() for t in lat.fields()]
        assert (r["steps"], r["converged"], r["diverged"]) == (ref["steps"], ref["converged"], ref["diverged"])
        for a, c in zip(f, want):
            assert np.array_equal(a, c)
