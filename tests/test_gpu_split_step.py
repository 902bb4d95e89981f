"""The split step (fluid and thermal lattices in kernels of their own, the fluid a step ahead) at the edges of its cell list,
its row lengths and its pipeline: the oracle's bits in FP32, the staged step's bits in 16-bit storage."""
import numpy as np
import pytest

from oracle.ref import Ref
from xadvcool_b200 import designs
from xadvcool_b200.lattice import Lattice

pytestmark = pytest.mark.gpu


def _mask(kind, nx, ny, nz):
    rng = np.random.default_rng(7)
    if kind == "solid":  # no fluid block at all
        return np.ones((nx, ny, nz), np.int32)
    if kind == "fluid":  # full warps, no inlet or outlet
        return np.zeros((nx, ny, nz), np.int32)
    if kind == "ends":  # inlet and outlet cells only, anywhere
        m = rng.integers(1, 4, (nx, ny, nz)).astype(np.int32)
        return m
    m = rng.integers(0, 2, (nx, ny, nz)).astype(np.int32)
    m[0, 1:-1, 1:-1], m[-1, 1:-1, 1:-1] = 2, 3
    return m


CASES = [("solid", 9, 4, 3), ("fluid", 32, 4, 2), ("ends", 11, 5, 4), ("mixed", 33, 5, 3), ("mixed", 64, 3, 3),
         ("mixed", 270, 3, 3), ("mixed", 320, 3, 3), ("mixed", 325, 4, 3)]


@pytest.mark.parametrize("case", CASES, ids=lambda c: f"{c[0]}{c[1]}")
@pytest.mark.parametrize("block", [64, 256])
def test_split_step_matches_oracle(case, block, cuda):
    kind, nx, ny, nz = case
    mask = _mask(kind, nx, ny, nz)
    heat = np.random.default_rng(8).random(mask.shape).astype(np.float32)
    kw = dict(tau_fluid=0.6, heat_power=0.01, u_inlet_val=0.02, heat_source=heat)
    lat = Lattice(mask, **kw)
    lat.tune(block, 0)
    done = 0
    for n in (1, 2, 8, 8, 3, 9, 8):  # single steps, direct launches, a length's first call and its graph, both parities
        lat.step(n)
        done += n
    got = [t.cpu().numpy() for t in lat.fields()]
    lat.close()
    ref = Ref(32).run_simulation(mask, max_steps=done, stats_every=10 ** 6, **kw)
    for g, k in zip(got, ("rho", "u", "T")):
        assert np.array_equal(g, ref[k]), k


@pytest.mark.parametrize("precision", ["fp16", "bf16", "fp32_t16"])
@pytest.mark.parametrize("nx", [30, 100, 270])
def test_split_step_matches_staged_step(precision, nx, cuda):
    mask, heat, _, _ = designs.gyroid_design(2, nx=nx, ny=11, nz=9, buf=3)
    out = []
    for variant in (0, 1):
        lat = Lattice(mask, tau_fluid=0.56, heat_power=0.05, u_inlet_val=0.02, heat_source=heat, precision=precision)
        lat.tune(64, variant)
        lat.step(13)
        lat.step(13)
        out.append([t.cpu().numpy() for t in lat.fields()])
        lat.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
