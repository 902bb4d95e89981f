"""The three forms of the step (one-pass, split, staged) at the edges of their row lengths, cell lists and runs, each forced
on lattices of any size: the oracle's bits in FP32, one another's bits in 16-bit storage."""
import numpy as np
import pytest

from oracle.ref import Ref
from xadvcool_b200 import _capi, designs
from xadvcool_b200.lattice import Lattice

pytestmark = pytest.mark.gpu

ROW, SPLIT, STAGED = 0, 1, 2


def _mask(kind, nx, ny, nz):
    rng = np.random.default_rng(7)
    if kind == "solid":
        return np.ones((nx, ny, nz), np.int32)
    if kind == "fluid":
        return np.zeros((nx, ny, nz), np.int32)
    if kind == "ends":  # inlet and outlet cells only, anywhere
        return rng.integers(1, 4, (nx, ny, nz)).astype(np.int32)
    m = rng.integers(0, 2, (nx, ny, nz)).astype(np.int32)
    m[0, 1:-1, 1:-1], m[-1, 1:-1, 1:-1] = 2, 3
    return m


CASES = [("solid", 9, 4, 3), ("fluid", 32, 4, 2), ("ends", 11, 5, 4), ("mixed", 33, 5, 3), ("mixed", 64, 3, 3),
         ("mixed", 270, 3, 3), ("mixed", 320, 3, 3), ("mixed", 325, 4, 3)]


def _run(lat, form, lengths):
    _capi.call("xac_test_step_form", lat._h, form)
    for n in lengths:
        lat.step(n)
    return [t.cpu().numpy() for t in lat.fields()]


FORMS = [(ROW, 64), (ROW, 256), (SPLIT, 64), (SPLIT, 256), (STAGED, 128)]  # form, block; staged rows end at 320


@pytest.mark.parametrize("case,form,block", [(c, f, b) for c in CASES for f, b in FORMS if f != STAGED or c[1] <= 320])
def test_form_matches_oracle(case, form, block, cuda):
    kind, nx, ny, nz = case
    mask = _mask(kind, nx, ny, nz)
    heat = np.random.default_rng(8).random(mask.shape).astype(np.float32)
    kw = dict(tau_fluid=0.6, heat_power=0.01, u_inlet_val=0.02, heat_source=heat)
    lengths = (1, 2, 8, 8, 3, 9, 8)  # single steps, direct launches, a length's first call and its graph, both parities
    with Lattice(mask, **kw) as lat:
        lat.tune(block, 0)
        got = _run(lat, form, lengths)
    ref = Ref(32).run_simulation(mask, max_steps=sum(lengths), stats_every=10 ** 6, **kw)
    for g, k in zip(got, ("rho", "u", "T")):
        assert np.array_equal(g, ref[k]), k


@pytest.mark.parametrize("precision", ["fp16", "bf16", "fp32_t16"])
@pytest.mark.parametrize("nx", [30, 100, 270, 310, 330])  # compile-time rows, rows of the split and staged steps only, runtime
def test_forms_agree(precision, nx, cuda):
    mask, heat, _, _ = designs.gyroid_design(2, nx=nx, ny=11, nz=9, buf=3)
    kw = dict(tau_fluid=0.56, heat_power=0.05, u_inlet_val=0.02, heat_source=heat, precision=precision)
    out = []
    for form in (ROW, SPLIT) + ((STAGED,) if nx <= 320 else ()):
        with Lattice(mask, **kw) as lat:
            out.append(_run(lat, form, (13, 13, 5)))
    for other in out[1:]:
        for a, b in zip(out[0], other):
            assert np.array_equal(a, b)


def test_forms_share_a_run(cuda):
    """A run that changes form on the way gives the bits of one that does not."""
    mask = designs.straight_fin_plate()
    kw = dict(tau_fluid=0.6, heat_power=1e-4, u_inlet_val=0.05, Pr=2.0, k_ratio=100.0)
    with Lattice(mask, **kw) as lat, Lattice(mask, **kw) as ref:
        for form, n in ((SPLIT, 9), (ROW, 3), (STAGED, 10), (SPLIT, 2), (-1, 16)):
            got = _run(lat, form, (n,))
        want = _run(ref, ROW, (40,))
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
