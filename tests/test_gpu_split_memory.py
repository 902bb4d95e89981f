"""The split step's own memory is made on its first use: on a design of a batch stepped by itself, and inside a capture."""
import numpy as np
import pytest
import torch

from xadvcool_b200 import _capi, designs
from xadvcool_b200.batch import Batch
from xadvcool_b200.lattice import Lattice

pytestmark = pytest.mark.gpu

SPLIT = 1
KW = dict(tau_fluid=0.6, heat_power=1e-4, u_inlet_val=0.05, Pr=2.0, k_ratio=100.0)


def _fields(lat):
    return [t.cpu().numpy() for t in lat.fields()]


@pytest.mark.parametrize("precision", ["fp32", "fp16"])
def test_batch_design_stepped_by_itself(precision, cuda):
    mask = designs.straight_fin_plate()
    with Lattice(mask, precision=precision, **KW) as ref:
        ref.step(120)
        want = _fields(ref)
    b = Batch([dict(mask=mask, **KW)], precision=precision)
    b.run(max_steps=100, stats_every=100, tol_ke=0.0, tol_T=0.0)
    lat = b.lattice(0)
    _capi.call("xac_test_step_form", lat._h, SPLIT)
    lat.step(20)
    got = _fields(lat)
    b.close()
    for a, c in zip(got, want):
        assert np.array_equal(a, c)


def test_first_split_step_inside_a_capture(cuda):
    mask = designs.straight_fin_plate()
    with Lattice(mask, **KW) as lat, Lattice(mask, **KW) as ref:
        lat.step(1)
        lat.stats()
        _capi.call("xac_test_step_form", lat._h, SPLIT)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            lat.step(10)
        g.replay()
        ref.step(11)
        for a, c in zip(_fields(lat), _fields(ref)):
            assert np.array_equal(a, c)
