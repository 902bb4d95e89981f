"""A staged step's wait that gave up (its status word written by the test hook, as the kernel would) is seen by the next
call that hands results to the caller, whichever it is, and also after the launch variant changed."""
import numpy as np
import pytest
import torch

from xadvcool_b200 import _capi, designs
from xadvcool_b200._tensors import stream_ptr
from xadvcool_b200.lattice import Lattice

pytestmark = pytest.mark.gpu

CALLS = {
    "stats": lambda lat: lat.stats(),
    "fields": lambda lat: lat.fields(),
    "scalars": lambda lat: lat.scalars(buf=8, core_nx=48, core_ny=32),
    "validate": lambda lat: lat.validate_raw(),
    "save_state": lambda lat: lat.save_state(),
    "run": lambda lat: lat.run(max_steps=200),
}


def _lattice():
    lat = Lattice(designs.straight_fin_plate(), tau_fluid=0.6, heat_power=1e-4, u_inlet_val=0.05, Pr=2.0, k_ratio=100.0)
    lat.tune(128, 1)
    lat.step(10)
    return lat


@pytest.mark.parametrize("switch", [False, True])
@pytest.mark.parametrize("name", list(CALLS))
def test_first_call_after_a_lost_copy_reports_it(name, switch, cuda):
    with _lattice() as lat:
        _capi.call("xac_test_set_step_status", lat._h, 1, stream_ptr(torch.device("cuda")))
        if switch:
            lat.tune(64, 0)
            lat.step(3)
        with pytest.raises(_capi.XacError) as e:
            CALLS[name](lat)
        assert e.value.code == _capi.XAC_ETIMEOUT
        with pytest.raises(_capi.XacError) as e:
            lat.step(1)
        assert e.value.code == _capi.XAC_ETIMEOUT
        lat.init_fields()
        lat.step(2)
        assert np.isfinite(lat.stats()).all()


def test_fields_of_staged_steps_under_capture(cuda):
    """Steps and fields that a caller captured: no wait inside the capture; a status set by a replay is seen afterwards."""
    with _lattice() as lat, _lattice() as ref:
        lat.stats()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            lat.step(2)
            out = lat.fields()
        g.replay()
        torch.cuda.synchronize()
        ref.step(2)
        assert all(torch.equal(a, b) for a, b in zip(out, ref.fields()))
        lat.stats()
        g.replay()
        _capi.call("xac_test_set_step_status", lat._h, 1, stream_ptr(torch.device("cuda")))
        with pytest.raises(_capi.XacError):
            lat.fields()
