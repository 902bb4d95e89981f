"""Device bytes of a design in a batch: populations, link words, fields, cell table and reduction rows, nothing of the split
step, which a batch never runs."""
import numpy as np
import pytest

from xadvcool_b200 import designs
from xadvcool_b200.batch import footprint

ELEM = {"fp32": (4, 4), "fp16": (2, 2), "bf16": (2, 2), "fp32_t16": (4, 2)}


@pytest.mark.parametrize("precision", list(ELEM))
def test_footprint_is_what_a_batch_reads(precision):
    mask = designs.gyroid_design(3, nx=148, ny=64, nz=32)[0]
    nx, ny, nz = mask.shape
    n, pitch, nonsolid = mask.size, (nx + 31) // 32 * 32, int((mask != 1).sum())
    p, q = ELEM[precision]
    fluid = 2 * 19 * ((nonsolid + 31) // 32 * 32) * p
    thermal = 2 * (ny * nz + 2 * (ny + 2)) * 19 * pitch * q
    table = (ny * nz + 2 * (ny + 1)) * (pitch // 32) * 8
    rest = footprint(dict(mask=mask), precision) - fluid - thermal - table - 29 * n  # reduction rows: 17 doubles a 1024 cells
    assert 0 < rest <= 8 * 17 * (n // 1024 + 1) + 8 * 40 * 592 + 1024


def test_footprint_does_not_depend_on_the_kind_of_fluid_cell():
    fluid = np.zeros((64, 8, 8), np.int32)
    ends = fluid.copy()
    ends[0], ends[-1] = 2, 3
    assert footprint(dict(mask=fluid)) == footprint(dict(mask=ends))
