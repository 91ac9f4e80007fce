"""Component packing: kept only where a component's fields cannot change (CPU only)."""
import ctypes as C
import dataclasses

import numpy as np
import pytest
import torch

import temgymcore_gb300 as t
from temgymcore_gb300 import _native as N
from temgymcore_gb300.run import pack_model


def _table(model):
    m, arr = pack_model(model)
    return [bytes(arr[i]) for i in range(m.n_components)]


@pytest.mark.parametrize("make", [lambda v: torch.tensor(v, dtype=torch.float64), lambda v: np.array(v)])
def test_fields_that_may_change_are_packed_anew(make):
    v = make(0.25)
    lens = t.Lens(z=0.5, focal_length=v)
    before = _table([lens])
    v += 0.25
    assert _table([lens]) == _table([t.Lens(z=0.5, focal_length=0.5)]) != before


def test_plain_components_and_grids_follow_replace():
    det = t.Detector(z=1.0, pixel_size=(1e-5, 2e-5), shape=(8, 9))
    model = [t.Lens(z=0.5, focal_length=0.2), det]
    assert _table(model) == _table(model)
    moved = dataclasses.replace(model[0], focal_length=0.3)
    assert _table([moved]) == _table([t.Lens(z=0.5, focal_length=0.3)])
    assert det._pixel_map() == det._pixel_map()
    wide = dataclasses.replace(det, pixel_size=(3e-5, 2e-5))
    m = wide.pixels_to_metres_mat
    assert wide._pixel_map() == (m[0, 0], m[0, 1], m[0, 2], m[1, 0], m[1, 1], m[1, 2])


def test_descanner_parameter_order():
    """p[]: scan position and tilt, the 4x4 matrix row by row, the offsets."""
    rng = np.random.default_rng(0)
    e = t.DescanError(*rng.normal(size=20))
    d = t.Descanner(z=0.1, scan_pos_x=1.0, scan_pos_y=2.0, scan_tilt_x=3.0, scan_tilt_y=4.0, descan_error=e)
    comp = N.TgComponent.from_buffer_copy(_table([d])[0])
    want = [1.0, 2.0, 3.0, 4.0, *e.as_matrix4().reshape(-1), *e.offsets()]
    assert list(comp.p)[:len(want)] == want and C.sizeof(comp) == len(bytes(comp))
