"""Components, grids and beams are read at every call: nothing that follows from
their fields is kept on them, whatever way a field is set or computed (CPU only)."""
import copy
import dataclasses

import numpy as np
import pytest
import torch

import temgymcore_gb300 as t
from temgymcore_gb300.gaussian import pixel_map
from temgymcore_gb300.run import pack_model
from temgymcore_gb300.scan import pack_scan_model


def _focal(lens, pack):
    _, arr = pack([lens])
    return arr[0].p[0]


class _Computed(t.Lens):
    """A plain subclass (it inherits the frozen dataclass) that computes its setting."""
    setting = 0.2

    def _params(self):
        return [type(self).setting]


@pytest.mark.parametrize("pack", [pack_model, pack_scan_model])
def test_a_setting_that_moves_is_packed_at_every_call(pack):
    lens = _Computed(z=0.5, focal_length=1.0)
    for v in (0.2, 0.3, 0.4, 0.5):
        _Computed.setting = v
        assert _focal(lens, pack) == v


@pytest.mark.parametrize("pack", [pack_model, pack_scan_model])
def test_a_frozen_field_that_is_set_all_the_same_is_packed(pack):
    lens = t.Lens(z=0.5, focal_length=0.2)
    for v in (0.2, 0.2, 0.3, 0.4):
        object.__setattr__(lens, "focal_length", v)
        assert _focal(lens, pack) == v
    other = copy.copy(lens)
    object.__setattr__(other, "focal_length", 0.6)
    assert _focal(other, pack) == 0.6 and _focal(lens, pack) == 0.4


def test_packing_leaves_nothing_on_a_component():
    det = t.Detector(z=1.0, pixel_size=(1e-5, 2e-5), shape=(8, 9))
    lens = t.Lens(z=0.5, focal_length=0.2)
    for _ in range(3):
        pack_model([lens, det])
    names = {f.name for c in (lens, det) for f in dataclasses.fields(c)}
    assert set(lens.__dict__) <= names and set(det.__dict__) <= names


def test_the_pixel_map_follows_the_grid():
    det = t.Detector(z=1.0, pixel_size=(1e-5, 2e-5), shape=(8, 9))
    pixel_map(det)
    for grid in (det, copy.copy(det)):
        object.__setattr__(grid, "pixel_size", (3e-5, 4e-5))
        assert list(pixel_map(grid).t) == list(pixel_map(dataclasses.replace(grid)).t)
    assert set(det.__dict__) <= {f.name for f in dataclasses.fields(det)}


def test_the_number_of_beams_follows_the_fields():
    def beams(n):
        return {k: torch.zeros(n, dtype=torch.float64) for k in ("x", "y", "dx", "dy", "pathlength")}

    b = t.GaussianRay(z=0.0, amplitude=1.0, waist_xy=np.ones((1, 2)), radii_of_curv=np.ones((1, 2)),
                      wavelength=1e-9, theta=0.0, **beams(5))
    assert b.size == 5
    for r in (copy.copy(b), b):
        for k, v in beams(7).items():
            object.__setattr__(r, k, v)
        assert r.size == 7


@pytest.mark.parametrize("flip", [False, True])
@pytest.mark.parametrize("centre", [(0.0, 0.0), (0, 0), (1e-6, -2e-6), [0.0, 0.0], (np.float64(0.0), 0.0)])
@pytest.mark.parametrize("rotation", [0.0, 0, 30.0, 45, -17.3, 359.9, 1e5, torch.tensor(0.0), np.float32(0.0)])
def test_the_pixel_map_is_the_matrices_product(centre, rotation, flip):
    r = np.random.default_rng(0)
    for shape in ((1, 1), (8, 9), (256, 255), (4096, 3)):
        ps = tuple(float(v) for v in r.uniform(1e-7, 1e-3, 2))
        det = t.Detector(z=1.0, pixel_size=ps, shape=shape, rotation=rotation, centre=centre, flip_y=flip)
        m = det.pixels_to_metres_mat
        assert det._pixel_map() == (m[0, 0], m[0, 1], m[0, 2], m[1, 0], m[1, 1], m[1, 2])


def test_a_grid_with_its_own_map():
    class Shifted(t.Detector):
        @property
        def pixels_to_metres_mat(self):
            return super().pixels_to_metres_mat + 1e-3

    det = Shifted(z=1.0, pixel_size=(1e-5, 1e-5), shape=(8, 9))
    m = det.pixels_to_metres_mat
    assert det._pixel_map() == (m[0, 0], m[0, 1], m[0, 2], m[1, 0], m[1, 1], m[1, 2])
