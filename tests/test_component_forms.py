"""Components of a user's own making: a parameter that is not in the instance's
dictionary, a descan error with its own matrix or of another type (CPU only)."""
import types

import numpy as np
import torch

import temgymcore_gb300 as t
from temgymcore_gb300.run import _grad_params, pack_model, param_gradient

SHARED = {"f": torch.tensor(0.2, dtype=torch.float64, requires_grad=True)}


class _Linked(t.Lens):
    """A lens whose focal length is looked up elsewhere."""
    focal_length = property(lambda self: SHARED["f"], lambda self, v: None)


class _Turned(t.DescanError):
    def as_matrix4(self):
        return super().as_matrix4().T

    def offsets(self):
        return [2.0 * v for v in super().offsets()]


def _descanner(error):
    return t.Descanner(z=0.1, scan_pos_x=1.0, scan_pos_y=2.0, scan_tilt_x=3.0, scan_tilt_y=4.0, descan_error=error)


def test_a_parameter_outside_the_instance_is_found():
    model = [_Linked(z=0.5, focal_length=None), t.Detector(z=1.0, pixel_size=(1e-5, 1e-5), shape=(8, 8))]
    (i, path, p), = _grad_params(model)
    assert (i, path) == (0, "focal_length") and p is SHARED["f"]


def test_a_descan_error_with_its_own_matrix():
    e = _Turned(*np.random.default_rng(0).normal(size=20))
    _, arr = pack_model([_descanner(e)])
    assert list(arr[0].p)[:24] == [1.0, 2.0, 3.0, 4.0, *e.as_matrix4().reshape(-1), *e.offsets()]


def test_a_descan_error_of_another_type():
    plain = t.DescanError(*np.random.default_rng(1).normal(size=20))
    e = types.SimpleNamespace(**plain._asdict(), as_matrix4=plain.as_matrix4, offsets=plain.offsets)
    e.pxo_pyi = torch.tensor(0.5, dtype=torch.float64, requires_grad=True)
    model = [_descanner(e)]
    _, arr = pack_model(model)
    assert list(arr[0].p)[4:24] == [*plain.as_matrix4().reshape(-1), *plain.offsets()]
    assert [path for _, path, _ in _grad_params(model)] == ["descan_error.pxo_pyi"]
    raw = np.arange(8.0).reshape(2, 4)
    assert param_gradient(model, 0, "descan_error.pxo_pyi", raw) == raw[1, 0] * 2.0  # times scan_pos_y
