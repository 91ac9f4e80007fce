"""What a caller could set on a plan and on its beams can be set (CPU only)."""
import numpy as np
import torch

import temgymcore_gb300 as t
from temgymcore_gb300.gaussian import BeamSet, FieldPlan


def test_the_method_can_be_set():
    plan = object.__new__(FieldPlan)
    plan.method = "direct"
    assert plan.method == "direct"
    plan.method = "fp64"
    assert plan.method == "fp64"


def test_wavelength_and_angle_can_be_set():
    z = torch.zeros(3, dtype=torch.float64)
    b = BeamSet(t.GaussianRay(x=z, y=z, dx=z, dy=z, z=0.0, pathlength=z, amplitude=1.0, waist_xy=np.ones((3, 2)),
                              radii_of_curv=np.ones((3, 2)), wavelength=1e-9, theta=0.0), torch.device("cpu"))
    assert b.wl.tolist() == [1e-9] * 3 and b.theta.tolist() == [0.0] * 3
    wl, theta = torch.full_like(z, 2e-9), torch.full_like(z, 0.5)
    b.wl, b.theta = wl, theta
    s = b.struct()
    assert b.wl is wl and b.theta is theta and (s.wavelength, s.theta) == (wl.data_ptr(), theta.data_ptr())


def test_a_wavelength_that_was_read_can_be_changed_in_place():
    """The array is the beams' own from its first reading on."""
    z = torch.zeros(3, dtype=torch.float64)
    b = BeamSet(t.GaussianRay(x=z, y=z, dx=z, dy=z, z=0.0, pathlength=z, amplitude=1.0, waist_xy=np.ones((3, 2)),
                              radii_of_curv=np.ones((3, 2)), wavelength=1e-9, theta=0.0), torch.device("cpu"))
    b.wl.mul_(2.0)
    b.theta.add_(0.5)
    assert b.wl.tolist() == [2e-9] * 3 and b.theta.tolist() == [0.5] * 3
    s = b.struct()
    assert (s.wavelength, s.theta) == (b.wl.data_ptr(), b.theta.data_ptr())
