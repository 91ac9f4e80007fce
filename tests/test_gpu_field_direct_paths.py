"""The direct field sum's per-strip choices (ratio table, recurrence, per
pixel, skip) against the float64 kernel, over beam widths and odd sizes."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(33, 31), (64, 257), (130, 100)])
@pytest.mark.parametrize("waist_px", [0.35, 1.5, 3.2, 3.41, 3.6, 9.0, 70.0])
def test_direct_matches_float64(cuda, waist_px, shape):
    """Each value is at most 31 steps of two factors, each within ~2^-23, from
    an anchor of that accuracy: 31 * 2^-22 < 1e-5, and so is the sum, normwise."""
    import temgymcore_gb300 as t
    from temgymcore_gb300.gaussian import FieldPlan
    px, n = 1e-5, 130
    rng = np.random.default_rng(int(waist_px * 100))
    half = 0.5 * px * np.array(shape)
    w = waist_px * px * rng.uniform(0.9, 1.1, (n, 2))
    rays = t.GaussianRay(
        x=rng.uniform(-1.1, 1.1, n) * half[1], y=rng.uniform(-1.1, 1.1, n) * half[0], dx=rng.normal(0, 1e-3, n),
        dy=rng.normal(0, 1e-3, n), z=0.0, pathlength=rng.normal(0, 1e-3, n),
        amplitude=rng.normal(size=n) + 1j * rng.normal(size=n), waist_xy=w, radii_of_curv=rng.normal(0, 0.5, (n, 2)),
        wavelength=5e-7, theta=rng.uniform(0, np.pi, n))
    plan = FieldPlan(rays, None, "direct", grid=t.Detector(z=0.0, pixel_size=(px, px), shape=shape))
    got, ref = plan.evaluate("direct").clone().cpu().numpy(), plan.evaluate("fp64").cpu().numpy()
    assert np.max(np.abs(got - ref)) <= 1e-5 * np.max(np.abs(ref))
