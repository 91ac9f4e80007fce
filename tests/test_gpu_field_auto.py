"""GPU: make_gaussian_image and evaluate_gaussian_input_image pick the method on
the device.  The same kernels run as for a plan whose method the host settled,
so the images are the same bit for bit; sizes about a tile of either method,
one beam and none separable among many, and no beams at all."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _beams(n, astigmatic, seed):
    import temgymcore_gb300 as t
    r = np.random.default_rng(seed)
    theta = np.zeros(n)
    waist = np.full((n, 2), 2e-6)
    if astigmatic == "all":
        theta, waist = r.uniform(0.1, 1.0, n), waist * np.array([1.0, 1.4])
    elif astigmatic == "last":
        theta[-1] = 0.4
        waist[-1, 1] *= 1.3
    return t.GaussianRay(x=r.normal(0, 1e-5, n), y=r.normal(0, 1e-5, n), dx=r.normal(0, 1e-5, n),
                         dy=r.normal(0, 1e-5, n), z=0.0, pathlength=np.zeros(n),
                         amplitude=np.ones(n, np.complex64), waist_xy=waist,
                         radii_of_curv=np.full((n, 2), np.inf), wavelength=1.97e-12, theta=theta)


@pytest.mark.parametrize("astigmatic", ["none", "last", "all"])
@pytest.mark.parametrize("n,h,w", [(1, 1, 1), (17, 33, 31), (300, 128, 129), (2000, 96, 320)])
def test_field_auto_is_the_settled_plan(cuda, astigmatic, n, h, w):
    import temgymcore_gb300 as t
    from temgymcore_gb300.gaussian import FieldPlan
    beams = _beams(n, astigmatic, n)
    det = t.Detector(z=1.0, pixel_size=(2e-7, 2e-7), shape=(h, w))
    model = [t.Lens(z=0.5, focal_length=0.4), det]
    plan = FieldPlan(beams, model)
    assert plan.method == ("separable" if astigmatic == "none" else "direct")
    assert torch.equal(t.make_gaussian_image(beams, model), plan.evaluate())
    own = FieldPlan(beams, None, grid=det)
    assert torch.equal(t.evaluate_gaussian_input_image(beams, det), own.evaluate())


def test_field_auto_captured(cuda):
    """A plan settled before is captured and replayed as it was."""
    import temgymcore_gb300 as t
    from temgymcore_gb300.gaussian import FieldPlan
    model = [t.Detector(z=0.5, pixel_size=(2e-7, 2e-7), shape=(64, 64))]
    plan = FieldPlan(_beams(100, "none", 1), model)
    want = plan.evaluate().clone()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        plan.evaluate()
    plan.out.zero_()
    g.replay()
    assert torch.equal(plan.out, want)
