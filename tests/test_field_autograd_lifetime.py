"""A differentiable field's plan (workspaces, records) lives as long as its graph and no
longer: it goes with the last reference, without the cyclic collector."""
import gc
import weakref

import numpy as np
import pytest
import torch


@pytest.fixture
def no_collector():
    gc.collect()
    gc.disable()
    yield
    gc.enable()


class _Plan:
    """Stands in for a FieldPlan on the CPU."""
    comps = _packed = None

    def __init__(self):
        self.out = torch.zeros(4, 4, dtype=torch.complex64)

    def evaluate(self):
        return self.out

    def vjp(self, grad, **_):
        return {"x": torch.ones(3, dtype=torch.float64)}


@pytest.mark.parametrize("backward", [True, False])
def test_no_plan_outlives_its_graph(no_collector, backward):
    from temgymcore_gb300.gaussian import _FieldFn
    x = torch.zeros(3, dtype=torch.float64, requires_grad=True)
    alive = []
    for _ in range(3):
        plan = _Plan()
        alive.append(weakref.ref(plan))
        out = _FieldFn.apply({"plan": plan, "beam_inputs": [("x", x)], "params": []}, x)
        del plan
        if backward:
            assert torch.autograd.grad(out.abs().sum(), x)[0].tolist() == [1.0] * 3
        del out
        assert all(ref() is None for ref in alive)


@pytest.mark.gpu
@pytest.mark.parametrize("own_plane", [False, True])
def test_memory_stays_flat_over_a_fit(cuda, no_collector, own_plane):
    import temgymcore_gb300 as t
    r = np.random.default_rng(0)
    n = 300
    x = torch.tensor(r.normal(0, 1e-6, n), device="cuda", requires_grad=True)
    z = torch.zeros(n, dtype=torch.float64, device="cuda")
    rays = t.GaussianRay(x=x, y=z, dx=z, dy=z, z=0.0, pathlength=z, amplitude=1.0, waist_xy=np.full((n, 2), 3e-6),
                         radii_of_curv=np.full((n, 2), np.inf), wavelength=1.97e-12, theta=0.0)
    det = t.Detector(z=0.0 if own_plane else 1.3, pixel_size=(2e-7, 2e-7), shape=(40, 36))
    f = torch.tensor(0.25, dtype=torch.float64, requires_grad=True)

    def step():
        if own_plane:
            return torch.autograd.grad(t.evaluate_gaussian_input_image(rays, det).abs().sum(), x)
        out = t.make_gaussian_image(rays, [t.Lens(z=0.5, focal_length=f), det])
        return torch.autograd.grad(out.abs().sum(), (x, f))

    held = []
    for _ in range(5):
        step()
        held.append(torch.cuda.memory_allocated())
    assert held[1:] == held[1:2] * 4
