"""GPU: the field's gradients formed for some inputs only are the ones of all of
them: beam coordinates one by one, step sums one by one, with a singular B (a
conjugate plane, where the field's formula and so its gradients are NaN), a
rotator and a biprism, and in the beams' own plane.

Tolerance: the same float64 algebra in groups of another width, on the same
moments; 1e-12 of the largest covers its rounding (1e-16) times the algebra's
condition (matrices of unit order here, focal lengths of a fraction of a metre)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

BEAM = ("amplitude", "pathlength", "x", "y", "dx", "dy")


def _model(name, params):
    import temgymcore_gb300 as t
    grid = dict(pixel_size=(2e-7, 2e-7), shape=(40, 36))
    f, z, ax, ang = params
    if name == "image":  # object and image plane of the lens: B = 0
        return [t.Lens(z=z, focal_length=f), t.Detector(z=1.0, **grid)]
    return [t.Lens(z=z, focal_length=f), t.Rotator(z=0.6, angle=ang), t.Biprism(z=0.7, def_x=ax),
            t.Detector(z=1.3, **grid)]


def _leaves(n, seed):
    r = np.random.default_rng(seed)
    dev = "cuda"
    c = lambda s: torch.tensor(r.normal(0, s, n), dtype=torch.float64, device=dev)  # noqa: E731
    beams = {"x": c(1e-6), "y": c(1e-6), "dx": c(1e-6), "dy": c(1e-6), "pathlength": c(1e-12),
             "amplitude": torch.tensor(r.normal(size=n) + 1j * r.normal(size=n), dtype=torch.complex64, device=dev)}
    params = [torch.tensor(v, dtype=torch.float64) for v in (0.25, 0.5, 1e-6, 3.0)]
    return beams, params


def _grads(name, leaves, want_beams, want_params):
    import temgymcore_gb300 as t
    beams, params = leaves
    beams = {k: v.clone().requires_grad_(k in want_beams) for k, v in beams.items()}
    params = [p.clone().requires_grad_(i in want_params) for i, p in enumerate(params)]
    n = beams["x"].numel()
    rays = t.GaussianRay(z=0.0, waist_xy=np.full((n, 2), 3e-6), radii_of_curv=np.full((n, 2), np.inf),
                         wavelength=1.97e-12, theta=np.linspace(0.0, 1.0, n), **beams)
    if name == "own":
        out = t.evaluate_gaussian_input_image(rays, t.Detector(z=0.0, pixel_size=(2e-7, 2e-7), shape=(40, 36)))
    else:
        out = t.make_gaussian_image(rays, _model(name, params))
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    up = torch.randn(40, 36, dtype=torch.complex64, device="cuda", generator=g)
    wanted = [beams[k] for k in want_beams] + [params[i] for i in want_params]
    got = torch.autograd.grad(out, wanted, up)
    return [v.cpu() for v in got]


def _same(got, want):
    nan = torch.isnan(want.abs())
    assert torch.equal(torch.isnan(got.abs()), nan)
    if not nan.all():
        assert (got - want)[~nan].abs().max() <= 1e-12 * want[~nan].abs().max()


@pytest.mark.parametrize("name", ["image", "column", "own"])
@pytest.mark.parametrize("n", [1, 65])
def test_field_gradients_of_subsets(cuda, name, n):
    leaves = _leaves(n, n)
    steps = {"image": [0, 1], "column": [0, 1, 2, 3], "own": []}[name]
    full = _grads(name, leaves, BEAM, steps)
    for i, k in enumerate(BEAM):
        _same(_grads(name, leaves, (k,), [])[0], full[i])
    for j, p in enumerate(steps):
        _same(_grads(name, leaves, (), [p])[0], full[len(BEAM) + j])


@pytest.mark.parametrize("name", ["image", "column"])
@pytest.mark.parametrize("n", [1, 64, 131])
def test_field_gradients_from_the_forward_records(cuda, name, n):
    """The unit-amplitude records that the differentiable forward leaves are the
    ones that the adjoint forms by itself (FieldPlan.vjp): bit for bit, NaN
    included, and so are the beams' gradients."""
    import temgymcore_gb300 as t
    from temgymcore_gb300.gaussian import FieldPlan
    beams, params = _leaves(n, n)
    rays = t.GaussianRay(z=0.0, waist_xy=np.full((n, 2), 3e-6), radii_of_curv=np.full((n, 2), np.inf),
                         wavelength=1.97e-12, theta=np.linspace(0.0, 1.0, n), **beams)
    model = _model(name, params)
    own, left = FieldPlan(rays, model), FieldPlan(rays, model, _unit=True)
    assert own.unit is None and left.unit is not None
    up = torch.ones(40, 36, dtype=torch.complex64, device="cuda")
    a, b = own.vjp(up), left.vjp(up)
    for k in a:
        assert torch.equal(torch.nan_to_num(torch.view_as_real(a[k]) if a[k].is_complex() else a[k]),
                           torch.nan_to_num(torch.view_as_real(b[k]) if b[k].is_complex() else b[k])), k
