"""GPU: gradients belong to one state of the inputs.  What is changed in place between
the forward and the backward pass (an optimiser's step while a graph is kept, a second
loss) does not mix with what the forward pass saw.

No tolerance: the same kernels on the same values give the same bits."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

P64 = dict(dtype=torch.float64, requires_grad=True)
GRID = dict(pixel_size=(2e-7, 2e-7), shape=(40, 36))


def _descan_error(r, dev):
    import temgymcore_gb300 as t
    scale = np.full(20, 0.1)
    scale[8:12] = 1e-7  # the offsets: metres and radians
    return t.DescanError(*(torch.tensor(v, device=dev, **P64) for v in r.normal(0, 1, 20) * scale))


def _field(dev, moved, astigmatic):
    """Gradients of a field; ``moved``: what changes in place before the backward pass."""
    import temgymcore_gb300 as t
    r = np.random.default_rng(0)
    n = 65
    c = lambda s: torch.tensor(r.normal(0, s, n), device="cuda", **P64)  # noqa: E731
    beams = {"x": c(1e-6), "y": c(1e-6), "dx": c(1e-6), "dy": c(1e-6), "pathlength": c(1e-12)}
    beams["amplitude"] = torch.tensor(r.normal(size=n) + 1j * r.normal(size=n), dtype=torch.complex64,
                                      device="cuda", requires_grad=True)
    other = {"waist_xy": torch.tensor(r.uniform(2e-6, 4e-6, (n, 2)) if astigmatic else np.full((n, 2), 3e-6),
                                      device="cuda"),
             "radii_of_curv": torch.full((n, 2), np.inf, dtype=torch.float64, device="cuda"),
             "wavelength": torch.full((n,), 1.97e-12, dtype=torch.float64, device="cuda"),
             "theta": torch.tensor(r.uniform(0, 1, n) if astigmatic else np.zeros(n), device="cuda")}
    f = torch.tensor(0.25, device=dev, **P64)
    spx = torch.tensor(1e-7, device=dev, **P64)
    err = _descan_error(r, dev)
    model = [t.Descanner(z=0.1, scan_pos_x=spx, scan_pos_y=2e-7, scan_tilt_x=1e-7, scan_tilt_y=3e-7, descan_error=err),
             t.Lens(z=0.5, focal_length=f), t.Detector(z=1.3, **GRID)]
    out = t.make_gaussian_image(t.GaussianRay(z=0.0, **beams, **other), model)
    leaves = {**beams, "f": f, "spx": spx, **err._asdict()}
    with torch.no_grad():
        for k in moved:
            v = {**leaves, **other}[k]
            v.mul_(1.5) if k != "theta" else v.add_(0.25)
    g = torch.Generator(device="cuda").manual_seed(1)
    up = torch.randn(40, 36, dtype=torch.complex64, device="cuda", generator=g)
    return dict(zip(leaves, torch.autograd.grad(out, list(leaves.values()), up)))


@pytest.mark.parametrize("dev", ["cpu", "cuda"])
@pytest.mark.parametrize("astigmatic", [False, True])
@pytest.mark.parametrize("moved", [("f",), ("x", "dy"), ("amplitude", "pathlength"), ("spx", "pxo_pxi"),
                                   ("waist_xy", "wavelength", "theta"), ("f", "x", "waist_xy")])
def test_field_gradients_are_the_forward_state_s(cuda, moved, astigmatic, dev):
    want, got = _field(dev, (), astigmatic), _field(dev, moved, astigmatic)
    assert all(v.abs().max() > 0 and torch.isfinite(v.abs()).all() for v in want.values())
    for k, v in want.items():
        assert torch.equal(got[k], v), k


def _trace(dev, moved):
    import temgymcore_gb300 as t
    r = np.random.default_rng(0)
    n = 1001
    rays = {k: torch.tensor(r.normal(0, 1e-3, n), dtype=torch.float32, device="cuda", requires_grad=True)
            for k in ("x", "y", "dx", "dy")}
    f, spx, spy = (torch.tensor(v, device=dev, **P64) for v in (0.25, 1e-4, 2e-4))
    err = _descan_error(r, dev)
    model = [t.Descanner(z=0.1, scan_pos_x=spx, scan_pos_y=spy, scan_tilt_x=1e-4, scan_tilt_y=3e-4, descan_error=err),
             t.Lens(z=0.5, focal_length=f), t.Biprism(z=0.7, def_x=1e-4), t.Detector(z=1.3, **GRID)]
    leaves = {**rays, "f": f, "spx": spx, "spy": spy, **err._asdict()}
    early, late = moved
    with torch.no_grad():
        for k in early:
            leaves[k].mul_(1.5)
    out = t.run_to_end(t.Ray(z=0.0, pathlength=0.0, **rays), model)
    with torch.no_grad():
        for k in late:
            leaves[k].mul_(1.5)
    g = torch.Generator(device="cuda").manual_seed(1)
    up = [torch.randn(n, device="cuda", generator=g) for _ in range(4)]
    return dict(zip(leaves, torch.autograd.grad([out.x, out.y, out.dx, out.dy], list(leaves.values()), up)))


def _equal(got, want):
    assert all(v.abs().max() > 0 for v in want.values())
    for k, v in want.items():
        assert torch.equal(got[k], v), k


@pytest.mark.parametrize("dev", ["cpu", "cuda"])
@pytest.mark.parametrize("moved", [("f",), ("spx", "spy"), ("pxo_pxi", "syo_pyi", "pyo_sxi"), ("f", "spy", "pxo_pyi")])
def test_trace_gradients_with_moved_parameters_are_the_forward_state_s(cuda, moved, dev):
    _equal(_trace(dev, ((), moved)), _trace(dev, ((), ())))


@pytest.mark.parametrize("dev", ["cpu", "cuda"])
@pytest.mark.parametrize("moved", [("x", "dy"), ("x", "f"), ("dx", "spx", "pxo_pxi")])
def test_trace_gradients_with_moved_rays_are_the_present_state_s(cuda, moved, dev):
    """The rays are not copied for the backward pass: where they moved, it reads
    the parameters at their present values too."""
    _equal(_trace(dev, ((), moved)), _trace(dev, (moved, ())))
