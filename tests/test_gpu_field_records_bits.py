"""GPU: the unit-amplitude records that the differentiable forward leaves are, byte for
byte, the ones that the adjoint forms by itself, and the gradients from either are equal
bit for bit: a singular B (NaN records), amplitudes of zero, infinity and NaN."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

RECORD, USED = 96, 88  # bytes of a beam's record, and those that hold values


def _bits(t):
    t = torch.view_as_real(t) if t.is_complex() else t
    return t.contiguous().view(torch.uint8).cpu()


@pytest.mark.parametrize("name", ["image", "column"])
@pytest.mark.parametrize("n", [1, 64, 131])
def test_records_and_gradients_bit_for_bit(cuda, name, n):
    import temgymcore_gb300 as t
    from temgymcore_gb300.gaussian import FieldPlan
    r = np.random.default_rng(n)
    c = lambda s: torch.tensor(r.normal(0, s, n), device="cuda")  # noqa: E731
    amp = r.normal(size=n) + 1j * r.normal(size=n)
    amp[5::7], amp[6::11], amp[7::13] = 0.0, np.inf, np.nan
    rays = t.GaussianRay(x=c(1e-6), y=c(1e-6), dx=c(1e-6), dy=c(1e-6), z=0.0, pathlength=c(1e-12),
                         amplitude=torch.tensor(amp, dtype=torch.complex64, device="cuda"),
                         waist_xy=np.full((n, 2), 3e-6), radii_of_curv=np.full((n, 2), np.inf),
                         wavelength=1.97e-12, theta=np.linspace(0.0, 1.0, n))
    grid = dict(pixel_size=(2e-7, 2e-7), shape=(40, 36))
    model = [t.Lens(z=0.5, focal_length=0.25), t.Detector(z=1.0, **grid)] if name == "image" else [
        t.Lens(z=0.5, focal_length=0.25), t.Rotator(z=0.6, angle=3.0), t.Biprism(z=0.7, def_x=1e-6),
        t.Detector(z=1.3, **grid)]
    own, left = FieldPlan(rays, model), FieldPlan(rays, model, _unit=True)
    up = torch.ones(40, 36, dtype=torch.complex64, device="cuda")
    a, b = own.vjp(up), left.vjp(up)
    first = -own._vjp_ws.data_ptr() % 256  # the workspace begins with the records
    formed, kept = own._vjp_ws[first:first + RECORD * n], left.unit[:RECORD * n]
    assert torch.equal(formed.view(n, RECORD)[:, :USED].cpu(), kept.view(n, RECORD)[:, :USED].cpu())
    assert set(a) == set(b)
    for k in a:
        assert torch.equal(_bits(a[k]), _bits(b[k])), k
