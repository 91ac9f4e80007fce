"""The lean adjoint's two forms about the sizes where the choice between them changes: two
to five components, with and without parameter sums.  Leaving out an upstream gradient
that is zero takes the other form, whose operations are the same in the same order."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sums", [False, True])
@pytest.mark.parametrize("k", [2, 3, 4, 5])
@pytest.mark.parametrize("n", [8, 2056, 400_000, 400_008, 1_249_992, 1_250_000])
def test_forms_of_the_lean_adjoint(cuda, n, k, sums):
    import temgymcore_gb300 as t
    g = torch.Generator(device="cuda").manual_seed(n)
    rays = [(torch.randn(n, generator=g, device="cuda") * s).requires_grad_(True) for s in (5e-4, 5e-4, 1e-3, 1e-3)]
    f = torch.tensor(0.4, dtype=torch.float64, requires_grad=sums)
    a = torch.tensor(20.0, dtype=torch.float64, requires_grad=sums and k > 3)
    model = [t.Lens(z=0.2, focal_length=f), t.Deflector(z=0.3, def_x=1e-4, def_y=2e-4), t.Rotator(z=0.4, angle=a),
             t.Scanner(z=0.5, scan_pos_x=1e-4, scan_pos_y=2e-4)][:k - 1]
    model.append(t.Detector(z=0.9, pixel_size=(1e-5, 1e-5), shape=(64, 64)))
    ray = t.Ray(x=rays[0], y=rays[1], dx=rays[2], dy=rays[3], z=0.0, pathlength=0.0)
    up = [torch.randn(n, device="cuda", generator=g) for _ in range(3)]
    leaves = rays + [p for p in (f, a) if p.requires_grad]

    def grads(explicit):
        out = t.run_to_end(ray, model)
        outs = [out.x, out.y, out.dx] + ([out.dy] if explicit else [])
        return torch.autograd.grad(outs, leaves, up + ([torch.zeros_like(out.dy)] if explicit else []))

    for u, v in zip(grads(True), grads(False)):
        assert torch.equal(u, v)
