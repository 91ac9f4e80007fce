"""The trace's backward pass when only some outputs feed the loss, for the lean
and the general adjoint, host and device parameters, aligned and odd rays."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

_OUT = ("x", "y", "dx", "dy", "pathlength")


def _case(n, seed, biprism, where, dtype=torch.float64):
    import temgymcore_gb300 as t
    g = torch.Generator(device="cuda").manual_seed(seed)
    rays = [(torch.randn(n, generator=g, device="cuda") * s).requires_grad_(True) for s in (5e-4, 5e-4, 1e-3, 1e-3)]
    pl = torch.rand(n, generator=g, device="cuda", dtype=torch.float64).requires_grad_(True)
    p = [torch.tensor(v, dtype=dtype, device=where, requires_grad=True) for v in (0.4, 1e-4, 1.01, 0.9)]
    model = [t.Scanner(z=0.1, scan_pos_x=p[1], scan_pos_y=2e-4),
             t.Descanner(z=0.1, scan_pos_x=1e-4, scan_pos_y=2e-4, descan_error=t.DescanError(pxo_pxi=p[2], syo_pyi=0.1)),
             t.Lens(z=0.3, focal_length=p[0]), t.Rotator(z=0.4, angle=20.0)]
    model += [t.Biprism(z=0.5, def_x=1e-4)] if biprism else [t.Deflector(z=0.5, def_x=1e-4, def_y=2e-4)]
    model.append(t.Detector(z=p[3], pixel_size=(1e-5, 1e-5), shape=(64, 64)))
    ray = t.Ray(x=rays[0], y=rays[1], dx=rays[2], dy=rays[3], z=0.0, pathlength=pl)
    return ray, model, rays + [pl] + p


@pytest.mark.parametrize("where", ["cpu", "cuda"])
@pytest.mark.parametrize("biprism", [False, True])
@pytest.mark.parametrize("n", [1, 2047, 4099])
@pytest.mark.parametrize("used", [("x",), ("x", "y"), ("dy",), ("pathlength",), ("y", "pathlength"), _OUT])
def test_missing_gradients_are_zero_gradients(cuda, n, biprism, used, where):
    """Gradients of a loss over some outputs equal those with explicit zero
    gradients for the others (which read and add the zeros)."""
    import temgymcore_gb300 as t
    up = {k: torch.randn(n, device="cuda", dtype=torch.float64 if k == "pathlength" else torch.float32) for k in used}

    def grads(explicit):
        ray, model, leaves = _case(n, 3, biprism, where)
        out = t.run_to_end(ray, model)
        keys = _OUT if explicit else used
        seeds = [up.get(k, torch.zeros_like(getattr(out, k))) for k in keys]
        return torch.autograd.grad([getattr(out, k) for k in keys], leaves, seeds, allow_unused=True)

    for a, b in zip(grads(False), grads(True)):
        assert a is not None and a.dtype == b.dtype and a.shape == b.shape and a.device == b.device
        a, b = a.double().cpu().numpy(), b.double().cpu().numpy()
        # float32 sums of n terms in a fixed order: within n + 16 roundings of the largest
        np.testing.assert_allclose(a, b, rtol=0, atol=(16 + n) * 2.0 ** -24 * max(np.max(np.abs(b)), 1e-30))


@pytest.mark.parametrize("n", [1, 8, 2047, 2048, 700_001])
@pytest.mark.parametrize("kind", ["lens", "shift", "deflect", "rotate"])
def test_short_chains(cuda, n, kind):
    """Chains of two components with every gradient given (their own form of the
    lean adjoint) against one gradient left out, zero (the other form): the same
    operations in the same order."""
    import temgymcore_gb300 as t
    g = torch.Generator(device="cuda").manual_seed(n)
    rays = [(torch.randn(n, generator=g, device="cuda") * s).requires_grad_(True) for s in (5e-4, 5e-4, 1e-3, 1e-3)]
    p = torch.tensor({"lens": 0.4, "shift": 1e-4, "deflect": 1e-4, "rotate": 20.0}[kind], dtype=torch.float64,
                     requires_grad=True)
    z = torch.tensor(0.3, dtype=torch.float64, requires_grad=True)
    first = {"lens": lambda: t.Lens(z=z, focal_length=p), "shift": lambda: t.Scanner(z=z, scan_pos_x=p, scan_pos_y=2e-4),
             "deflect": lambda: t.Deflector(z=z, def_x=p, def_y=2e-4), "rotate": lambda: t.Rotator(z=z, angle=p)}[kind]()
    model = [first, t.Detector(z=0.9, pixel_size=(1e-5, 1e-5), shape=(64, 64))]
    ray = t.Ray(x=rays[0], y=rays[1], dx=rays[2], dy=rays[3], z=0.0, pathlength=0.0)
    up = [torch.randn(n, device="cuda", generator=g) for _ in range(3)]

    def grads(explicit):
        out = t.run_to_end(ray, model)
        outs = [out.x, out.y, out.dx] + ([out.dy] if explicit else [])
        return torch.autograd.grad(outs, rays + [p, z], up + ([torch.zeros_like(out.dy)] if explicit else []))

    for a, b in zip(grads(True), grads(False)):
        a, b = a.double().cpu().numpy(), b.double().cpu().numpy()
        np.testing.assert_allclose(a, b, rtol=0, atol=2.0 ** -20 * max(np.max(np.abs(b)), 1e-30))
