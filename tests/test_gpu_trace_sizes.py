"""The fused trace at the sizes where its launches change, and its pixel
indices next to rounding ties over many detector sizes."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


def _model():
    import temgymcore_gb300 as t
    return [t.Scanner(z=0.1, scan_pos_x=1e-4, scan_pos_y=-2e-4), t.Lens(z=0.3, focal_length=0.4),
            t.Deflector(z=0.4, def_x=1e-4, def_y=-3e-4), t.Rotator(z=0.5, angle=33.0),
            t.Biprism(z=0.55, def_x=2e-4), t.Aperture(z=0.6, radius=2e-3),
            t.Detector(z=0.9, pixel_size=(9e-6, 9e-6), shape=(250, 301))]


def _rays(n, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn(n, generator=g, device="cuda") * s for s in (5e-4, 5e-4, 1e-3, 1e-3)]


@pytest.mark.parametrize("n", [3, 1024, 1025, 700_001, 6_000_000, 9_000_003])
def test_launch_shapes_agree(cuda, n):
    """One call equals the same rays in pieces, bit for bit (every ray is
    independent), whatever the number of blocks and their turns."""
    import temgymcore_gb300 as t
    model = _model()
    cols = _rays(n)

    def call(lo, hi):
        x, y, dx, dy = (c[lo:hi].clone() for c in cols)
        return t.trace_to_image(t.Ray(x=x, y=y, dx=dx, dy=dy, z=0.0, pathlength=0.25), model)

    out, pix, img = call(0, n)
    cuts = [0] + ([n // 3, n // 3 + 1] if n > 3 else []) + [n]
    parts = [call(a, b) for a, b in zip(cuts, cuts[1:])]
    for k in ("x", "y", "dx", "dy", "pathlength"):
        assert torch.equal(getattr(out, k), torch.cat([getattr(p[0], k) for p in parts])), k
    assert torch.equal(pix.y, torch.cat([p[1].y for p in parts]))
    assert torch.equal(pix.x, torch.cat([p[1].x for p in parts]))
    assert torch.equal(img, sum(p[2] for p in parts))


@pytest.mark.parametrize("shape,rotation,centre", [
    ((32, 32), 0.0, (0.0, 0.0)), ((257, 64), 0.0, (3e-4, -7e-4)), ((512, 512), 31.0, (0.0, 0.0)),
    ((4096, 4095), 0.0, (0.0, 0.0)), ((60000, 60001), 12.5, (1e-2, 2e-2)), ((300, 300), 45.0, (30.0, -20.0)),
])
def test_pixels_next_to_ties(cuda, shape, rotation, centre):
    """Coordinates at the float32 neighbours of half-integer pixels: the index
    equals the float64 rounding of the float64 formula."""
    import temgymcore_gb300 as t
    px = 1e-5
    det = t.Detector(z=0.0, pixel_size=(px, px), shape=shape, rotation=rotation, centre=centre)
    rng = np.random.default_rng(5)
    n = 60_000
    row, col = rng.integers(-2, shape[0] + 2, n) + 0.5, rng.integers(-2, shape[1] + 2, n) + 0.5
    x, y = (np.asarray(v, np.float32) for v in det.pixels_to_metres((row, col)))
    for _ in range(3):
        x = np.where(rng.random(n) < 0.5, np.nextafter(x, np.float32(9)), x)
        y = np.where(rng.random(n) < 0.5, np.nextafter(y, np.float32(-9)), y)
    pix = det.metres_to_pixels((torch.tensor(x, device=cuda), torch.tensor(y, device=cuda)))
    g = {"pixel_size": (px, px), "shape": shape, "rotation": rotation, "centre": centre}
    py, pxx = oracle.metres_to_pixels(g, x.astype(np.float64), y.astype(np.float64))
    assert np.array_equal(pix.y.cpu().numpy(), py) and np.array_equal(pix.x.cpu().numpy(), pxx)
