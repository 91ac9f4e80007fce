"""The field GEMM's epilogue at images that fill part of a 128 x 128 tile: rows of a warp
and 32-column chunks inside, on the edge and outside, even and odd widths.  With the same
pixel map, and up to 32 beams in one K block, a small image is the corner of a large one,
bit for bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

PX = 2.0 ** -20


def _grid(shape):
    """A grid whose pixel (0, 0) lies at the origin, whatever its shape."""
    import temgymcore_gb300 as t
    m = t.Detector(z=0.0, pixel_size=(PX, PX), shape=shape)._pixel_map()
    return t.Detector(z=0.0, pixel_size=(PX, PX), shape=shape, centre=(m[2], -m[5]))


@pytest.mark.parametrize("n", [1, 32])
@pytest.mark.parametrize("shape", [(1, 1), (1, 33), (31, 2), (32, 32), (33, 31), (64, 97), (65, 96), (96, 128), (129, 130),
                                   (160, 129)])
def test_partial_tiles(cuda, shape, n):
    import temgymcore_gb300 as t
    r = np.random.default_rng(n)
    c = lambda s: torch.tensor(r.normal(0, s, n), device="cuda")  # noqa: E731
    rays = t.GaussianRay(x=c(PX * 50), y=c(PX * 50), dx=c(1e-5), dy=c(1e-5), z=0.0, pathlength=c(1e-9),
                         amplitude=torch.tensor(r.normal(size=n) + 1j * r.normal(size=n), dtype=torch.complex64,
                                                device="cuda"),
                         waist_xy=np.full((n, 2), 60 * PX), radii_of_curv=np.full((n, 2), np.inf), wavelength=1e-9,
                         theta=0.0)
    small, large = _grid(shape), _grid((256, 256))
    assert small._pixel_map() == large._pixel_map()
    got = t.evaluate_gaussian_input_image(rays, small, method="separable")
    want = t.evaluate_gaussian_input_image(rays, large, method="separable")[:shape[0], :shape[1]]
    assert torch.equal(torch.view_as_real(got), torch.view_as_real(want.contiguous())) and got.abs().max() > 0
