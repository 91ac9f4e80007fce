"""Scans whose rows are not whole 16-byte vectors, written pixel by pixel: widths about
the block's 256 threads, a few columns, a few rows; one image of more than 2^31 pixels."""
import numpy as np
import pytest
import torch

from test_gpu_scan import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rays", [1, 1001])
@pytest.mark.parametrize("semi", [5e-3, 6e-2])
@pytest.mark.parametrize("shape", [(161, 203), (90, 255), (80, 257), (61, 513), (2100, 13), (7, 4099), (25001, 1)])
def test_scan_rows_of_any_width(cuda, rays, semi, shape):
    import temgymcore_gb300 as t
    from temgymcore_gb300.workloads import stem_4d, stem_model
    w = stem_4d(seed=7, scan=(2, 2), rays_per_probe=rays, semi_conv=semi, det_shape=shape)
    model = stem_model(w)
    ray = t.Ray(x=torch.tensor(w["x"], device=cuda), y=torch.tensor(w["y"], device=cuda),
                dx=torch.tensor(w["dx"], device=cuda), dy=torch.tensor(w["dy"], device=cuda),
                z=0.0, pathlength=0.0)
    half = 0.5 * shape[0] * w["detector"]["pixel_size"][0]
    pos = np.array([[0.0, 0.0], [half * 0.9, 0.0], [0.0, -half], [50.0, 50.0]])  # the last one misses
    out = torch.full((len(pos), *shape), 777, dtype=torch.int32, device=cuda)
    imgs, xy = t.scan_images(ray, model, positions=pos, out=out, return_xy=True)
    _check(w, imgs, xy, pos)
    assert int(imgs[3].abs().sum()) == 0


def test_scan_image_of_more_than_two_to_the_31_pixels(cuda):
    import temgymcore_gb300 as t
    h, w, n = 46_342, 46_343, 100
    px = 1e-6
    det = t.Detector(z=0.1, pixel_size=(px, px), shape=(h, w))
    rows = torch.linspace(0, h - 1, n, device=cuda, dtype=torch.float64).round()
    z = torch.zeros(n, device=cuda)
    x, y = det.pixels_to_metres((rows.cpu().numpy(), np.full(n, 5.0)))
    out = torch.full((1, h, w), 7, dtype=torch.int32, device=cuda)
    t.scan_images(t.Ray(x=torch.tensor(np.float32(x), device=cuda), y=torch.tensor(np.float32(y), device=cuda), dx=z,
                        dy=z, z=0.0, pathlength=0.0), [det], positions=np.zeros((1, 2)), out=out)
    assert int(out.sum(dtype=torch.int64)) == n and int(out[0, :, :64].sum()) == n
    assert int(out[0, 0].sum()) == 1 and int(out[0, h - 1].sum()) == 1
