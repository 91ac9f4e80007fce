"""Scans whose discs or bundles exceed one shared-memory window: bands of the
window, whole-image counters in shared memory, and global atomics, against the
oracle's per-probe run_to_end + into_image."""
import numpy as np
import pytest
import torch

from test_gpu_scan import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rays,semi,shape", [
    (4096, 6e-2, (256, 256)),   # largest bundle of packed pixels, a disc of many bands
    (1000, 1e-1, (161, 203)),   # bands with rows that are not 16-byte aligned
    (1, 5e-3, (128, 144)),      # the largest image of six CTAs an SM, one ray
    (2047, 4e-2, (190, 200)),   # the last bundle before, and
    (2048, 4e-2, (190, 200)),   # the first of the whole-image counters beside three CTAs
    (4097, 4e-2, (230, 240)),   # counters beside two CTAs
    (4097, 6e-2, (192, 192)),   # smallest bundle of the whole-image counters
    (5003, 3e-2, (33, 47)),     # an odd number of pixels
    (4099, 5e-3, (336, 336)),   # counters that leave room for one CTA an SM
    (4101, 5e-3, (340, 344)),   # an image beyond shared memory
    (65535, 2e-2, (64, 64)),    # the most rays a 16-bit counter holds
    (65536, 2e-2, (64, 64)),    # one more
])
def test_scan_image_paths(cuda, rays, semi, shape):
    import temgymcore_gb300 as t
    from temgymcore_gb300.workloads import stem_4d, stem_model
    w = stem_4d(seed=11, scan=(2, 2), rays_per_probe=rays, semi_conv=semi, det_shape=shape)
    model = stem_model(w)
    ray = t.Ray(x=torch.tensor(w["x"], device=cuda), y=torch.tensor(w["y"], device=cuda),
                dx=torch.tensor(w["dx"], device=cuda), dy=torch.tensor(w["dy"], device=cuda),
                z=0.0, pathlength=0.0)
    half = 0.5 * shape[0] * w["detector"]["pixel_size"][0]
    pos = np.array([[0.0, 0.0], [half * 0.9, 0.0], [0.0, -half], [5.0, 5.0]])  # the last one misses
    out = torch.full((len(pos), *shape), 777, dtype=torch.int32, device=cuda)
    imgs, xy = t.scan_images(ray, model, positions=pos, out=out, return_xy=True)
    _check(w, imgs, xy, pos)
    assert int(imgs[3].abs().sum()) == 0
    assert torch.equal(t.scan_images(ray, model, positions=pos), imgs)


def test_scan_image_one_pixel_holds_every_ray(cuda):
    """All 65,535 rays on one pixel: the counter's largest value, in either
    half of its word, without a carry into its neighbour."""
    import temgymcore_gb300 as t
    n = 65535
    z = torch.zeros(n, device=cuda)
    model = [t.Detector(z=0.1, pixel_size=(1e-5, 1e-5), shape=(32, 32))]
    pos = np.zeros((2, 2))
    for shift in (0.4e-5, -0.6e-5):
        imgs = t.scan_images(t.Ray(x=z + shift, y=z + 0.4e-5, dx=z, dy=z, z=0.0, pathlength=0.0), model,
                             positions=pos)
        assert imgs.max().item() == n and int(imgs.sum()) == 2 * n and int((imgs != 0).sum()) == 2
