"""GPU: rays on the axis of a detector with an even number of pixels (an exact tie, which
the float64 path decides), with threads left over at the end of a block and of a launch."""
import numpy as np
import pytest
import torch

from oracle import grid as OG

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("hw", [8, 256])
@pytest.mark.parametrize("n", [1, 3, 255, 1025, 4097, 9001])
def test_ties_and_threads_without_a_ray(cuda, n, hw, off):
    import temgymcore_gb300 as t
    px = 2.0 ** -16
    det = t.Detector(z=0.0, pixel_size=(px, px), shape=(hw, hw))
    r = np.random.default_rng(n)
    xy = np.where(r.random((2, n)) < 0.5, 0.0, r.integers(-hw, hw, (2, n)) * px / 2).astype(np.float32)
    xy[0, -1] = np.nan if n > 1 else 0.0
    buf = torch.zeros(4, n + 8, device=cuda)
    rows = [buf[i, off:off + n] for i in range(4)]
    for row, v in zip(rows, xy):
        row.copy_(torch.tensor(v))
    ray = t.Ray(x=rows[0], y=rows[1], dx=rows[2], dy=rows[3], z=0.0, pathlength=0.0)
    out, pix, img = t.trace_to_image(ray, [det])
    g = {"pixel_size": (px, px), "shape": (hw, hw)}
    py, pxx = OG.metres_to_pixels(g, xy[0].astype(np.float64), xy[1].astype(np.float64))
    assert np.array_equal(pix.y.cpu().numpy(), py) and np.array_equal(pix.x.cpu().numpy(), pxx)
    assert np.array_equal(img.cpu().numpy(), OG.into_image(g, py, pxx))
    imgs = t.scan_images(ray, [det], positions=np.zeros((3, 2)))
    assert all(np.array_equal(i.cpu().numpy(), img.cpu().numpy()) for i in imgs)
    # the NaN is reported, the threads without a ray are not
    assert t._native.error_word(clear=True) == (t._native.EW_NONFINITE if n > 1 else 0)
