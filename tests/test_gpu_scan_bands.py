"""Boxes larger than the window's one band: bands of the window where every SM is full and
rows are left to the bulk copies (by image size, rows lit and probes), a zero fill with
atomics elsewhere, bands in host memory.  Against the oracle's per-probe images."""
import numpy as np
import pytest
import torch

from test_gpu_scan import _check

pytestmark = pytest.mark.gpu

PROBES = 700  # above four CTAs an SM


def _bundle(cuda, shape, rows, rays):
    """A workload whose bundle lights about ``rows`` rows, and its ray and model."""
    import temgymcore_gb300 as t
    from temgymcore_gb300.workloads import stem_4d, stem_model
    w = stem_4d(seed=3, scan=(2, 2), rays_per_probe=rays, det_shape=shape)
    wide = np.float32(0.5 * rows * w["detector"]["pixel_size"][0] / (0.1 * np.abs(w["dy"]).max()))
    w["dx"], w["dy"] = w["dx"] * wide, w["dy"] * wide
    ray = t.Ray(**{k: torch.tensor(w[k], device=cuda) for k in ("x", "y", "dx", "dy")}, z=0.0, pathlength=0.0)
    return w, ray, stem_model(w)


def _scan(cuda, shape, rows, rays, probes, **kw):
    import temgymcore_gb300 as t
    w, ray, model = _bundle(cuda, shape, rows, rays)
    px = w["detector"]["pixel_size"][0]
    pos = np.random.default_rng(4).uniform(-3 * px, 3 * px, (probes, 2))
    pos[1] = [1e3, 1e3]  # this one misses
    imgs, xy = t.scan_images(ray, model, positions=pos, return_xy=True, **kw)
    return w, imgs, xy, pos


@pytest.mark.parametrize("rays", [257, 1024])
@pytest.mark.parametrize("rows", [110, 130, 190])
@pytest.mark.parametrize("shape", [(200, 200), (199, 200), (300, 300), (260, 340), (200, 202)])
def test_many_probes(cuda, shape, rows, rays):
    w, imgs, xy, pos = _scan(cuda, shape, rows, rays, PROBES)
    lit = imgs[0].sum(1).nonzero()
    assert int(lit.max() - lit.min()) > 0.85 * rows
    pick = [0, 1, 2, 3, PROBES // 2, PROBES - 1]
    _check(w, imgs[pick], xy[pick], pos[pick])
    # every probe: the few-probe route (a zero fill and atomics) writes the same images
    import temgymcore_gb300 as t
    _, ray, model = _bundle(cuda, shape, rows, rays)
    few = [t.scan_images(ray, model, positions=pos[i:i + 70]) for i in range(0, PROBES, 70)]
    assert torch.equal(imgs, torch.cat(few))


@pytest.mark.parametrize("shape", [(257, 256), (201, 203)])
def test_images_in_host_memory(cuda, shape):
    out = torch.full((5, *shape), 9, dtype=torch.int32).pin_memory()
    w, imgs, xy, pos = _scan(cuda, shape, 190, 1024, 5, out=out)
    torch.cuda.synchronize()
    _check(w, imgs, xy, pos)


@pytest.mark.parametrize("first", [1, 2, 3])
@pytest.mark.parametrize("shape", [(201, 203), (225, 225), (1, 20001)])
def test_zero_fill_of_unaligned_images(cuda, first, shape):
    """Images that do not start on 16 bytes, between neighbours that stay as they are."""
    n = 4 * shape[0] * shape[1]
    whole = torch.full((n + 8,), 7, dtype=torch.int32, device=cuda)
    out = whole[first:first + n].view(4, *shape)
    w, imgs, xy, pos = _scan(cuda, shape, 190, 300, 4, out=out)
    _check(w, imgs, xy, pos)
    assert (whole[:first] == 7).all() and (whole[first + n:] == 7).all()
