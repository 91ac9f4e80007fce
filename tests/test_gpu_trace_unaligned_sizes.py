"""GPU: arrays of any alignment about the size where a thread takes four rays instead of
one (1,536 rays an SM: 233,472 on 152 SMs): the same bits as aligned arrays give."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _model(k, hw):
    import temgymcore_gb300 as t
    m = [t.Lens(z=.2, focal_length=.4), t.Deflector(z=.3, def_x=1e-4, def_y=1e-5), t.Rotator(z=.4, angle=3.),
         t.Aperture(z=.6, radius=2e-3), t.Biprism(z=.7, def_x=1e-4), t.Descanner(z=.8, scan_pos_x=1e-4, scan_pos_y=0.)]
    return m[:k - 1] + [t.Detector(z=1.0, pixel_size=(1e-5, 1e-5), shape=(hw, hw))]


@pytest.mark.parametrize("dtype", [torch.int32, torch.int64])
@pytest.mark.parametrize("hw", [32, 200])  # 32: counters in shared memory
@pytest.mark.parametrize("k,n", [(1, 1), (3, 257), (7, 100_001), (2, 233_472), (7, 233_473)])
def test_one_and_four_rays_a_thread(cuda, k, n, hw, dtype):
    import temgymcore_gb300 as t
    model = _model(k, hw)
    g = torch.Generator(device=cuda).manual_seed(n)
    runs = []
    for off in (0, 1, 3):
        rows = []
        g.manual_seed(n)
        for _ in range(4):
            b = torch.empty(n + 4, device=cuda)
            b[off:off + n] = (torch.rand(n, device=cuda, generator=g) - 0.5) * 2e-3
            rows.append(b[off:off + n])
        p = t.TracePlan(model, *rows, detector=model[-1], pixels=True, hist_dtype=dtype).run()
        runs.append([*p.out, p.pathlength, *p.pix, p.image])
    for other in runs[1:]:
        assert all(torch.equal(a, b) for a, b in zip(runs[0], other))
    assert int(runs[0][-1].sum()) <= n and np.isfinite(runs[0][0].cpu().numpy()).all()
