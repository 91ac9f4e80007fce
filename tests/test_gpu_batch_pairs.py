"""GPU: the batched trace two rays at a time (2 and 4 rays a thread, at most four
biprisms) against one at a time: every ray's outputs, pathlength and aperture
decision the same bit for bit, over 0 to 6 biprisms (5 and 6 always run one by
one), with and without apertures, and ray counts about a block and a tile.

The loss is a sum of squares: its float32 part has at most 16 additions a value,
so it may differ by 2^-20 of itself between the two orders."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _models():
    import temgymcore_gb300 as t
    r = np.random.default_rng(4)
    out = []
    for nb in range(7):
        for ap in (False, True):
            comps, z = [], 0.0
            for b in range(max(nb, 1)):
                z += 0.1
                comps.append(t.Lens(z=z, focal_length=float(r.uniform(0.3, 2.0))))
                if b < nb:
                    z += 0.05
                    comps.append(t.Biprism(z=z, def_x=float(r.normal(0, 1e-3))))
                if ap:
                    z += 0.05
                    comps.append(t.Aperture(z=z, radius=float(r.uniform(1e-3, 3e-3))))
            out.append(comps)
    return out


@pytest.mark.parametrize("counts", [[1, 255, 256, 257, 511, 512, 513], [0, 31, 600, 1024, 1025, 2, 77]])
def test_batched_pairs_of_rays(cuda, counts):
    from temgymcore_gb300.batched import BatchedTrace
    models = _models()
    bt = BatchedTrace(models, [c for c in counts for _ in (0, 1)], tile_rays=512)
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    rays = [torch.randn(bt.total, device="cuda", generator=g) * s for s in (1e-3, 1e-3, 1e-3, 1e-3, 1e-3, 1e-3)]
    rays[0][::9] = 0.0  # on a biprism's edge while nothing has moved the ray
    rays[2][::9] = 0.0
    got = {}
    for block, rpt in ((256, 1), (256, 2), (128, 4), (512, 2)):
        out = bt.alloc_outputs()
        raw = torch.zeros((int(bt.step_offsets[-1]), 4), dtype=torch.float64, device="cuda")
        alive = torch.empty(bt.total, dtype=torch.uint8, device="cuda")
        loss = torch.empty(len(models), dtype=torch.float64, device="cuda")
        bt.run(*rays[:4], out, (rays[4], rays[5]), raw, block, rpt, alive=alive, loss=loss)
        got[block, rpt] = ([v.clone() for v in out], alive, loss)
    one, alive, loss = got[256, 1]
    assert 0 < int(alive.sum()) < bt.total
    for key, (out, a, ls) in got.items():
        for v, w in zip(out, one):
            assert torch.equal(v, w), key
        assert torch.equal(a, alive), key
        assert torch.all((ls - loss).abs() <= 2.0 ** -20 * loss), key
