"""GPU: the largest records of a batched model, alone and side by side: those that are
held twice over (at most four biprisms) and those that are not, in every launch shape.
Outputs and aperture decisions are the ones of one ray a thread, bit for bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _model(bip, ap, seed):
    import temgymcore_gb300 as t
    r = np.random.default_rng(seed)
    kinds = np.array([1] * bip + [0] * ap)
    r.shuffle(kinds)
    out = [t.Lens(z=0.1, focal_length=0.8)] if bip + ap < 60 else []
    for i, k in enumerate(kinds):
        z = 0.2 + 0.005 * i
        out.append(t.Biprism(z=z, def_x=float(r.normal(0, 1e-4))) if k else
                   t.Aperture(z=z, radius=float(r.uniform(3e-3, 6e-3))))
    return out


LARGE = {"pairs": [(4, 56)], "many": [(16, 44)], "both": [(4, 56), (16, 44), (0, 60), (5, 3), (1, 1), (3, 57)]}


@pytest.mark.parametrize("which", list(LARGE))
def test_largest_records(cuda, which):
    from temgymcore_gb300.batched import BatchedTrace
    models = [_model(b, a, i) for i, (b, a) in enumerate(LARGE[which])] * 3
    bt = BatchedTrace(models, [257 + 300 * i for i in range(len(models))], tile_rays=512)
    g = torch.Generator(device="cuda").manual_seed(3)
    rays = [torch.randn(bt.total, device="cuda", generator=g) * 1e-3 for _ in range(6)]
    got = {}
    for block in (128, 256, 512):
        for rpt in (1, 2, 4):
            out = bt.alloc_outputs()
            raw, alive, loss = bt.alloc_raw(), bt.alloc_alive(), bt.alloc_loss()
            bt.run(*rays[:4], out, (rays[4], rays[5]), raw, block, rpt, alive=alive, loss=loss)
            got[block, rpt] = [*out, alive]
    assert 0 < int(got[128, 1][-1].sum()) < bt.total
    for key, v in got.items():
        assert all(torch.equal(a, b) for a, b in zip(v, got[128, 1])), key
