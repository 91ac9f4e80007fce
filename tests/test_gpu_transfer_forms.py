"""GPU: the stack transfer's forms (transfer.py:6-50): full matrices, a last row
0 0 0 0 1, x and y unmixed; plane counts about the four that are written
together; ray counts about a warp and a block; zeros, powers of two (where the
rounding to float64 changes its grid) and rays outside the double-float range.

Tolerance: a product keeps 2^-46 of its magnitude and a sum of five 2^-45, so
each result lies within 2^-44 of the sum of its terms' magnitudes."""
import numpy as np
import pytest

import oracle  # noqa: F401
from oracle import transfer as OT

pytestmark = pytest.mark.gpu


def _matrices(form, m, rng):
    mats = rng.normal(0, 1, (m, 5, 5)) * 0.6
    if form != "full":
        mats[:, 4] = [0, 0, 0, 0, 1]
    if form == "split":
        mats[:, [0, 2]] *= np.array([1, 0, 1, 0, 1.0])
        mats[:, [1, 3]] *= np.array([0, 1, 0, 1, 1.0])
    if form == "mixed":  # unmixed until a rotation half way
        mats[m - m // 2:] = _matrices("split", m // 2, rng)
    return mats


@pytest.mark.parametrize("form", ["full", "affine", "split", "mixed"])
@pytest.mark.parametrize("n,m", [(1, 1), (31, 2), (33, 3), (255, 4), (257, 5), (1000, 8), (700, 17)])
def test_transfer_forms(cuda, form, n, m):
    import temgymcore_gb300 as t
    rng = np.random.default_rng(n * 100 + m)
    mats = _matrices(form, m, rng)
    rays = np.hstack([rng.normal(0, 1e-3, (n, 4)), np.ones((n, 1))])
    rays[::5, 2] = 0.0
    rays[::7] = [0.5, -0.25, 2.0 ** -30, -(2.0 ** -20), 1.0]
    rays[n // 2, 0] = 1e-200  # outside the range: float64
    rays[-1, 1] = 1e30
    got = t.transfer_rays(rays, mats).cpu().numpy()
    ref = OT.transfer_rays(rays, mats)
    cum = OT.accumulate_matrices_cumulative(mats)
    scale = np.einsum("mij,nj->nmi", np.abs(cum), np.abs(rays))
    assert np.all(np.abs(got - ref) <= 2.0 ** -44 * scale + 1e-300)


def test_transfer_not_finite(cuda):
    """Infinities and NaN go through all 25 terms, as in float64."""
    import temgymcore_gb300 as t
    rng = np.random.default_rng(2)
    rays = np.hstack([rng.normal(0, 1e-3, (70, 4)), np.ones((70, 1))])
    rays[3, 0], rays[40, 3] = np.inf, np.nan
    mats = _matrices("split", 5, rng)
    got = t.transfer_rays(rays, mats).cpu().numpy()
    with np.errstate(invalid="ignore"):
        ref = OT.transfer_rays(rays, mats)
    np.testing.assert_array_equal(np.isnan(got), np.isnan(ref))
    np.testing.assert_array_equal(np.isinf(got), np.isinf(ref))
