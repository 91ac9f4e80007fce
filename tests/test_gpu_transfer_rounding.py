"""GPU: the last step of the double-float transfer, a pair of float32 to one float64.

The products and sums here are exact in a float32 pair, so the expected value is
exact too and no tolerance is needed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _out(rays, mats):
    import temgymcore_gb300 as t
    return t.transfer_rays(rays, mats).cpu().numpy()


def _scaled(c, full):
    """Every component times c (the last row too with full)."""
    m = np.diag([c, c, c, c, 1.0])
    if full:
        m[4] = [c, 0.0, 0.0, 0.0, 0.0]
    return m[None]


@pytest.mark.parametrize("full", [False, True])
@pytest.mark.parametrize("e", [-78, -77, -76, -75, -74, -73, -1, 0, 1])
def test_a_power_of_two_with_a_tail_of_the_other_sign(cuda, e, full):
    """hi = 2^e, lo = -2^(e - 30): the scale of the tail is at the edge of float32 at e = -75."""
    entry, comp = 2.0 ** (e // 2) * (1.0 - 2.0 ** -30), 2.0 ** (e - e // 2)
    rays = np.ones((5, 5))
    rays[:, :4] = comp * np.array([1.0, -1.0, 1.0, -1.0])
    rays[4, :4] = 0.0
    out = _out(rays, _scaled(entry, full))[:, 0]
    assert np.array_equal(out[:, :4], rays[:, :4] * entry)
    assert np.array_equal(out[:, 4], rays[:, 0] * entry if full else rays[:, 4])


@pytest.mark.parametrize("full", [False, True])
def test_a_sum_of_two_floats_is_rounded_to_nearest(cuda, full):
    """x' = x + dx of two float32 values is exact as a pair: the float64 sum of
    them is the result, for a tail of any size and sign and for powers of two."""
    r = np.random.default_rng(0)
    n = 20_000
    big = (r.uniform(1.0, 2.0, (2, n)) * 2.0 ** r.integers(0, 11, (2, n))).astype(np.float32)
    big[:, ::4] = 2.0 ** r.integers(0, 11, (2, n))[:, ::4]
    small = (r.uniform(1.0, 2.0, (2, n)) * 2.0 ** r.integers(-38, -16, (2, n))).astype(np.float32)
    rays = np.ones((n, 5))
    rays[:, :2] = (big * r.choice([-1, 1], (2, n))).T
    rays[:, 2:4] = (small * r.choice([-1, 1], (2, n))).T
    m = np.eye(5)
    m[0, 2] = m[1, 3] = 1.0
    if full:
        m[4] = [1.0, 0.0, 1.0, 0.0, 0.0]
    out = _out(rays, m[None])[:, 0]
    assert np.array_equal(out[:, :2], rays[:, :2] + rays[:, 2:4])
    assert np.array_equal(out[:, 2:4], rays[:, 2:4])
    assert np.array_equal(out[:, 4], rays[:, 0] + rays[:, 2] if full else rays[:, 4])


@pytest.mark.parametrize("n,m", [(1, 1), (257, 3), (38_912, 4), (38_913, 4), (5_000, 61), (8_000, 19), (8_000, 20)])
def test_planes_a_thread(cuda, n, m):
    """One, two or four planes a thread (by blocks): each plane of a stack is the
    last of the stack's first planes alone, bit for bit."""
    r = np.random.default_rng(n)
    mats = r.normal(0, 0.6, (m, 5, 5))
    mats[:, 4] = [0.0, 0.0, 0.0, 0.0, 1.0]
    rays = r.normal(0, 1.0, (n, 5))
    rays[:, 4] = 1.0
    out = _out(rays, mats)
    for p in {0, m // 2, m - 1}:
        # result[k] is the product of the last k + 1 matrices
        alone = np.concatenate([_out(rays[i:i + 500], mats[m - 1 - p:])[:, -1] for i in range(0, n, 500)])
        assert np.array_equal(out[:, p], alone)
