"""Pair sets of the LBVH around the sizes where its pair keys change width and
with degenerate box distributions, against brute force."""
import numpy as np
import pytest

from distance3d_gb300.bvh import LBVH

pytestmark = pytest.mark.gpu


def brute(a, b):
    hit = np.ones((len(a), len(b)), dtype=bool)
    for k in range(3):
        hit &= (a[:, None, k, 0] <= b[None, :, k, 1]) & (a[:, None, k, 1] >= b[None, :, k, 0])
    return np.argwhere(hit)


def boxes(n, seed, kind):
    rng = np.random.default_rng(seed)
    c = rng.uniform(-3, 3, (n, 3))
    if kind == "line":
        c[:, 1:] = 0.0
    if kind == "same":
        c[:] = 0.25
    if kind == "far" and n:
        c[::max(1, n // 3)] *= 1e9
    e = rng.uniform(0.0, 0.4, (n, 3))
    return np.stack([c - e, c + e], axis=2)


@pytest.mark.parametrize("kind", ["uniform", "line", "same", "far"])
@pytest.mark.parametrize("n,m", [(1, 1), (2, 3), (3, 2), (4, 5), (255, 257), (257, 1), (1025, 64), (1500, 1023)])
def test_pairs(n, m, kind):
    if kind == "same" and n > 300:
        n = 300
    a, q = boxes(n, n, kind), boxes(m, m + 7, kind)
    t = LBVH(a)
    s = brute(a, a)
    assert np.array_equal(t.self_pairs().cpu().numpy(), s[s[:, 0] < s[:, 1]])
    assert np.array_equal(t.query(q).cpu().numpy(), brute(a, q))
    moved = boxes(n, n + 1, kind)
    t.refit(moved).refit(moved)
    s = brute(moved, moved)
    assert np.array_equal(t.self_pairs().cpu().numpy(), s[s[:, 0] < s[:, 1]])


def test_unordered_boxes():
    """Empty (lower above upper) and NaN boxes overlap as the comparisons say."""
    a = boxes(400, 3, "uniform")
    a[::5, 0] = a[::5, 0, ::-1]
    a[::7, 1, 0] = np.nan
    a[::11, 2] = [-np.inf, np.inf]
    t = LBVH(a)
    s = brute(a, a)
    assert np.array_equal(t.self_pairs().cpu().numpy(), s[s[:, 0] < s[:, 1]])
    assert np.array_equal(t.query(a[:50]).cpu().numpy(), brute(a, a[:50]))
