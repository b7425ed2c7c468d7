"""The order of the LBVH's leaves is that of 63-bit Morton codes computed in 64
bits ((center - least) / extent, 21 bits per axis), ties by index, at any scale
and position of the scene."""
import numpy as np
import pytest

from distance3d_gb300.bvh import LBVH

pytestmark = pytest.mark.gpu


def spread(v):
    r = np.zeros_like(v)
    for b in range(21):
        r |= ((v >> np.uint64(b)) & np.uint64(1)) << np.uint64(3 * b)
    return r


def order(a):
    with np.errstate(all="ignore"):
        c = 0.5 * (a[:, :, 0] + a[:, :, 1])
        q = []
        for k in range(3):
            v = c[:, k][~np.isnan(c[:, k])]
            least, ext = (v.min(), v.max() - v.min()) if len(v) else (np.nan, np.nan)
            x = (c[:, k] - least) / ext * 2097152.0 if ext > 0 else np.zeros(len(c))
            x = np.where(np.isnan(x) | (x <= 0), 0.0, np.minimum(x, 2097151.0))
            q.append(x.astype(np.uint64))
    return np.argsort((spread(q[0]) << np.uint64(2)) | (spread(q[1]) << np.uint64(1)) | spread(q[2]), kind="stable")


@pytest.mark.parametrize("kind", ["uniform", "large", "huge", "small", "tiny", "far_off", "grid", "flat", "one_place",
                                  "nan"])
@pytest.mark.parametrize("n", [1, 2, 3, 257, 60001])
def test_leaf_order(kind, n):
    rng = np.random.default_rng(n)
    c = rng.uniform(-1, 1, (n, 3))
    e = rng.uniform(0, 0.01, (n, 3))
    scale = {"large": 1e30, "huge": 1e200, "small": 1e-30, "tiny": 1e-306}.get(kind, 1.0)
    c, e = c * scale, e * scale
    if kind == "far_off":
        c += [1e6, -3e7, 5.0]
    if kind == "grid":
        c, e = np.round(c * 64) / 64, np.zeros_like(e)
    if kind == "flat":
        c[:, 1], e[:, 1] = 0.5, 0.0
    if kind == "one_place":
        c[:], e[:] = 0.25, 0.0
    a = np.stack([c - e, c + e], 2)
    if kind == "nan":
        a[::5, 1, 0] = np.nan
    t = LBVH(a)
    leaves = t.tree[512:512 + 4 * n].cpu().numpy().view(np.int32)  # after the header and the flags
    assert np.array_equal(leaves, order(a))
