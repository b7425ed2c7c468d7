"""The FP32 polytope search gives a pair the same bits with 8, 16 or 32 lanes
(by batch and polytope size) and with a whole warp (more than 255 face slots)."""
import numpy as np
import pytest

from distance3d_gb300 import workloads
from distance3d_gb300.epa import epa_batch
from distance3d_gb300.gjk import gjk_distance_batch
from distance3d_gb300.store import ColliderStore

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=["types", "meshes"])
def pairs(request):
    types = workloads.ALL_TYPES if request.param == "types" else workloads.ALL_TYPES_MESH
    cs, _, _ = workloads.pairs_all_types(900, seed=8, center_half_width=0.4, types=types)
    rng = np.random.default_rng(2)
    i = rng.integers(0, len(cs), 90001).astype(np.int32)
    j = rng.integers(0, len(cs), 90001).astype(np.int32)
    st = ColliderStore(cs)
    r = gjk_distance_batch(st, i, j, precision="mixed")
    hit = np.flatnonzero(((r["dist"] == 0) & (r["n_simplex"] == 4)).cpu().numpy())
    assert len(hit) > 16000  # above the size where several pairs share a warp
    return st, i[hit], j[hit], r["simplex"].cpu().numpy()[hit]


def run(pairs, sel, **kw):
    st, i, j, s = pairs
    r = epa_batch(st, i[sel], j[sel], s[sel], precision="mixed", **kw)
    return {k: v.cpu().numpy() for k, v in r.items()}


# fewer slots than a warp has lanes, tight edge lists, 2.8 KB and 4.5 KB polytopes
@pytest.mark.parametrize("kw", [dict(max_faces=4), dict(max_faces=9, max_loose_edges=3), dict(max_loose_edges=6),
                                dict(), dict(max_faces=256, max_loose_edges=128), dict(max_iter=0), dict(max_iter=3),
                                dict(max_iter=125, max_faces=300, max_loose_edges=255)])
def test_batch_sizes(pairs, kw):
    n = len(pairs[1])
    whole = run(pairs, slice(0, n), **kw)
    for size in (1, 2, 31, 700, 7295, 7297, 14600):
        lo = (n - size) // 2
        part = run(pairs, slice(lo, lo + size), **kw)
        for k in whole:
            assert np.array_equal(part[k], whole[k][lo:lo + size], equal_nan=k == "mtv"), (size, k)


def test_whole_warp(pairs):
    sel = slice(0, 9001)
    a = run(pairs, sel, max_iter=150, max_faces=255, max_loose_edges=255)  # byte ids
    b = run(pairs, sel, max_iter=150, max_faces=304, max_loose_edges=255)  # 304 slots: a warp per pair
    fits = b["n_faces"] < 200  # never near the smaller limit
    assert fits.mean() > 0.5
    for k in a:
        assert np.array_equal(a[k][fits], b[k][fits], equal_nan=k == "mtv"), k


def test_faces(pairs):
    n = 8000
    whole = run(pairs, slice(0, n), return_faces=True)
    part = run(pairs, slice(100, 400), return_faces=True)
    for r in range(300):
        f = part["n_faces"][r]
        assert f == whole["n_faces"][100 + r]
        assert np.array_equal(part["faces"][r, :f], whole["faces"][100 + r, :f], equal_nan=True)
