"""The FP64 EPA's block kernel where its branches change: polytopes around 64
faces, loose-edge lists longer than a warp's lanes, pairs with close vertices
and every mix of collider types in a block: bit for bit the oracle's results."""
import numpy as np
import pytest
import torch

from distance3d_gb300 import workloads
from distance3d_gb300.collider_set import HULL, SPHERE, ColliderSet
from distance3d_gb300.epa import epa_batch
from distance3d_gb300.store import ColliderStore
from oracle import oracle

pytestmark = pytest.mark.gpu


def check(cs, i, j, **opt):
    g = oracle.gjk_distance(cs, i, j)
    k = np.flatnonzero((g["dist"] == 0) & (g["n_simplex"] == 4))
    i, j, simplex = np.asarray(i)[k], np.asarray(j)[k], g["simplex"][k]
    r = epa_batch(ColliderStore(cs), i, j, simplex, return_faces=True, **opt)
    ref = oracle.epa(cs, i, j, simplex, want_faces=True, **opt)
    assert np.array_equal(r["status"].cpu().numpy(), ref["status"])
    assert np.array_equal(r["n_faces"].cpu().numpy(), ref["n_faces"])
    assert np.array_equal(r["mtv"].cpu().numpy(), ref["mtv"], equal_nan=True)
    faces = r["faces"].cpu().numpy()
    for q, n in enumerate(ref["n_faces"]):
        assert np.array_equal(faces[q, :n], ref["faces"][q, :n], equal_nan=True)
    return len(k)


@pytest.mark.parametrize("opt", [dict(max_faces=f) for f in (4, 63, 64, 65, 66, 130)] +
                         [dict(max_faces=256, max_loose_edges=e) for e in (3, 28, 31, 33, 128)] +
                         [dict(epsilon=0.0), dict(epsilon=1e-2), dict(epsilon=0.3), dict(max_iter=1)])
def test_limits(opt):
    cs, i, j = workloads.pairs_all_types(900, seed=17, center_half_width=0.2, margin_fraction=0.3,
                                         types=workloads.ALL_TYPES_MESH)
    assert check(cs, i, j, **opt) > 300


@pytest.mark.parametrize("n", [1, 3, 4, 5, 40])
def test_large_horizons(n):
    """Dense hulls against spheres: new points see many faces at once."""
    rng = np.random.default_rng(n)
    nv = 200
    p = rng.standard_normal((n, nv, 3))
    p /= np.linalg.norm(p, axis=2, keepdims=True)
    p *= np.array([1.0, 1.0, 0.05])
    types = np.tile([HULL, SPHERE], n)
    poses = np.zeros((2 * n, 12))
    poses[:, [0, 4, 8]] = 1.0
    poses[1::2, 9:] = rng.uniform(-0.02, 0.02, (n, 3))
    params = np.zeros((2 * n, 4))
    params[1::2, 0] = 0.3
    off, cnt = np.full(2 * n, -1), np.zeros(2 * n, dtype=np.int64)
    off[::2], cnt[::2] = nv * np.arange(n), nv
    cs = ColliderSet(types, poses, params, off, cnt, p.reshape(-1, 3))
    k = np.arange(n, dtype=np.int32)
    check(cs, 2 * k, 2 * k + 1, max_faces=256, max_loose_edges=128)
