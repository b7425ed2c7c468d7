"""The FP64 GJK kernel's pool of pairs per block, at the batch sizes where its
distribution changes (a block per pair, blocks partly filled, every block
full and refilled) and on inputs where its hull scan, clipping and iteration
bound decide: bit for bit the oracle's results."""
import numpy as np
import pytest
import torch

from distance3d_gb300 import workloads
from distance3d_gb300.collider_set import HULL, ColliderSet
from distance3d_gb300.gjk import gjk_distance_batch, gjk_intersection_batch
from distance3d_gb300.store import ColliderStore
from oracle import oracle

pytestmark = pytest.mark.gpu


def check(cs, i1, i2, **opt):
    st = ColliderStore(cs)
    r = {k: v.cpu().numpy() for k, v in gjk_distance_batch(st, i1, i2, **opt).items()}
    o = dict(opt)
    if "max_iterations" in o:
        o["max_iter"] = o.pop("max_iterations")
    ref = oracle.gjk_distance(cs, i1, i2, **o)
    for k in ("dist", "cp1", "cp2", "simplex", "n_simplex", "status"):
        assert np.array_equal(r[k], ref[k], equal_nan=ref[k].dtype.kind == "f"), k
    assert np.array_equal(r["iterations"], ref["iterations"])
    kw = {k: v for k, v in opt.items() if k in ("tolerance", "max_iterations")}
    h = gjk_intersection_batch(st, i1, i2, **kw)
    okw = {k: v for k, v in o.items() if k in ("tolerance", "max_iter")}
    hit = oracle.gjk_intersection(cs, i1, i2, **okw)
    assert np.array_equal(h["hit"].cpu().numpy(), hit["hit"])
    assert np.array_equal(h["status"].cpu().numpy(), hit["status"])


SMS = 152


@pytest.mark.parametrize("n", [1, 2, 2 * SMS - 1, 2 * SMS + 1, 4095, 4097, 2 * SMS * 32 + 5, 2 * SMS * 256 - 1,
                               2 * SMS * 256 + 77])
def test_batch_sizes(n):
    check(*workloads.pairs_all_types(n, seed=n, margin_fraction=0.2))


@pytest.mark.parametrize("opt", [dict(max_distance_squared=0.02), dict(max_iterations=1), dict(max_iterations=7),
                                 dict(tolerance=0.05)])
def test_bounds(opt):
    check(*workloads.pairs_all_types(3001, seed=9, types=workloads.ALL_TYPES_MESH), **opt)


@pytest.mark.parametrize("nv", [1, 2, 31, 32, 33, 64, 65, 257, 1000])
def test_hulls_with_tied_vertices(nv):
    """Vertices on an integer grid, many of them repeated: the first maximum wins."""
    rng = np.random.default_rng(nv)
    n = 64
    v = rng.integers(-2, 3, size=(2 * n * nv, 3)).astype(float)
    v += np.repeat(rng.integers(-2, 3, size=(2 * n, 3)), nv, axis=0)
    eye = np.tile(np.concatenate([np.eye(3).reshape(9), np.zeros(3)]), (2 * n, 1))
    cs = ColliderSet(np.full(2 * n, HULL), eye, np.zeros((2 * n, 4)), nv * np.arange(2 * n), np.full(2 * n, nv), v)
    k = np.arange(n, dtype=np.int32)
    check(cs, 2 * k, 2 * k + 1)
    d = rng.integers(-1, 2, size=(2 * n, 3)).astype(float)
    s = ColliderStore(cs).support(np.arange(2 * n), torch.from_numpy(d)).cpu().numpy()
    assert np.array_equal(s, oracle.support_batch(cs, np.arange(2 * n), d))
